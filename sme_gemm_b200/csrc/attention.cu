// Causal attention against an f16 key/value cache, and the append into that cache (sm_100a) -- the attention step of
// SelfAttention::accumulate (src/self_attention.rs:189-231) between its two projections:
//   attention_kv_causal_f16 / attention_kv_f16 (src/kernels/kv_attention.rs:29-331): query row i of a block attends to
//   keys 0..=start+i; per head softmax(f16(q * scale) . k) @ v, f32 sums, f32 probabilities exp(s - max), the division by
//   their sum last.  Query head h uses KV head h / (heads / kv_heads).
//   KvCache::extend (:499-520): a block's key and value rows copied to the cache's next positions.
//
// attn_tc_kernel forms both products on the 5th-generation tensor cores.  The query rows of one KV head -- every row of the
// block times every head of the group -- are the M dimension, 128 to a tile, so that grouped queries share one read of the
// keys and values; a key block is 128 keys.  Two passes over the keys of a tile:
//   1. S = Q K^T into tensor memory, the row maxima from it;
//   2. S again (not where both blocks of a short range are still in tensor memory), p = exp(s - max), O += P V.
// With the exact maximum known first, a probability is the reference's exp(s - max) whatever the order of the blocks, and no
// sum is ever rescaled; the second Q K^T costs a quarter of the tensor work, and the tensor pipe waits for the exponentials
// anyway.  Operands are exact: q and k are f16 already, and the f32 probability travels as the sum of two f16 numbers (p * 2^15 =
// hi + lo: 22 significant bits down to probabilities of 2^-29), two MMAs per step of P V.  The tensor core cuts its f32 sums off
// where an addition would round them, which grows with the length of a chain; so tensor memory holds one block's sums (the low
// parts', then the high parts'), and the softmax warps add them up in registers.  Error against 64 bits (2-norm), 512 rows over
// 1024 keys of 128 depths, flat / sharp scores: 4.4e-7 / 6.3e-7; the scalar f32 statement 6.2e-7 / 13.8e-7; one chain over all
// keys 20.1e-7 / 13.3e-7, at 31.5 us against 34.7.  (Two blocks a chain: 6.9e-7, 35.6 us.)
//
// Roles (320 threads): warps 0-7 (softmax; warp = 32 rows x 64 keys of a block, a thread one row), warp 8 (TMA: K and V
// blocks as three-dimensional boxes, so that a head of less than 64 depths and the rows past the last key read as zero),
// warp 9 (MMA).  P goes back into the S columns it was read from (A operand in tensor memory), V is taken as it lies in the
// cache ([key][depth]: an MN-major B operand).
//
// What bounds it: the chain of hand-offs of one CTA per SM -- about 14 instructions for each of a block's 16384 scores are
// ~1900 cycles per block on the four schedulers against ~1500 of tensor time, but a block takes ~4900: at 512 rows over 1024
// keys the issue slots are 32 % busy, the tensor pipe 15 %, and waits for tensor-memory loads lead the stalls.  A short prompt or a decode step has too few (tile, KV head)
// pairs for the machine: there a cluster of 2, 4 or 8 CTAs shares one tile's key blocks, each against the maximum of its own
// range, and the parts meet over distributed shared memory (out = sum_c e^(m_c - m) O_c / sum_c e^(m_c - m) l_c, in rank
// order).
#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace smeg {
namespace {

constexpr int kAtThreads = 320;
constexpr int kAtKeys = 128;                      // keys of a block
constexpr int kAtChunk = 128 * 128;               // bytes of 128 rows x 64 depths
constexpr int kAtMaxSlots = 8;
constexpr uint32_t kAtOCol = 256;                 // tensor memory: S / P buffers at columns 0 and 128, O behind them
constexpr float kAtPScale = 32768.0f;             // probabilities are scaled by 2^15 on their way into two f16 parts

// MN-major tile stored as rows of 64 MN elements (128 bytes, 128-byte swizzle) per K index: 8-row groups along K 1024 bytes
// apart, 64-element chunks along MN one kAtChunk apart.
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3fffu);
    d |= (uint64_t)(kAtChunk >> 4) << 16;         // leading byte offset: next 64 elements along MN
    d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset: next 8 rows along K
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* tmap, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t cluster_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_dsmem_f32x4(uint32_t cluster_addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
    return v;
}

// (x, y) += (a, b) in one instruction
__device__ __forceinline__ void add2(float& x, float& y, uint32_t a, uint32_t b) {
    asm("{\n\t.reg .b64 u, v;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tadd.rn.f32x2 u, u, v;\n\tmov.b64 {%0, %1}, u;\n\t}" : "+f"(x), "+f"(y) : "r"(a), "r"(b));
}
// Largest of a warp's 64 scores per row; keys from `lim` on do not count.
template <bool MASK>
__device__ __forceinline__ float block_max(uint32_t taddr, int lim, float mx) {
    uint32_t r[2][32];
    tmem_ld32(taddr, r[0]);
    tmem_ld32(taddr + 32, r[1]);
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float s = __uint_as_float(r[h][i]);
            mx = (!MASK || 32 * h + i < lim) ? fmaxf(mx, s) : mx;
        }
    return mx;
}

// p = exp(s - mx) of a warp's 64 scores per row, added to `sum`, and written over them as two f16 parts, 16 keys at a time: eight
// columns of high parts (two keys to a column), eight of low ones.
template <bool MASK>
__device__ __forceinline__ float block_exp(uint32_t taddr, int lim, float mx, float sum) {
    float sum2 = 0.0f;
    uint32_t r[2][16];
    tmem_ld16(taddr, r[0]);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        uint32_t hi[8], lo[8];
        tmem_ld_wait();
        if (h < 3) tmem_ld16(taddr + 16 * (h + 1), r[(h + 1) & 1]);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            float e0 = expf(__uint_as_float(r[h & 1][i]) - mx), e1 = expf(__uint_as_float(r[h & 1][i + 1]) - mx);
            if (MASK) {
                e0 = 16 * h + i < lim ? e0 : 0.0f;
                e1 = 16 * h + i + 1 < lim ? e1 : 0.0f;
            }
            sum += e0;
            sum2 += e1;
            e0 *= kAtPScale;
            e1 *= kAtPScale;
            const uint32_t p = pack2_t<0>(e0, e1);
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&p));
            hi[i / 2] = p;
            lo[i / 2] = pack2_t<0>(e0 - f.x, e1 - f.y);
        }
        tmem_st8(taddr + 16 * h, hi);
        tmem_st8(taddr + 16 * h + 8, lo);
    }
    tmem_st_wait();
    return sum + sum2;
}

// Eight results: two 16-byte stores (one as f16) where every row of out starts on a 16-byte boundary, else one by one.
template <int OUT16>
__device__ __forceinline__ void store8(const AttnArgs& p, size_t off, const float (&v)[8]) {
    if (OUT16) {
        uint4 o;
        o.x = pack2_t<0>(v[0], v[1]); o.y = pack2_t<0>(v[2], v[3]); o.z = pack2_t<0>(v[4], v[5]); o.w = pack2_t<0>(v[6], v[7]);
        uint16_t* d = reinterpret_cast<uint16_t*>(p.out) + off;
        if (p.out_vec) {
            *reinterpret_cast<uint4*>(d) = o;
            return;
        }
        const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = (uint16_t)(w[e / 2] >> (16 * (e & 1)));
    } else {
        float* d = reinterpret_cast<float*>(p.out) + off;
        if (p.out_vec) {
            *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(d + 4) = make_float4(v[4], v[5], v[6], v[7]);
            return;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = v[e];
    }
}

// Depths [c0, c1) of one (query row, head) by the scalar statement, a warp's work (all 32 lanes, the same arguments).  The
// products above are formed a key block at a time with the probabilities in two parts, so an infinity or NaN among the
// values reaches rows that do not attend to it (0 * inf) and an infinity turns into NaN (inf * 0 in the low part): a row
// whose result is not finite although its probabilities are is formed again here.  (With a NaN score the probabilities'
// sum is NaN and so is the scalar result: nothing to do.)  `base` is the row's maximum, to rounding.  A group of lanes takes
// a key, a lane eight of its depths in K and V: four keys of every group are on their way at once, and nothing but the
// score's reduction crosses lanes.  Every row formed again (an infinity at position 0):
// 512 rows over 1024 keys, 32 heads of 128, 1.7 ms, one row 0.19 ms; the scalar kernel that this one replaced took 1.3 and 0.08
// whatever the values, a thread per eight depths some hundreds.
template <int QF32, int OUT16>
__device__ __noinline__ void attend_exact_row(const AttnArgs& p, int i, int head, int c0, int c1, float base) {
    constexpr int B = 4;
    const int lane = threadIdx.x & 31;
    const int hd = p.head_dim, ld = p.kv_heads * hd, off = head / (p.heads / p.kv_heads) * hd, len = p.start + i + 1;
    int per = 1;                                               // lanes of a key
    while (per * 8 < hd) per *= 2;
    const int d = (lane & (per - 1)) * 8, keys = 32 / per;
    const bool in_k = d < hd, in_v = d >= c0 && d < c1;
    float q[8], acc[8], sum = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const size_t qo = (size_t)i * p.q_stride + (size_t)head * hd + d + e;
        float x = 0.0f;
        if (in_k) x = QF32 ? reinterpret_cast<const float*>(p.q)[qo] : __half2float(__ushort_as_half(reinterpret_cast<const uint16_t*>(p.q)[qo]));
        q[e] = __half2float(__float2half_rn(__fmul_rn(x, p.scale)));
        acc[e] = 0.0f;
    }
    for (int t0 = lane / per; __any_sync(0xffffffffu, t0 < len); t0 += keys * B) {
        uint4 k[B], v[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const size_t at = (size_t)min(t0 + b * keys, len - 1) * ld + off + d;
            k[b] = v[b] = make_uint4(0, 0, 0, 0);
            if (in_k) k[b] = *reinterpret_cast<const uint4*>(p.k + at);
            if (in_v) v[b] = *reinterpret_cast<const uint4*>(p.v + at);
        }
        // (the keys' chains side by side)
        float s[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const uint32_t w[4] = {k[b].x, k[b].y, k[b].z, k[b].w};
            s[b] = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                s[b] = __fadd_rn(s[b], __fmul_rn(q[2 * e], f.x));
                s[b] = __fadd_rn(s[b], __fmul_rn(q[2 * e + 1], f.y));
            }
        }
        for (int o = per >> 1; o; o >>= 1)
#pragma unroll
            for (int b = 0; b < B; ++b) s[b] += __shfl_xor_sync(0xffffffffu, s[b], o);
#pragma unroll
        for (int b = 0; b < B; ++b) s[b] = expf(__fsub_rn(s[b], base));
#pragma unroll
        for (int b = 0; b < B; ++b) {
            if (t0 + b * keys >= len) break;
            const uint32_t w[4] = {v[b].x, v[b].y, v[b].z, v[b].w};
            sum += s[b];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                acc[2 * e] = __fadd_rn(acc[2 * e], __fmul_rn(s[b], f.x));
                acc[2 * e + 1] = __fadd_rn(acc[2 * e + 1], __fmul_rn(s[b], f.y));
            }
        }
    }
    __syncwarp();
    for (int o = per; o < 32; o <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    }
    if (!in_v || lane >= per) return;
    const size_t dst = ((size_t)i * p.heads + head) * hd + d;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float r = __fdiv_rn(acc[e], sum);
        if (OUT16) reinterpret_cast<uint16_t*>(p.out)[dst + e] = __half_as_ushort(__float2half_rn(r));
        else reinterpret_cast<float*>(p.out)[dst + e] = r;
    }
}
__device__ __forceinline__ bool all_finite(const float (&v)[8]) {
    bool ok = true;
#pragma unroll
    for (int e = 0; e < 8; ++e) ok = ok && fabsf(v[e]) <= 3.402823466e38f;
    return ok;
}

// Behind a pass in which every lane stored eight results (`mask`: the lanes whose are not finite, with a good sum) at depth c of the tile's row r:
// the rows of the warp's bad results again, over the depths the warp holds of each (lanes of a row are neighbours, depths
// ascending; r < 0: no result).
template <int QF32, int OUT16>
__device__ __noinline__ void redo_bad(const AttnArgs& p, unsigned mask, int r, int c, float base, int row0, int kvh) {
    const int group = p.heads / p.kv_heads;
    while (mask) {
        const int first_bad = __ffs(mask) - 1, rr = __shfl_sync(0xffffffffu, r, first_bad);
        const unsigned same = __ballot_sync(0xffffffffu, r == rr);
        const int c0 = __shfl_sync(0xffffffffu, c, __ffs(same) - 1), c1 = __shfl_sync(0xffffffffu, c, 31 - __clz(same)) + 8;
        const int i = (row0 + rr) / group, g = (row0 + rr) - i * group;
        __syncwarp();
        attend_exact_row<QF32, OUT16>(p, i, kvh * group + g, c0, c1, __shfl_sync(0xffffffffu, base, first_bad));
        mask &= ~same;
    }
}

// Grid: (CTAs per tile, tiles of 128 query rows x heads of a group, KV heads); the CTAs of a tile are a cluster.
// NO: depths a softmax thread sums, half a head's, 64 or 128.
template <int QF32, int OUT16, int NO>
__global__ void __launch_bounds__(kAtThreads, 1) attn_tc_kernel(const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                                                                const __grid_constant__ AttnArgs p) {
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    __shared__ __align__(8) uint64_t bars[2 * kAtMaxSlots + 11];
    __shared__ float red_m[2][128], red_l[2][128];             // per half of the softmax warps and row: maximum, sum
    __shared__ float part_m[128], part_l[128];                 // of this CTA's key range
    __shared__ unsigned bad_rows[2][4];                        // per half and quarter: rows whose result is not finite
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    uint64_t *full = bars, *empty = full + kAtMaxSlots, *q_full = empty + kAtMaxSlots, *s_full = q_full + 1, *s_free = s_full + 2,
             *p_full = s_free + 2, *pv_done = p_full + 2, *o_free = pv_done + 2;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int hd = p.head_dim, group = p.heads / p.kv_heads, kvh = blockIdx.z;
    const int tile = gridDim.y - 1 - blockIdx.y;               // the tiles with the most keys first
    const int splits = gridDim.x, rank = blockIdx.x;
    const int row0 = tile * 128, nrow = min(128, p.rows * group - row0);
    const int nch = (hd + 63) >> 6, tile_bytes = nch * kAtChunk, hd16 = (hd + 15) & ~15;
    const int nslots = p.slots;
    // key blocks of the tile, and this CTA's share of them
    const int keys = p.start + (row0 + nrow - 1) / group + 1;
    const int nblk = (keys + kAtKeys - 1) / kAtKeys, per = (nblk + splits - 1) / splits;
    const int blk0 = min(rank * per, nblk), nb = min(per, nblk - blk0);
    const bool resident = nb <= 2;                             // both S buffers keep their block from pass 1 to pass 2
    unsigned char* q_s = smem;
    unsigned char* ring = smem + tile_bytes;

    if (tid == 0) {
        abort_word = 0;
        for (int i = 0; i < nslots; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_init(q_full, 256);
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 8); mbar_init(&p_full[i], 8); mbar_init(&pv_done[i], 1); mbar_init(&o_free[i], 8); }
        fence_barrier_init();
    }
    pdl_wait();                                                // (before the allocation: the kernel ahead may still hold tensor memory)
    if (warp == 9) {
        tmem_alloc(&tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = tmem_slot;

    if (warp == 8) {                                           // ---- K and V blocks ----
        if (elect_one()) {
            int n = 0;
            auto load = [&](const CUtensorMap* map, int j) {
                const int slot = n % nslots, round = n / nslots;
                ++n;
                if (round && !mbar_wait(&empty[slot], (round - 1) & 1, abort_flag, p.status)) return;
                mbar_expect_tx(&full[slot], tile_bytes);
                for (int c = 0; c < nch; ++c)
                    tma_load_3d(ring + (size_t)slot * tile_bytes + c * kAtChunk, map, c * 64, kvh, (blk0 + j) * kAtKeys, &full[slot]);
            };
            for (int j = 0; j < nb; ++j) load(&tk, j);
            if (!resident && nb) load(&tk, 0);
            for (int j = 0; j < nb; ++j) {
                if (!resident && j + 1 < nb) load(&tk, j + 1);
                load(&tv, j);
            }
        }
        __syncwarp();
    } else if (warp == 9) {                                    // ---- MMA ----
        const uint32_t idesc_s = umma_idesc(0, 128, kAtKeys);
        const uint32_t idesc_o = umma_idesc(0, 128, hd16) | (1u << 16);          // B is MN-major
        const int ksteps = hd16 >> 4;
        const uint32_t q_a = smem_u32(q_s), ring_a = smem_u32(ring);
        int n = 0;
        bool ok = nb > 0 && __all_sync(0xffffffffu, mbar_wait(q_full, 0, abort_flag, p.status));
        auto take = [&](uint32_t& addr, int& slot) {
            slot = n % nslots;
            addr = ring_a + (uint32_t)slot * tile_bytes;
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[slot], (n / nslots) & 1, abort_flag, p.status));
            ++n;
            tc_fence_after();
        };
        auto issue_s = [&](int b) {
            uint32_t addr;
            int slot;
            take(addr, slot);
            if (!ok) return;
            if (elect_one()) {
                for (int s = 0; s < ksteps; ++s) {
                    const uint32_t off = (uint32_t)((s >> 2) * kAtChunk + (s & 3) * 32);
                    umma_f16(tmem + 128 * b, umma_desc_sw128(q_a + off), umma_desc_sw128(addr + off), idesc_s, s > 0);
                }
                umma_commit(&empty[slot]);
                umma_commit(&s_full[b]);
            }
            __syncwarp();
        };
        for (int j = 0; ok && j < nb; ++j) {
            const int b = j & 1;
            if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&s_free[b], ((j >> 1) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (ok) { tc_fence_after(); issue_s(b); }
        }
        // pass 2: the scores of block j + 1 are formed while the softmax warps work on block j
        auto again = [&](int j) {
            const int b = j & 1, used = (nb - b + 1) >> 1;                       // uses of buffer b in pass 1
            if (j < 2) ok = ok && __all_sync(0xffffffffu, mbar_wait(&s_free[b], (used - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            else ok = ok && __all_sync(0xffffffffu, mbar_wait(&pv_done[b], ((j >> 1) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (ok) { tc_fence_after(); issue_s(b); }
        };
        if (!resident) again(0);
        for (int j = 0; ok && j < nb; ++j) {
            if (!resident && j + 1 < nb) again(j + 1);
            const int b = j & 1;
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&p_full[b], (j >> 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            // the sums of the block before (two blocks before, where tensor memory holds two) are in registers
            if (NO == 64 ? j >= 2 : j >= 1)
                ok = ok && __all_sync(0xffffffffu, NO == 64 ? mbar_wait(&o_free[b], ((j >> 1) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT)
                                                            : mbar_wait(&o_free[0], (j - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            uint32_t addr;
            int slot;
            take(addr, slot);
            if (!ok) break;
            if (elect_one()) {
                const uint32_t o = tmem + kAtOCol + (NO == 64 ? 128 * b : 0);
                for (int s = 0; s < kAtKeys / 16; ++s)           // the low parts first: small numbers
                    umma_f16_ts(o, tmem + 128 * b + 16 * s + 8, umma_desc_sw128_mn(addr + s * 2048), idesc_o, s > 0);
                for (int s = 0; s < kAtKeys / 16; ++s)
                    umma_f16_ts(o, tmem + 128 * b + 16 * s, umma_desc_sw128_mn(addr + s * 2048), idesc_o, 1);
                umma_commit(&empty[slot]);
                umma_commit(&pv_done[b]);
            }
            __syncwarp();
        }
    } else {                                                   // ---- softmax ----
        const int q4 = warp & 3, half = warp >> 2, row = q4 * 32 + lane;
        // the tile's queries: f16(q * scale), K-major with the 128-byte swizzle (rows past the tile's last are never read)
        for (int it = tid; it < nrow * nch * 8; it += 256) {
            const int r = it / (nch * 8), c = it - r * (nch * 8);                // row, run of 8 depths
            const int i = (row0 + r) / group, g = (row0 + r) - i * group;
            uint4 o = make_uint4(0, 0, 0, 0);
            if (c * 8 < hd) {
                const size_t src = (size_t)i * p.q_stride + (size_t)(kvh * group + g) * hd + c * 8;
                float x[8];
                if (QF32) {
                    const float* q = reinterpret_cast<const float*>(p.q) + src;
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = q[e];
                } else if (p.q_vec) {
                    const uint4 v = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.q) + src);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                        x[2 * e] = f.x;
                        x[2 * e + 1] = f.y;
                    }
                } else {
                    const uint16_t* q = reinterpret_cast<const uint16_t*>(p.q) + src;
#pragma unroll
                    for (int e = 0; e < 8; ++e) x[e] = __half2float(__ushort_as_half(q[e]));
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = __fmul_rn(x[e], p.scale);
                o.x = pack2_t<0>(x[0], x[1]); o.y = pack2_t<0>(x[2], x[3]); o.z = pack2_t<0>(x[4], x[5]); o.w = pack2_t<0>(x[6], x[7]);
            }
            *reinterpret_cast<uint4*>(q_s + (c >> 3) * kAtChunk + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = o;
        }
        fence_proxy_async();
        mbar_arrive(q_full);

        const bool live = q4 * 32 < nrow;                                        // does the warp hold rows of the tile?
        const uint32_t t_s = tmem + ((uint32_t)(q4 * 32) << 16) + 64 * half;
        const int len = row < nrow ? p.start + (row0 + row) / group + 1 : 0;     // keys this row attends to
        const int len_all = p.start + row0 / group + 1;                          // keys that every row of the tile attends to
        bool ok = true;
        float mx = -INFINITY;
        for (int j = 0; ok && j < nb; ++j) {
            const int b = j & 1, key0 = (blk0 + j) * kAtKeys + 64 * half;
            ok = __all_sync(0xffffffffu, mbar_wait(&s_full[b], (j >> 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (!ok) break;
            tc_fence_after();
            if (live) mx = key0 + 64 <= len_all ? block_max<false>(t_s + 128 * b, 0, mx) : block_max<true>(t_s + 128 * b, len - key0, mx);
            if (!resident) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_free[b]);
            }
        }
        red_m[half][row] = mx;
        named_barrier_sync(1, 256);
        mx = fmaxf(mx, red_m[half ^ 1][row]);
        const float mx_e = mx == -INFINITY ? 0.0f : mx;                          // no key of this range counts for the row
        float sum = 0.0f;
        // the two halves of the warps take a half of the depths each
        const int c_begin = half ? ((hd / 8 + 1) / 2) * 8 : 0, c_end = half ? hd : ((hd / 8 + 1) / 2) * 8;
        float o[NO];
#pragma unroll
        for (int c = 0; c < NO; ++c) o[c] = 0.0f;
        auto add_block = [&](int j) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait(&pv_done[j & 1], (j >> 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (!ok) return;
            tc_fence_after();
            if (live) {
                const uint32_t t_o = tmem + ((uint32_t)(q4 * 32) << 16) + kAtOCol + (NO == 64 ? 128 * (j & 1) : 0) + c_begin;
#pragma unroll
                for (int c = 0; c < NO; c += 32) {
                    uint32_t r[4][8];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (c_begin + c + 8 * u < c_end) tmem_ld8(t_o + c + 8 * u, r[u]);
                    tmem_ld_wait();
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (c_begin + c + 8 * u < c_end) {
#pragma unroll
                            for (int e = 0; e < 8; e += 2) add2(o[c + 8 * u + e], o[c + 8 * u + e + 1], r[u][e], r[u][e + 1]);
                        }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_free[NO == 64 ? j & 1 : 0]);
        };
        for (int j = 0; ok && j < nb; ++j) {
            const int b = j & 1, key0 = (blk0 + j) * kAtKeys + 64 * half;
            if (!resident) {
                const int used = (nb - b + 1) >> 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&s_full[b], (used + (j >> 1)) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
                if (!ok) break;
                tc_fence_after();
            }
            if (live) sum = key0 + 64 <= len_all ? block_exp<false>(t_s + 128 * b, 0, mx_e, sum) : block_exp<true>(t_s + 128 * b, len - key0, mx_e, sum);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[b]);
            if (j > 0) add_block(j - 1);
        }
        red_l[half][row] = sum;
        if (nb > 0) add_block(nb - 1);
        named_barrier_sync(1, 256);
        sum = red_l[0][row] + red_l[1][row];
        if (splits == 1) {
            const int i = (row0 + row) / group, g = (row0 + row) - i * group;
            const size_t dst = (size_t)i * p.heads * hd + (size_t)(kvh * group + g) * hd;
            bool bad = false;
#pragma unroll
            for (int c = 0; c < NO; c += 8) {
                if (!ok || c_begin + c >= c_end) break;
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = __fdiv_rn(o[c + e] * (1.0f / kAtPScale), sum);
                if (row < nrow) {
                    bad = bad || (sum > 0.0f && !all_finite(v));
                    store8<OUT16>(p, dst + c_begin + c, v);
                }
            }
            // rows to form again: the two warps that hold a row's halves take every other one, whole
            const unsigned mine = __ballot_sync(0xffffffffu, bad);
            if (lane == 0) bad_rows[half][q4] = mine;
            named_barrier_sync(1, 256);
            for (unsigned mask = (bad_rows[0][q4] | bad_rows[1][q4]) & (half ? 0xaaaaaaaau : 0x55555555u); mask; mask &= mask - 1) {
                const int l = __ffs(mask) - 1, tr = row0 + q4 * 32 + l;
                attend_exact_row<QF32, OUT16>(p, tr / group, kvh * group + tr % group, 0, hd, __shfl_sync(0xffffffffu, mx_e, l));
            }
        } else {
            if (half == 0) { part_m[row] = nb > 0 ? mx : -INFINITY; part_l[row] = sum; }
            float* o_s = reinterpret_cast<float*>(smem);                         // the operands are not needed any more
#pragma unroll
            for (int c = 0; c < NO; c += 4)
                if (c_begin + c < c_end && row < nrow) *reinterpret_cast<float4*>(o_s + (size_t)row * (hd + 4) + c_begin + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
        }
    }
    if (splits > 1) {                                          // ---- the parts of a cluster meet ----
        cluster_sync_all();
        const uint32_t o_a = smem_u32(smem), m_a = smem_u32(part_m), l_a = smem_u32(part_l);
        const int items = nrow * (hd / 8);
        // (warp by warp: `it0` is the warp's first item; a lane past the last one repeats it without a store)
        const bool sound = __all_sync(0xffffffffu, *abort_flag == 0);
        for (int it0 = rank * kAtThreads + (tid & ~31); sound && it0 < items; it0 += splits * kAtThreads) {
            const bool mine = it0 + lane < items;
            const int it = mine ? it0 + lane : items - 1, r = it / (hd / 8), c = (it - r * (hd / 8)) * 8;
            float m[8], l[8];
            float4 o[8][2];
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (s >= splits) break;
                m[s] = ld_dsmem_f32(mapa_shared(m_a + r * 4, s));
                l[s] = ld_dsmem_f32(mapa_shared(l_a + r * 4, s));
                const uint32_t oa = mapa_shared(o_a + (uint32_t)(r * (hd + 4) + c) * 4, s);
                o[s][0] = ld_dsmem_f32x4(oa);
                o[s][1] = ld_dsmem_f32x4(oa + 16);
            }
            float mx = -INFINITY;
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (s < splits) mx = fmaxf(mx, m[s]);
            float sum = 0.0f, v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (s >= splits || (m[s] == -INFINITY && l[s] == 0.0f)) continue;       // no key of this run counts (a NaN score does: l is NaN)
                const float f = expf(m[s] - mx);
                sum = fmaf(f, l[s], sum);
                v[0] = fmaf(f, o[s][0].x, v[0]); v[1] = fmaf(f, o[s][0].y, v[1]); v[2] = fmaf(f, o[s][0].z, v[2]); v[3] = fmaf(f, o[s][0].w, v[3]);
                v[4] = fmaf(f, o[s][1].x, v[4]); v[5] = fmaf(f, o[s][1].y, v[5]); v[6] = fmaf(f, o[s][1].z, v[6]); v[7] = fmaf(f, o[s][1].w, v[7]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __fdiv_rn(v[e] * (1.0f / kAtPScale), sum);
            const int i = (row0 + r) / group, g = (row0 + r) - i * group;
            if (mine) store8<OUT16>(p, (size_t)i * p.heads * hd + (size_t)(kvh * group + g) * hd + c, v);
            const unsigned mask = __ballot_sync(0xffffffffu, mine && sum > 0.0f && !all_finite(v));
            if (mask) redo_bad<QF32, OUT16>(p, mask, mine ? r : -1, c, mx, row0, kvh);
        }
        tc_fence_before();
        cluster_sync_all();                                    // nobody leaves while its shared memory is read
    } else {
        tc_fence_before();
        __syncthreads();
    }
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Decode: query rows x heads of a group up to 16 per KV head.  The tensor-core form above needs ~10 us for it whatever the
// number of keys -- tensor memory, a query tile of 128 rows, two passes handed from warp to warp.  Here a CTA is 8 warps on a
// run of keys of one KV head, the (at most 16) query rows are the M of mma.m16n8k16, and there are three barriers:
//   scores    B fragments straight from the cache, 16 bytes a lane (a lane's eight depths are two instructions' k indices,
//             the query fragments are taken in the same order), while the values of the run arrive in shared memory
//   softmax   two rows per warp: exact maximum, exp, the probabilities in two f16 parts as above
//   values    a warp owns eight depths at a time, ldmatrix.trans makes its B fragments
// The runs of one KV head are a cluster of up to eight CTAs and meet over distributed shared memory as above.
constexpr int kAdThreads = 256;
struct AdSmem {                                    // byte offsets; KC = keys of a CTA, a multiple of 16
    int q, s, hi, lo, v, o, total;
};
__host__ __device__ inline AdSmem ad_smem(int hd, int kc) {
    AdSmem a;
    a.q = 0;                                       // [16][hd32 + 8] f16, depths padded to whole runs of 32
    a.s = a.q + 16 * (((hd + 31) & ~31) + 8) * 2;  // [16][kc + 4] f32
    a.hi = a.s + 16 * (kc + 4) * 4;                // [16][kc + 8] f16
    a.lo = a.hi + 16 * (kc + 8) * 2;
    a.v = a.lo + 16 * (kc + 8) * 2;                // [kc][hd + 8] f16
    a.o = a.v + kc * (hd + 8) * 2;                 // [16][hd + 4] f32
    a.total = a.o + 16 * (hd + 4) * 4;
    return a;
}
constexpr int kAdMaxSmem = 226 * 1024;

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int QF32, int OUT16>
__global__ void __launch_bounds__(kAdThreads, 1) attn_decode_kernel(const __grid_constant__ AttnArgs p, int kc) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float part_m[16], part_l[16];
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int hd = p.head_dim, hd32 = (hd + 31) & ~31, group = p.heads / p.kv_heads, kvh = blockIdx.z;
    const int splits = gridDim.x, rank = blockIdx.x, nrow = p.rows * group;
    const int len = p.start + p.rows;
    const int key0 = rank * kc, nk = max(0, min(kc, len - key0)), nk16 = (nk + 15) & ~15;
    const AdSmem L = ad_smem(hd, kc);
    uint16_t* q_s = reinterpret_cast<uint16_t*>(smem + L.q);
    float* s_s = reinterpret_cast<float*>(smem + L.s);
    uint16_t *hi_s = reinterpret_cast<uint16_t*>(smem + L.hi), *lo_s = reinterpret_cast<uint16_t*>(smem + L.lo), *v_s = reinterpret_cast<uint16_t*>(smem + L.v);
    float* o_s = reinterpret_cast<float*>(smem + L.o);
    const size_t ld = (size_t)p.kv_heads * hd;
    pdl_launch_dependents();
    pdl_wait();
    // ---- values on their way, queries in place ----
    {
        const int per = hd / 8;
        const uint16_t* src = p.v + (size_t)key0 * ld + (size_t)kvh * hd;
        // (whole keys to a warp at a time: no division of an index for every 16 bytes)
        const int keys = 32 / per, mine = lane / per, c = (lane - mine * per) * 8;
        for (int r = warp * keys + mine; mine < keys && r < nk16; r += 8 * keys) {
            const uint32_t bytes = r < nk ? 16u : 0u;                            // (zeros behind the last key: nothing is read)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(v_s + (size_t)r * (hd + 8) + c)),
                         "l"(bytes ? src + (size_t)r * ld + c : p.v), "r"(bytes)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // A tile's keys leave before the queries, or the products of the tile before, are there: a trip to the cache is most of a short run
    // (with the index divisions gone from the two loops, us: 32 heads of 128 on 8 KV heads, 1024 keys 9.0 -> 8.1, 4096 keys 17.4 -> 16.1; 6 heads
    // of 64 at 128 keys 5.0, as before).
    const uint16_t* kb = p.k + (size_t)key0 * ld + (size_t)kvh * hd + 8 * t;
    auto load = [&](int tile, uint4 (&kv)[8]) {
        const int key = tile * 8 + g;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            kv[c] = make_uint4(0, 0, 0, 0);
            if (key < nk && 32 * c + 8 * t < hd) kv[c] = *reinterpret_cast<const uint4*>(kb + (size_t)key * ld + 32 * c);
        }
    };
    uint4 kv[8];
    load(warp, kv);
    for (int r = warp; r < 16; r += 8) {
        const int i = r / group;
        const size_t row = (size_t)i * p.q_stride + (size_t)(kvh * group + r - i * group) * hd;
        for (int d = lane; d < hd32; d += 32) {
            float x = 0.0f;
            if (r < nrow && d < hd) {
                x = QF32 ? reinterpret_cast<const float*>(p.q)[row + d] : __half2float(__ushort_as_half(reinterpret_cast<const uint16_t*>(p.q)[row + d]));
                x = __fmul_rn(x, p.scale);
            }
            q_s[r * (hd32 + 8) + d] = __half_as_ushort(__float2half_rn(x));
        }
    }
    __syncthreads();
    // ---- scores: a warp eight keys at a time ----
    {
        uint4 nx[8];
        for (int tile = warp; tile < nk16 / 8; tile += 8) {
            load(tile + 8, nx);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (32 * c >= hd) break;
                const uint4 qa = *reinterpret_cast<const uint4*>(q_s + g * (hd32 + 8) + 32 * c + 8 * t);
                const uint4 qb = *reinterpret_cast<const uint4*>(q_s + (g + 8) * (hd32 + 8) + 32 * c + 8 * t);
                mma_16816(acc, qa.x, qb.x, qa.y, qb.y, kv[c].x, kv[c].y);
                mma_16816(acc, qa.z, qb.z, qa.w, qb.w, kv[c].z, kv[c].w);
            }
            *reinterpret_cast<float2*>(s_s + g * (kc + 4) + tile * 8 + 2 * t) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(s_s + (g + 8) * (kc + 4) + tile * 8 + 2 * t) = make_float2(acc[2], acc[3]);
#pragma unroll
            for (int c = 0; c < 8; ++c) kv[c] = nx[c];
        }
    }
    __syncthreads();
    // ---- softmax of the run: two rows per warp ----
    for (int r = 2 * warp; r < min(2 * warp + 2, nrow); ++r) {
        const int lim = min(nk, p.start + r / group + 1 - key0);                 // keys of the run this row attends to
        const float* sr = s_s + r * (kc + 4);
        float mx = -INFINITY;
        for (int j = lane; j < lim; j += 32) mx = fmaxf(mx, sr[j]);
#pragma unroll
        for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float base = mx == -INFINITY ? 0.0f : mx;                          // no key of this run counts for the row
        float sum = 0.0f;
        for (int j = lane; j < nk16; j += 32) {
            float e = j < lim ? expf(sr[j] - base) : 0.0f;
            sum += e;
            e *= kAtPScale;
            const __half hi = __float2half_rn(e);
            hi_s[r * (kc + 8) + j] = __half_as_ushort(hi);
            lo_s[r * (kc + 8) + j] = __half_as_ushort(__float2half_rn(e - __half2float(hi)));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) { part_m[r] = mx; part_l[r] = sum; }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // ---- values: a warp eight depths at a time ----
    for (int n0 = warp * 8; n0 < hd; n0 += 64) {
        // 64 keys' high parts at a time: the instruction cuts its sums off where f32 addition rounds them
        float acc[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f}, run[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < nk16; k0 += 16) {
            uint32_t b0, b1;
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                         : "=r"(b0), "=r"(b1)
                         : "r"(smem_u32(v_s + (size_t)(k0 + (lane & 15)) * (hd + 8) + n0))
                         : "memory");
            const uint16_t *h = hi_s + g * (kc + 8) + k0 + 2 * t, *l = lo_s + g * (kc + 8) + k0 + 2 * t;
            const int down = 8 * (kc + 8);
            auto w = [](const uint16_t* x) { return *reinterpret_cast<const uint32_t*>(x); };
            mma_16816(run, w(h), w(h + down), w(h + 8), w(h + down + 8), b0, b1);
            mma_16816(low, w(l), w(l + down), w(l + 8), w(l + down + 8), b0, b1);
            if ((k0 & 48) == 48) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc[e] += run[e];
                    run[e] = 0.0f;
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] += run[e] + low[e];
        *reinterpret_cast<float2*>(o_s + g * (hd + 4) + n0 + 2 * t) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2*>(o_s + (g + 8) * (hd + 4) + n0 + 2 * t) = make_float2(acc[2], acc[3]);
    }
    // ---- the runs meet ----
    if (splits > 1) cluster_sync_all();
    else __syncthreads();
    const uint32_t o_a = smem_u32(o_s), m_a = smem_u32(part_m), l_a = smem_u32(part_l);
    const int items = nrow * (hd / 8);
    for (int it0 = rank * kAdThreads + (tid & ~31); it0 < items; it0 += splits * kAdThreads) {
        const bool mine = it0 + lane < items;                  // (a lane past the last item repeats it without a store)
        const int it = mine ? it0 + lane : items - 1, r = it / (hd / 8), c = (it - r * (hd / 8)) * 8;
        float m[8], l[8], mx = -INFINITY;
        float4 o[8][2];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (s >= splits) break;
            m[s] = ld_dsmem_f32(mapa_shared(m_a + r * 4, s));
            l[s] = ld_dsmem_f32(mapa_shared(l_a + r * 4, s));
            const uint32_t oa = mapa_shared(o_a + (uint32_t)(r * (hd + 4) + c) * 4, s);
            o[s][0] = ld_dsmem_f32x4(oa);
            o[s][1] = ld_dsmem_f32x4(oa + 16);
        }
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < splits) mx = fmaxf(mx, m[s]);
        float sum = 0.0f, v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (s >= splits || (m[s] == -INFINITY && l[s] == 0.0f)) continue;       // no key of this run counts (a NaN score does: l is NaN)
            const float f = expf(m[s] - mx);
            sum = fmaf(f, l[s], sum);
            v[0] = fmaf(f, o[s][0].x, v[0]); v[1] = fmaf(f, o[s][0].y, v[1]); v[2] = fmaf(f, o[s][0].z, v[2]); v[3] = fmaf(f, o[s][0].w, v[3]);
            v[4] = fmaf(f, o[s][1].x, v[4]); v[5] = fmaf(f, o[s][1].y, v[5]); v[6] = fmaf(f, o[s][1].z, v[6]); v[7] = fmaf(f, o[s][1].w, v[7]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = __fdiv_rn(v[e] * (1.0f / kAtPScale), sum);
        const int i = r / group, head = kvh * group + r - i * group;
        if (mine) store8<OUT16>(p, (size_t)i * p.heads * hd + (size_t)head * hd + c, v);
        const unsigned mask = __ballot_sync(0xffffffffu, mine && sum > 0.0f && !all_finite(v));
        if (mask) redo_bad<QF32, OUT16>(p, mask, mine ? r : -1, c, mx, 0, kvh);
    }
    if (splits > 1) cluster_sync_all();                        // nobody leaves while its shared memory is read
}

template <int QF32, int OUT16>
cudaError_t attn_decode_launch(const AttnArgs& a, int splits, int kc, cudaStream_t stream) {
    auto kern = attn_decode_kernel<QF32, OUT16>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kAdMaxSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, 1, a.kv_heads);
    cfg.blockDim = dim3(kAdThreads);
    cfg.dynamicSmemBytes = ad_smem(a.head_dim, kc).total;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, a, kc);
}

// rows x row_len f16 values from a strided source (the k or v part of projected [q | k | v] rows) to cache rows pos...; a
// thread moves 8 values of each (VEC: every address involved is 16-byte aligned) or one.
template <int VEC>
__global__ void kv_append_kernel(uint16_t* __restrict__ kc, uint16_t* __restrict__ vc, const uint16_t* __restrict__ src, size_t stride,
                                 size_t k_off, size_t v_off, size_t row_len, size_t pos, size_t rows) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t per = row_len / VEC, idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= rows * per) return;
    const size_t r = idx / per, c = (idx - r * per) * VEC;
    if (VEC == 8) {
        *reinterpret_cast<uint4*>(kc + (pos + r) * row_len + c) = *reinterpret_cast<const uint4*>(src + r * stride + k_off + c);
        *reinterpret_cast<uint4*>(vc + (pos + r) * row_len + c) = *reinterpret_cast<const uint4*>(src + r * stride + v_off + c);
    } else {
        kc[(pos + r) * row_len + c] = src[r * stride + k_off + c];
        vc[(pos + r) * row_len + c] = src[r * stride + v_off + c];
    }
}

template <int QF32, int OUT16>
cudaError_t attn_tc_launch(const CUtensorMap& tk, const CUtensorMap& tv, const AttnArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kern = a.head_dim <= 128 ? attn_tc_kernel<QF32, OUT16, 64> : attn_tc_kernel<QF32, OUT16, 128>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kAtThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = grid.x;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, tk, tv, a);
}

cudaError_t attn_launch(AttnArgs a, int q_f32, int sm_count, cudaStream_t stream) {
    a.out_vec = ((uintptr_t)a.out & 15) == 0;                  // (rows are heads * head_dim long: multiples of 16 bytes)
    if (a.rows * (a.heads / a.kv_heads) <= 16) {
        // runs of 64 keys and up; caches whose runs do not fit shared memory (about 4 k keys at 128 depths) stay below
        const int total = a.start + a.rows;
        int runs = 1;
        while (runs < 8 && total > 64 * runs && a.kv_heads * runs < sm_count) runs *= 2;
        const int kc = ((total + runs - 1) / runs + 15) & ~15;
        if (total <= 8 * 4096 && ad_smem(a.head_dim, kc).total <= kAdMaxSmem) {
            if (a.out16) return q_f32 ? attn_decode_launch<1, 1>(a, runs, kc, stream) : attn_decode_launch<0, 1>(a, runs, kc, stream);
            return q_f32 ? attn_decode_launch<1, 0>(a, runs, kc, stream) : attn_decode_launch<0, 0>(a, runs, kc, stream);
        }
    }
    TensorMapEncodeFn enc = tensor_map_encoder();
    if (!enc) return cudaErrorNotSupported;
    // [depth][KV head][position], a box = 64 depths of one head at 128 positions
    const size_t len = (size_t)a.start + a.rows, row = (size_t)a.kv_heads * a.head_dim;
    const cuuint64_t dim[3] = {(cuuint64_t)a.head_dim, (cuuint64_t)a.kv_heads, (cuuint64_t)len};
    const cuuint64_t stride[2] = {(cuuint64_t)a.head_dim * 2, (cuuint64_t)row * 2};
    const cuuint32_t box[3] = {64, 1, (cuuint32_t)kAtKeys}, estr[3] = {1, 1, 1};
    CUtensorMap tk, tv;
    if (enc(&tk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)a.k, dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
        enc(&tv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)a.v, dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    const size_t tiles = ((size_t)a.rows * (a.heads / a.kv_heads) + 127) / 128, blocks = (len + kAtKeys - 1) / kAtKeys;
    // a cluster shares a tile's key blocks while the machine has SMs to spare and every CTA keeps a block
    unsigned splits = 1;
    while (splits < 8 && splits * 2 <= blocks && tiles * a.kv_heads * splits * 2 <= (size_t)sm_count) splits *= 2;
    // ring of K / V blocks beside the query tile: at least two slots (heads of 256 depths)
    const int tile_bytes = ((a.head_dim + 63) / 64) * kAtChunk;
    a.slots = (216 * 1024 - tile_bytes) / tile_bytes;
    if (a.slots > kAtMaxSlots) a.slots = kAtMaxSlots;
    size_t smem = 1024 + (size_t)tile_bytes * (1 + a.slots);
    const size_t parts = 1024 + 128 * (size_t)(a.head_dim + 4) * 4;              // what a cluster's CTAs exchange lies over the operands
    if (splits > 1 && smem < parts) smem = parts;
    a.q_vec = a.q_stride % 8 == 0 && ((uintptr_t)a.q & 15) == 0;
    const dim3 grid(splits, (unsigned)tiles, (unsigned)a.kv_heads);
    if (a.out16) return q_f32 ? attn_tc_launch<1, 1>(tk, tv, a, grid, smem, stream) : attn_tc_launch<0, 1>(tk, tv, a, grid, smem, stream);
    return q_f32 ? attn_tc_launch<1, 0>(tk, tv, a, grid, smem, stream) : attn_tc_launch<0, 0>(tk, tv, a, grid, smem, stream);
}

}  // namespace

cudaError_t attn_kv_causal_launch(AttnArgs a, int q_f32, int sm_count, cudaStream_t stream) {
    // as many query rows to a launch as its grid has tiles of 128 rows x heads of a group (8.4 M of them)
    const int most = 65535 * 128 / (a.heads / a.kv_heads), rows = a.rows;        // (heads are at most 65535)
    for (int r = 0; r < rows; r += most) {
        AttnArgs s = a;
        s.start = a.start + r;
        s.rows = rows - r < most ? rows - r : most;
        s.q = static_cast<const char*>(a.q) + (size_t)r * a.q_stride * (q_f32 ? 4 : 2);
        s.out = static_cast<char*>(a.out) + (size_t)r * a.heads * a.head_dim * (a.out16 ? 2 : 4);
        const cudaError_t e = attn_launch(s, q_f32, sm_count, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t kv_append_launch(uint16_t* kc, uint16_t* vc, const uint16_t* src, size_t stride, size_t k_off, size_t v_off, size_t row_len,
                             size_t pos, size_t rows, cudaStream_t stream) {
    if (rows * row_len == 0) return cudaSuccess;
    const bool vec = row_len % 8 == 0 && stride % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0 &&
                     (((uintptr_t)kc | (uintptr_t)vc | (uintptr_t)src) & 15) == 0;
    const size_t threads = rows * row_len / (vec ? 8 : 1);
    const dim3 grid((unsigned)((threads + 255) / 256));
    if (vec) return launch_pdl(kv_append_kernel<8>, grid, dim3(256), 0, stream, kc, vc, src, stride, k_off, v_off, row_len, pos, rows);
    return launch_pdl(kv_append_kernel<1>, grid, dim3(256), 0, stream, kc, vc, src, stride, k_off, v_off, row_len, pos, rows);
}

}  // namespace smeg
