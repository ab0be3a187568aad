// 2-bit / 1-bit matmul for one to sixteen activation rows (sm_100a): the exact int32 block sums of matmul_q2 / matmul_q1
// (run_q2_gemv, csrc/gemm_q2.cc:300-404; block_sums, src/kernels/lowbit/matmul.rs:373-421) on int8 warp-level tensor-core
// instructions, the activations' quantisation in front (quantize_row, src/kernels/lowbit/matmul.rs:354-371) and the
// reference's ordered fold behind, in one launch.
//
// mma.m16n8k32 takes a packed unit's lane vector as its A fragment (16 weight columns = M, 8 activation rows = N) and issues
// once per 8 to 10 cycles, as the f16 m16n8k16 does, so int8 halves both the instructions and the activations' bytes against codes
// held as f16.  2-bit weights are looked up in their codebook by byte permutes.  1-bit weights are not even shifted where K-blocks
// have 128 depths and more: bit p of every byte is the number 2^p, the eight bit positions of a word go to four accumulators, of
// weight 2^0, 2^2, 2^4, 2^6 (twice that for columns g + 8), and 4-fold adds and one shift at a block's end make the sum of them.
//
// One CTA of sixteen warps per SM.  It quantises the rows into shared memory itself, in the order of the B fragments (or copies
// the codes act_quant_kernel made, where lowbit_rows_quantises says no: every CTA repeats it), while its weights are on their way: a lane copies its own 16 bytes of every unit into its own ring slots (cp.async).  A warp takes a column group, or a part of
// its depth where a CTA has fewer groups than warps; block sums are whole in a warp, so the first part folds them in registers as
// they come, in K order (total = fmaf((float)sum, scale * sa, total), the reference's bits), and each later one keeps its sums in
// lane-private shared memory until the part before hands its totals on.
//
// What bounds it: instruction issue and, at its ends, latency (350 warp instructions a 1-bit unit at eight rows, 110 of them the
// quantisation, issue slots half busy; of 16000 cycles of an 8 x 4096 x 14336 call 5200 go into the quantisation, 6700 into the
// products, 2600 into the second parts' folds and the stores).  Against act_quant_kernel and the kernels that took these calls
// before (dp4a to four rows, f16 MMAs on subnormal weights above; us, graph replays; rows x depth x columns): 1-bit 8 x 4096 x 14336 15.9 ->
// 8.4, 1 x 4096 x 4096 6.1 -> 3.9, 1 x 4096 x 14336 11.3 -> 5.8, 16 x 4096 x 14336 27.3 -> 13.7; 2-bit 1 x 4096 x 11008 7.75 -> 6.1, 3 x 4096 x 14336
// 16.4 -> 8.5.
#include "epilogue.cuh"
#include "kernels.h"
#include "layout.h"

namespace smeg {
namespace {

constexpr int kRWarps = 16;
constexpr int kRThreads = 32 * kRWarps;
constexpr size_t kRSmemMost = 220 * 1024;

__device__ __forceinline__ void cpa16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(0u), "r"(sel));
    return d;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
// D (16 weight columns x 8 rows, s32) += A (16 x 32) * B (32 x 8, s8), or = (`fresh`); A unsigned for sign bits, signed for codebook values
template <int BITS>
__device__ __forceinline__ void mma_i8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, bool fresh) {
    const int c[4] = {fresh ? 0 : d[0], fresh ? 0 : d[1], fresh ? 0 : d[2], fresh ? 0 : d[3]};
    if (BITS == 1)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}

// Where the four codes of depths d..d+3 (d a multiple of 4) of a row lie: [unit][16-byte chunk][row][t][word of the chunk].  A
// lane's words of a unit are in the order of its B registers; `paired`: of the 1-bit form that multiplies two words at once.
template <int BITS, int PAIRED>
__device__ __forceinline__ int code_at(int d, int row, int m) {
    constexpr int UD = BITS == 2 ? kQ2UnitDepth : kQ1UnitDepth, CH = UD / 64;
    const int u = (unsigned)d / UD, r = d & (UD - 1), t = (r >> 3) & 3, qh = (r >> 2) & 1;
    const int word = BITS == 1 && PAIRED ? (r >> 7) * 8 + (((r >> 5) & 1) * 2 + qh) * 2 + ((r >> 6) & 1) : (r >> 5) * 2 + qh;
    return ((u * CH + (word >> 2)) * m * 4 + row * 4 + t) * 16 + (word & 3) * 4;
}

// amax -> 127 / amax (0 where there is none, an infinity or a NaN: every code is then 0, those of infinities and NaNs too).
__device__ __forceinline__ float block_inv(float amax) { return amax > 0.0f && amax <= 65504.0f ? __fdiv_rn(127.0f, amax) : 0.0f; }
// The codes of eight values.  v + 1.5 2^23 leaves v, rounded to nearest even, in the low bits; |v| <= 127 (1 + 2^-23).  (The sum is
// scalar: a packed product and a packed sum became one instruction, of one rounding.)
__device__ __forceinline__ uint2 codes8(const uint4& h, float inv) {
    const uint32_t w[4] = {h.x, h.y, h.z, h.w};
    uint32_t q[8];
    uint64_t iv;
    asm("mov.b64 %0, {%1, %1};" : "=l"(iv) : "f"(inv));
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(as_h2(w[e]));
        float a, b;
        asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%2, %3};\n\tmul.rn.f32x2 v, v, %4;\n\tmov.b64 {%0, %1}, v;\n\t}" : "=f"(a), "=f"(b) : "f"(f.x), "f"(f.y), "l"(iv));
        q[2 * e] = __float_as_uint(__fadd_rn(a, 12582912.0f));
        q[2 * e + 1] = __float_as_uint(__fadd_rn(b, 12582912.0f));
    }
    const uint32_t keep = inv > 0.0f ? 0xffffffffu : 0u;
    return make_uint2(__byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410) & keep,
                      __byte_perm(__byte_perm(q[4], q[5], 0x0040), __byte_perm(q[6], q[7], 0x0040), 0x5410) & keep);
}
// Largest |x| of the even and of the odd ones of eight values, a NaN above everything.
__device__ __forceinline__ uint32_t amax8(const uint4& h) {
    const __half2 a = __hmax2_nan(__habs2(as_h2(h.x)), __habs2(as_h2(h.y))), b = __hmax2_nan(__habs2(as_h2(h.z)), __habs2(as_h2(h.w)));
    const __half2 c = __hmax2_nan(a, b);
    return *reinterpret_cast<const uint32_t*>(&c);
}
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __half2 c = __hmax2_nan(as_h2(a), as_h2(b));
    return *reinterpret_cast<const uint32_t*>(&c);
}

// Eight consecutive depths of a row as f16 bits, zeros past k.
__device__ __forceinline__ uint4 load8(const LowbitGemvArgs& p, const uint16_t* row, int d) {
    if (d >= p.k) return make_uint4(0, 0, 0, 0);
    if (p.a_vec_ok) return *reinterpret_cast<const uint4*>(row + d);                              // (k is a multiple of 8 then)
    __align__(16) uint16_t h[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = d + e < p.k ? row[d + e] : (uint16_t)0;
    return *reinterpret_cast<uint4*>(h);
}
__device__ __noinline__ void codes_out(const LowbitGemvArgs& p, int r, int d, uint2 q) {
    for (int e = 0; e < 8; ++e)
        if (d + e < p.k) p.q_out[(size_t)r * p.k + d + e] = (int8_t)((e < 4 ? q.x : q.y) >> (8 * (e & 3)));
}

// quantize_row (src/kernels/lowbit/matmul.rs:354-371) of the CTA's rows, f16 in global memory, to codes in the order of the B
// fragments and each K-block's scale and sum of codes (SQ: [nb][scales, sums][M8]).  A warp takes 256 depths of eight rows (RB = 4:
// four at a time, whose maxima and sums share shuffles and whose divisions share lanes) or of the one row there is (RB = 1).
// LB: log2 of the K-block where the kernel is of one.
template <int BITS, int PAIRED, int RB, int LB>
__device__ __forceinline__ void quantise_rows(const LowbitGemvArgs& p, unsigned char* Qs, float* SQ, float* AMX, int m8) {
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int m = p.m, kq = p.kq, lb = LB ? LB : p.log2_block, chunks = (kq + 255) >> 8;
    // warps to a run of rows: the rows are dealt out where there are fewer runs of depths than warps
    const int deal = RB == 1 || chunks > 8 ? 1 : chunks > 4 ? 2 : 4, runs = chunks < kRWarps ? chunks : kRWarps;   // (deal x runs <= 16)
    int c0 = warp, row0 = 0;
    while (c0 >= runs) { c0 -= runs; row0 += RB; }
    const int row_step = RB * deal, m_mine = row0 < row_step ? m : 0;  // (a warp over has no rows, but meets the barriers)
    const bool out = p.q_out && blockIdx.x == 0;
    const int lanes = 1 << (lb < 8 ? lb - 3 : 5), mine = lane & (RB - 1);   // lanes of a K-block; the row whose division this lane does
    for (int pass = lb > 8 ? 0 : 1; pass < 2; ++pass) {                // (K-blocks longer than a warp's run: their maxima first)
        for (int c = c0; c < chunks; c += kRWarps) {
            const int d = c * 256 + lane * 8;
            unsigned char* to0 = Qs + code_at<BITS, PAIRED>(d, 0, m);
            const bool whole = p.a_vec_ok && d < p.k;                  // (k is a multiple of 8 then)
            const int to4 = code_at<BITS, PAIRED>(d + 4, 0, m) - code_at<BITS, PAIRED>(d, 0, m);
            for (int r00 = row0; r00 < m_mine; r00 += 2 * row_step) {
                uint4 hh[2][RB];
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int e = 0; e < RB; ++e) {
                        const int r = r00 + b * row_step + e;
                        hh[b][e] = make_uint4(0, 0, 0, 0);
                        if (r < m) hh[b][e] = whole ? *reinterpret_cast<const uint4*>(p.a + (size_t)(uint32_t)r * (uint32_t)p.k + d) : load8(p, p.a + (size_t)r * p.k, d);
                    }
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const uint4 (&h)[RB] = hh[b];
                    const int r0 = r00 + b * row_step;
                    if (r0 >= m) break;
                    float amax = 0.0f;
                    if (lb <= 8 || pass == 0) {
                        if (RB == 1) {
                            uint32_t a = amax8(h[0]);
                            a = max2(a, a >> 16);
                            for (int o = 1; o < lanes; o <<= 1) a = max2(a, __shfl_xor_sync(0xffffffffu, a, o));
                            amax = __half2float(__ushort_as_half((uint16_t)a));
                        } else {
                            // two rows in the halves of a word
                            const uint32_t a0 = amax8(h[0]), a1 = amax8(h[1 % RB]), a2 = amax8(h[2 % RB]), a3 = amax8(h[3 % RB]);
                            uint32_t m01 = max2(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632));
                            uint32_t m23 = max2(__byte_perm(a2, a3, 0x5410), __byte_perm(a2, a3, 0x7632));
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                if (o >= lanes) break;
                                m01 = max2(m01, __shfl_xor_sync(0xffffffffu, m01, o));
                                m23 = max2(m23, __shfl_xor_sync(0xffffffffu, m23, o));
                            }
                            const uint32_t mm = (mine & 2) ? m23 : m01;
                            amax = __half2float(__ushort_as_half((uint16_t)((mine & 1) ? mm >> 16 : mm)));
                        }
                    }
                    if (lb > 8) {
                        float* cell = AMX + (size_t)(d >> lb) * m8 + r0 + mine;
                        if (pass == 0) {
                            // (as integers: ordered like the values, a NaN above everything)
                            if (lane < RB && r0 + lane < m) atomicMax(reinterpret_cast<int*>(cell), __float_as_int(amax));
                            continue;
                        }
                        amax = r0 + mine < m && d < kq ? *cell : 0.0f;
                    }
                    const float inv_mine = block_inv(amax), sa_mine = __fdiv_rn(amax, 127.0f);
                    int qs[RB];
#pragma unroll
                    for (int e = 0; e < RB; ++e) {
                        const float inv = RB == 1 ? inv_mine : __shfl_sync(0xffffffffu, inv_mine, (lane & 28) | e);
                        const uint2 q = codes8(h[e], inv);
                        if (r0 + e < m && d < kq) {
                            *reinterpret_cast<uint32_t*>(to0 + (r0 + e) * 64) = q.x;
                            *reinterpret_cast<uint32_t*>(to0 + to4 + (r0 + e) * 64) = q.y;
                            if (out) codes_out(p, r0 + e, d, q);
                        }
                        qs[e] = BITS == 1 ? __dp4a((int)q.x, 0x01010101, __dp4a((int)q.y, 0x01010101, 0)) : 0;
                    }
                    int sum = 0;
                    if (BITS == 1 && RB == 1) {
                        sum = qs[0];
                        for (int o = 1; o < lanes; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    } else if (BITS == 1) {
                        // sums of at most 256 codes, two rows to a word
                        int s01 = qs[0] + qs[1 % RB] * 65536, s23 = qs[2 % RB] + qs[3 % RB] * 65536;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            if (o >= lanes) break;
                            s01 += __shfl_xor_sync(0xffffffffu, s01, o);
                            s23 += __shfl_xor_sync(0xffffffffu, s23, o);
                        }
                        const int ss = (mine & 2) ? s23 : s01, low = (int)(int16_t)ss;
                        sum = (mine & 1) ? (ss - low) >> 16 : low;
                    }
                    // lane e of a K-block's run has row r0 + e
                    if ((lane & (lanes - 1)) < RB && r0 + mine < m && d < kq) {
                        float* cell = SQ + (size_t)(d >> lb) * 2 * m8 + r0 + mine;
                        if (lb <= 8 || ((d - 8 * lane) & ((1 << lb) - 1)) == 0) {
                            cell[0] = sa_mine;
                            if (p.sa_out && blockIdx.x == 0 && (d >> lb) < p.nb_real) p.sa_out[(size_t)(r0 + mine) * p.nb_real + (d >> lb)] = sa_mine;
                        }
                        if (BITS == 1) {
                            if (lb <= 8) reinterpret_cast<int*>(cell)[m8] = sum;
                            else atomicAdd(reinterpret_cast<int*>(cell) + m8, sum);
                        }
                    }
                }
            }
        }
        if (pass == 0) __syncthreads();
    }
}

// NT: tiles of eight rows.  LONG: K-blocks of 128 depths (2: of 128 exactly).  ONE: one row (its cells alone are folded).
// SUMS: the block sums are stored as well.
template <int BITS, int NT, int LONG, int ONE, int SUMS>
__global__ void __launch_bounds__(kRThreads, 1) lowbit_rows_kernel(const __grid_constant__ LowbitGemvArgs p) {
    constexpr int UD = BITS == 2 ? kQ2UnitDepth : kQ1UnitDepth, CH = UD / 64, M8 = 8 * NT, PF = kRowsRing;
    constexpr int PAIRED = BITS == 1 && LONG;
    constexpr int NA = PAIRED ? 4 : LONG ? 2 : 1;                   // accumulators of a block
    constexpr int UB = LONG == 2 ? UD / 128 : 1;                    // K-blocks of a unit (whose sums are taken together)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int m = p.m, nb = p.nb, ku = p.ku, lb = p.log2_block;
    const int lparts = p.ns, parts = 1 << lparts, at_once = kRWarps >> lparts;      // parts of a column group's depth, column groups in work
    const int part = warp & (parts - 1), grp = warp >> lparts;
    unsigned char* at = smem_raw;
    unsigned char* Qs = at;
    at += (size_t)m * p.kq;
    float* SQ = reinterpret_cast<float*>(at);                       // [nb][activation scales, sums of codes][M8]
    at += (size_t)nb * M8 * 8;
    float* AMX = reinterpret_cast<float*>(at);                      // [nb][M8] (K-blocks longer than 256)
    if (lb > 8) at += (size_t)nb * M8 * 4;
    // then an area for each column group in work (a CTA with fewer groups than its warps could take has no more areas than groups)
    at += (size_t)grp * p.u_bytes;
    const uint4* ring = reinterpret_cast<const uint4*>(at) + part * PF * 32 + lane;
    at += (size_t)PF * kUnitBytes << lparts;
    uint16_t* SCs = reinterpret_cast<uint16_t*>(at);               // [nb][16]
    at += (size_t)nb * 32;
    float* hand = reinterpret_cast<float*>(at) + lane * 4;         // [NT][32] x 4: the totals between parts
    at += NT * 512;
    // this warp's run of the depth, whole K-blocks
    const int lbu = max(lb - (BITS == 2 ? 7 : 8), 0), nbu = (ku + (1 << lbu) - 1) >> lbu;
    const int u_begin = ((part * nbu) >> lparts) << lbu, u_end = min((((part + 1) * nbu) >> lparts) << lbu, ku), mine = u_end - u_begin;
    const int blk0 = (int)(((size_t)u_begin * UD) >> lb);
    // the sums of the parts behind the first, lane-private: [parts - 1][gpt blocks][NT][32]
    float4* keep = reinterpret_cast<float4*>(at) + (size_t)((part - 1) * p.gpt) * NT * 32 + lane;
    // this CTA's column groups
    const int first = (int)blockIdx.x * p.dq + min((int)blockIdx.x, p.dr), share = p.dq + ((int)blockIdx.x < p.dr ? 1 : 0);

    pdl_launch_dependents();
    auto unit_src = [&](int c) { return p.codes + ((size_t)(first + c) * ku + u_begin) * kUnitBytes + lane * 16; };
    auto start_group = [&](int c) {
        // the group's scale rows by the warps that share it, then this warp's first units
        const unsigned char* src = reinterpret_cast<const unsigned char*>(p.scales + (size_t)(first + c) * nb * 16);
        for (int ch = part * 32 + lane; ch < nb * 2; ch += parts * 32) cpa16(smem_u32(SCs) + ch * 16, src + (size_t)ch * 16);
        const unsigned char* lp = unit_src(c);
#pragma unroll
        for (int i = 0; i < PF; ++i) {
            if (i < mine) cpa16(smem_u32(ring + i * 32), lp + i * kUnitBytes);
            cpa_commit();
        }
    };
    if (grp < share) start_group(grp);
    // (rows past m and the parts that add up are zeros)
    for (int i = tid; i < nb * M8 * (lb > 8 ? 3 : 2); i += kRThreads) SQ[i] = 0.0f;
    __syncthreads();
    pdl_wait();                                                     // the activations may come from the kernel ahead
    if (p.a) quantise_rows<BITS, PAIRED, ONE ? 1 : 4, LONG == 2 ? 7 : 0>(p, Qs, SQ, AMX, M8);
    else {
        for (int i = tid; i < m * (p.kq / 16); i += kRThreads) {
            const int r = i / (p.kq / 16), d = (i % (p.kq / 16)) * 16;
            const uint4 v = *reinterpret_cast<const uint4*>(p.q + (size_t)r * p.kq + d);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) *reinterpret_cast<uint32_t*>(Qs + code_at<BITS, PAIRED>(d + 4 * e, r, m)) = w[e];
        }
        for (int i = tid; i < m * nb; i += kRThreads) {
            float* cell = SQ + (size_t)(i % nb) * 2 * M8 + i / nb;
            cell[0] = p.sa[i];
            reinterpret_cast<int*>(cell)[M8] = p.qsum ? p.qsum[i] : 0;
        }
    }
    cpa_wait<PF - 1>();                                             // the scale rows: the first group of copies
    __syncthreads();

    for (int c = grp; c < share; c += at_once) {
        const unsigned char* lp = unit_src(c) + (size_t)PF * kUnitBytes;
        float tot[NT][4];
        int acc[NT][NA][4];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                tot[n][j] = 0.0f;
#pragma unroll
                for (int q = 0; q < NA; ++q) acc[n][q][j] = 0;
            }
        const int col = (first + c) * 16 + g;
        // a graph of up to four scalars and column vectors (p.kc), resolved for columns g and g + 8
        float eo[4][2];
        if (p.kc) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < p.ep.n_nodes) {
                    const uint16_t* v = p.ep.nodes[q].ptr;
                    const bool vec = (p.kc >> (8 * q)) & 8;
                    eo[q][0] = !vec ? p.ep.nodes[q].scalar : col < p.n ? __half2float(__ushort_as_half(v[col])) : 0.0f;
                    eo[q][1] = !vec ? p.ep.nodes[q].scalar : col + 8 < p.n ? __half2float(__ushort_as_half(v[col + 8])) : 0.0f;
                }
        }
        // block sums in their place: total += sum * (scale * sa); sum = 2 S - sum(q) of sign bits
        int blk = blk0;
        const unsigned char* sc_at = reinterpret_cast<const unsigned char*>(SCs) + blk0 * 32 + 4 * g;
        const float* sq_at = SQ + blk0 * M8 * 2 + 2 * t;
        struct Ops { float2 sc, sa[NT]; int2 qs[NT]; };              // what a K-block's sums meet
        auto ops = [&](int b) {
            Ops o;
            o.sc = __half22float2(as_h2(*reinterpret_cast<const uint32_t*>(sc_at + 32 * b)));                    // columns g, g + 8
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                o.sa[n] = *reinterpret_cast<const float2*>(sq_at + 2 * M8 * b + 8 * n);                             // rows 2t, 2t + 1
                o.qs[n] = BITS == 1 ? *reinterpret_cast<const int2*>(sq_at + 2 * M8 * b + 8 * n + M8) : make_int2(0, 0);
            }
            return o;
        };
        // sum = 2 S - sum(q) of sign bits, as a float
        auto as_float = [&](int n, const int (&s)[4], const Ops& o, float (&v)[4]) {
            const int w[4] = {s[0] - o.qs[n].x, s[1] - o.qs[n].y, s[2] - o.qs[n].x, s[3] - o.qs[n].y};
            if (SUMS && blk < p.nb_real) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int row = 8 * n + 2 * t + (j & 1), cj = col + 8 * (j >> 1);
                    if (row < m && cj < p.n) p.sums_out[((size_t)row * p.n + cj) * p.nb_real + blk] = w[j];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = ONE && (j & 1) ? 0.0f : (float)w[j];
        };
        auto fold = [&](int n, const float (&v)[4], const Ops& o) {
            tot[n][0] = fmaf(v[0], __fmul_rn(o.sc.x, o.sa[n].x), tot[n][0]);
            tot[n][2] = fmaf(v[2], __fmul_rn(o.sc.y, o.sa[n].x), tot[n][2]);
            if (!ONE) {
                tot[n][1] = fmaf(v[1], __fmul_rn(o.sc.x, o.sa[n].y), tot[n][1]);
                tot[n][3] = fmaf(v[3], __fmul_rn(o.sc.y, o.sa[n].y), tot[n][3]);
            }
        };
        float4* kp = keep;
        // the sums of a K-block out of its accumulators
        auto sums_of = [&](const int (&a)[NT][NA][4], int n, int (&s)[4]) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[j] = 0;
                if (ONE && (j & 1)) continue;
                if (PAIRED) {
                    // weights 1, 4, 16, 64 (j < 2) or 2, 8, 32, 128: 64 times the sum, or 128 times; twice the sum is wanted
                    const int v = ((a[n][0][j] * 4 + a[n][1 % NA][j]) * 4 + a[n][2 % NA][j]) * 4 + a[n][3 % NA][j];
                    s[j] = v >> (j < 2 ? 5 : 6);
                } else {
                    const int v = a[n][0][j] + (NA == 2 ? a[n][1 % NA][j] : 0);
                    s[j] = BITS == 1 ? 2 * v : v;
                }
            }
        };
        auto next_block = [&]() {
            kp += NT * 32;
            ++blk;
            sc_at += 32;
            sq_at += M8 * 2;
        };
        // a K-block's end, its accumulators cleared for the next.  (K-blocks past the last one are zeros times zeros: a total is
        // never -0, so adding them changes nothing.)
        auto flush = [&]() {
            const Ops o = ops(0);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                int s[4];
                sums_of(acc, n, s);
                float v[4];
                as_float(n, s, o, v);
                if (part == 0) fold(n, v, o);
                else kp[n * 32] = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
                for (int q = 0; q < NA; ++q)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[n][q][j] = 0;
            }
            next_block();
        };
        const int bmask = (1 << lb) - 1;
        const uint4* slot = ring;
        const unsigned char* x_at = Qs + u_begin * CH * m * 64 + min(g, m - 1) * 64 + t * 16;
        const int x_up = (min(8 + g, m - 1) - min(g, m - 1)) * 64;     // (columns of rows past m are computed and left)
        int d1 = (u_begin + 1) * UD;                                // the unit's last depth and one
        for (int u = 0; u < mine; ++u) {
            cpa_wait<PF - 1>();                                     // this lane's copy of the unit has landed
            const uint4 wv = *slot;
            uint4 x[NT][CH];
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                x[0][j] = *reinterpret_cast<const uint4*>(x_at);
                if (NT == 2) x[NT - 1][j] = *reinterpret_cast<const uint4*>(x_at + x_up);
                x_at += m * 64;
            }
            const uint32_t words[4] = {wv.x, wv.y, wv.z, wv.w};
            const bool last = u == mine - 1;
            // (K-blocks of 128: what their sums will meet is read before the products, and the blocks of a unit are folded together,
            // so that no step waits for the one before it)
            Ops ob[UB];
            int sb[UB][NT][4];
            if (LONG == 2) {
#pragma unroll
                for (int b = 0; b < UB; ++b) ob[b] = ops(b);
            }
            if constexpr (PAIRED) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t wa = words[2 * h], wb = words[2 * h + 1];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t m0 = 0x01010101u << (2 * q), m1 = m0 << 1;
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            const uint4& xv = x[n][(h * 2 + (q >> 1)) % CH];
                            mma_i8<BITS>(acc[n][q % NA], wa & m0, wa & m1, wb & m0, wb & m1, (q & 1) ? xv.z : xv.x, (q & 1) ? xv.w : xv.y, LONG == 2);
                        }
                    }
                    if (LONG == 2) {
#pragma unroll
                        for (int n = 0; n < NT; ++n) sums_of(acc, n, sb[h % UB][n]);
                    } else if (((d1 - 128 * (1 - h)) & bmask) == 0 || (last && h == 1)) flush();
                }
            } else {
#pragma unroll
                for (int s = 0; s < UD / 32; ++s) {
                    uint32_t a[4];
                    if (BITS == 2) {
                        const uint32_t w = words[s & 3], e = w & 0x33333333u, o = (w >> 2) & 0x33333333u;
                        a[0] = prmt(p.lut, e); a[1] = prmt(p.lut, o); a[2] = prmt(p.lut, e >> 16); a[3] = prmt(p.lut, o >> 16);
                    } else {
                        const uint32_t w = words[s >> 1] >> (4 * (s & 1));
#pragma unroll
                        for (int j = 0; j < 4; ++j) a[j] = (w >> j) & 0x01010101u;
                    }
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const uint4& xv = x[n][s >> 1];
                        mma_i8<BITS>(acc[n][s % NA], a[0], a[1], a[2], a[3], (s & 1) ? xv.z : xv.x, (s & 1) ? xv.w : xv.y, LONG == 2 && s < 2);
                    }
                    if (!LONG && (((d1 - UD + 32 * (s + 1)) & bmask) == 0 || (last && s == UD / 32 - 1))) flush();
                }
                if (LONG == 2) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) sums_of(acc, n, sb[0][n]);
                } else if (LONG && ((d1 & bmask) == 0 || last)) flush();
            }
            if (LONG == 2) {
                float vb[UB][NT][4];
#pragma unroll
                for (int b = 0; b < UB; ++b) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) as_float(n, sb[b][n], ob[b], vb[b][n]);
                    next_block();
                }
#pragma unroll
                for (int b = 0; b < UB; ++b)
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (part == 0) fold(n, vb[b][n], ob[b]);
                        else kp[((b - UB) * NT + n) * 32] = make_float4(vb[b][n][0], vb[b][n][1], vb[b][n][2], vb[b][n][3]);
                    }
            }
            d1 += UD;
            if (u + PF < mine) cpa16(smem_u32(slot), lp);
            cpa_commit();
            lp += kUnitBytes;
            slot = slot + 32 == ring + PF * 32 ? ring : slot + 32;
        }
        if (parts > 1) {
            const int id = 1 + grp * (parts - 1) + part;            // of the hand-over to this part: id - 1
            if (part > 0) {
                asm volatile("bar.sync %0, 64;" ::"r"(id - 1) : "memory");
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const float4 v = *reinterpret_cast<const float4*>(hand + n * 128);
                    tot[n][0] = v.x; tot[n][1] = v.y; tot[n][2] = v.z; tot[n][3] = v.w;
                }
                const int end = blk;
                sc_at -= (blk - blk0) * 32;
                sq_at -= (blk - blk0) * M8 * 2;
                kp = keep;
#pragma unroll 4
                for (blk = blk0; blk < end; ++blk) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const float4 w = kp[n * 32];
                        const float v[4] = {w.x, w.y, w.z, w.w};
                        fold(n, v, ops(0));
                    }
                    kp += NT * 32;
                    sc_at += 32;
                    sq_at += M8 * 2;
                }
            }
            if (part < parts - 1) {
#pragma unroll
                for (int n = 0; n < NT; ++n) *reinterpret_cast<float4*>(hand + n * 128) = make_float4(tot[n][0], tot[n][1], tot[n][2], tot[n][3]);
                asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
                break;                                              // (one round where the depth is split)
            }
        }
        // ---- epilogue, store ----
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float x[4];
            if (p.kc) {
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = __half2float(__float2half_rn(tot[n][j]));
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int op = (p.kc >> (8 * q)) & 7;               // 1 add, 2 mul, 3 sub, 5 max, 6 min
                    if (op == 0) break;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float o = eo[q][j >> 1];
                        x[j] = op == 1 ? __fadd_rn(x[j], o) : op == 2 ? __fmul_rn(x[j], o) : op == 3 ? __fsub_rn(x[j], o) : op == 5 ? fmaxf(x[j], o) : fminf(x[j], o);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = 8 * n + 2 * t + (j & 1), cj = col + 8 * (j >> 1);
                if ((!ONE || !(j & 1)) && row < m && cj < p.n)
                    p.c[(size_t)row * p.n + cj] = p.kc ? __half_as_ushort(__float2half_rn(x[j])) : ep_store_value<0>(p.ep, tot[n][j], (size_t)row, (size_t)cj);
            }
        }
        if (c + at_once < share) {
            __syncwarp();                                           // the scale rows have been read
            start_group(c + at_once);
            cpa_wait<PF - 1>();
            __syncwarp();
        }
    }
    cpa_wait<0>();
}

// Column groups of a CTA, parts of their depth and K-blocks of a part, the bytes of a column group's area and the shared memory of it
// all (0: too much, or better left to the kernels for what does not fit).  Only what is at work is counted: a ring a warp that has a
// part, an area a column group in work.  (With rings and areas for sixteen warps whatever the share, a CTA of one or two groups ran
// out of memory for its parts' sums and one warp a group did the work; us, that / this, and the kernels before in brackets: columns x depth: 2-bit
// blocks of 64, 1 row 4096 x 14336 27.5 / 18.2 (17.6), 1-bit 8 rows 1024 x 8192 22.2 / 12.8 (15.3), blocks of 256, 16 rows 1024 x 8192
// 18.1 / 12.4 (12.9), blocks of 32, 2-bit 1 row 1024 x 8192 19.2 / 9.6 (13.7).)
size_t rows_plan(const LowbitGemvArgs& a, int bits, int sm_count, int* grid, int* parts, int* keep_blocks, int* area) {
    const int lu = bits == 2 ? 7 : 8, nt = a.m > 8 ? 2 : 1;
    const int bu = a.log2_block > lu ? 1 << (a.log2_block - lu) : 1, nbu = (a.ku + bu - 1) / bu;
    *grid = a.n16 < sm_count ? a.n16 : sm_count;
    const int share = (a.n16 + *grid - 1) / *grid;
    const size_t rows = (size_t)a.m * a.kq + (size_t)a.nb * 8 * nt * 4 * (a.log2_block > 8 ? 3 : 2);
    // Four parts at most, eight for long depths: every part's fold waits for the one before it (us with up to 2 / 4 / 8 / 16 parts: 2-bit
    // 1 row 512 x 2048 3.1 / 2.7 / 3.3 / 3.8, 1-bit 1024 x 4096 3.6 / 3.3 / 3.6 / 4.6, 4096 x 14336 12.0 / 11.8 / 9.9 / 9.9).
    for (int q = a.ku >= 48 ? 8 : 4; q >= 1; q >>= 1) {
        if (q > 1 && (q * share > kRWarps || q > nbu)) continue;
        // the most K-blocks of a part: of ceil(nbu / q) runs of bu units
        const size_t blocks = q > 1 ? (((size_t)((nbu + q - 1) / q) * bu << lu) >> a.log2_block) + 1 : 0;
        const size_t group = (size_t)q * kRowsRing * kUnitBytes + (size_t)a.nb * 32 + nt * 512 + (q - 1) * blocks * nt * 512;
        const size_t bytes = rows + (size_t)(kRWarps / q < share ? kRWarps / q : share) * group;
        if (bytes > kRSmemMost) continue;
        // More than eight rows in one part, with one group a CTA (or two, of K-blocks whose sums lowbit_mma_kernel has room for): one or
        // two of sixteen warps would do all the work (us, this / the other kernels: 1-bit 16 rows 1024 x 8192 blocks of 64 31.8 / 29.1, 12 rows
        // 1024 x 16384 blocks of 512 26.2 / 19.5, 4096 x 14336 blocks of 256 26.3 / 25.0; but blocks of 64, 4096 x 8192 30.3 / 33.6).
        if (q == 1 && nt == 2 && nbu >= 4 && (share == 1 || (share == 2 && a.log2_block >= 8))) return 0;
        *area = (int)group;
        *parts = q;
        *keep_blocks = (int)blocks;
        return bytes;
    }
    return 0;
}

}  // namespace

bool lowbit_rows_supported(const LowbitGemvArgs& a, int bits, int sm_count) {
    int grid, parts, blocks, area;
    return a.m >= 1 && a.m <= 16 && a.ku >= 1 && a.k >= 1 && a.log2_block >= 5 && rows_plan(a, bits, sm_count, &grid, &parts, &blocks, &area) != 0;
}

// Up to 40960 values (us, in the CTAs / in front, 1-bit blocks of 128: 16 rows 512 x 256 3.8 / 4.9, 8 rows 4096 x 14336 8.5 / 9.6, 9 rows 4096 x
// 4096 9.0 / 9.2; rows of 8192 depths and more meet earlier, 5 of 8192 x 1024 9.4 / 8.3).  K-blocks longer than a warp's run are read twice,
// for their maxima first: one round of sixteen runs of eight rows, or two of one row (blocks of 512, 1-bit: 8 rows 4096 x 4096 7.3 / 7.5, 1 row
// 8192 x 4096 6.3 / 7.0; 9 rows 4096 x 4096 9.9 / 8.4, 2 rows 8192 x 4096 9.3 / 7.8, 6 rows 6144 x 8192 11.8 / 9.4).
bool lowbit_rows_quantises(const LowbitGemvArgs& a) {
    if (a.log2_block <= 8) return (size_t)a.m * a.k <= 40960;
    const int chunks = (a.kq + 255) / 256, deal = a.m == 1 || chunks > 8 ? 1 : chunks > 4 ? 2 : 4;      // (as in quantise_rows)
    return (chunks + kRWarps - 1) / kRWarps * ((a.m + 8 * deal - 1) / (8 * deal)) <= (a.m == 1 ? 2 : 1);
}

cudaError_t lowbit_rows_launch(LowbitGemvArgs a, int bits, int sm_count, cudaStream_t stream) {
    int grid_x = 1, parts = 1, blocks = 0, area = 0;
    const size_t smem = rows_plan(a, bits, sm_count, &grid_x, &parts, &blocks, &area);
    if (!smem) return cudaErrorInvalidValue;
    a.ns = 0; a.gpt = blocks; a.u_bytes = area;
    while ((1 << a.ns) < parts) ++a.ns;
    // Graphs of up to four scalars and column vectors without an activation or a division are resolved once a lane: a byte a
    // node, its operation and 8 for a vector.
    a.kc = 0;
    for (int q = 0; q < a.ep.n_nodes; ++q) {
        int what = 0;
        if (q < 4)
            switch (a.ep.nodes[q].op & 0xffu) {
            case 0: what = 1; break; case 4: what = 9; break;
            case 1: what = 2; break; case 5: what = 10; break;
            case 11: what = 3; break; case 13: what = 11; break;
            case 9: what = 5; break; case 20: what = 13; break;
            case 10: what = 6; break; case 23: what = 14; break;
            default: break;
            }
        if (!what) { a.kc = 0; break; }
        a.kc |= what << (8 * q);
    }
    a.dq = a.n16 / grid_x; a.dr = a.n16 % grid_x;
    const bool two = a.m > 8, sums = a.sums_out != nullptr, one = a.m == 1 && !sums;
    const int big = a.log2_block == 7 ? 2 : a.log2_block > 7 ? 1 : 0;
    cudaError_t e;
#define SMEG_LR(BB, NN, GG, OO, SS)                                                                                        \
    if (bits == BB && two == (NN == 2) && big == GG && one == (OO == 1) && sums == (SS == 1)) {                            \
        e = cudaFuncSetAttribute(lowbit_rows_kernel<BB, NN, GG, OO, SS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRSmemMost); \
        return e != cudaSuccess ? e : launch_pdl(lowbit_rows_kernel<BB, NN, GG, OO, SS>, dim3(grid_x), dim3(kRThreads), smem, stream, a); \
    }
#define SMEG_LR3(BB, NN, OO, SS) SMEG_LR(BB, NN, 0, OO, SS) SMEG_LR(BB, NN, 1, OO, SS) SMEG_LR(BB, NN, 2, OO, SS)
    SMEG_LR3(1, 1, 0, 0) SMEG_LR3(1, 1, 1, 0) SMEG_LR3(1, 2, 0, 0) SMEG_LR3(1, 1, 0, 1) SMEG_LR3(1, 2, 0, 1)
    SMEG_LR3(2, 1, 0, 0) SMEG_LR3(2, 1, 1, 0) SMEG_LR3(2, 2, 0, 0) SMEG_LR3(2, 1, 0, 1) SMEG_LR3(2, 2, 0, 1)
#undef SMEG_LR3
#undef SMEG_LR
    return cudaErrorInvalidValue;
}

}  // namespace smeg
