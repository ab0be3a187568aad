// Decode GEMV for a few activation rows, straight from global memory (sm_100a):
//   q4_stage_kernel       C[m][n] = ep( A[m][k] @ dequant(W) ), Q4 weights, f16, K-blocks of 32 and up, one or two rows
//                         of whole 16-byte words, on warp-level tensor-core instructions
//   q4_direct_kernel      the same in packed f16 arithmetic, for depths below 1793, and the form that norms its rows
//   lowbit_direct_kernel  2-bit / 1-bit weights against int8-quantised activations (matmul_q2 / matmul_q1): one to four rows under
//                         K-blocks of 16, short calls of one and two rows (lowbit_direct_shorter)
//
// They replace the reference's SME GEMV kernels for the batch sizes a decode step has
// (run_q4_gemv1 / run_q4_gemv, csrc/gemm_f16f16_q4.h:236-431; run_q2_gemv, csrc/gemm_q2.cc:300-404).
//
// A call of this size is a few microseconds long, so what it costs is the time to the first byte
// and the instructions issued per weight, not steady-state bandwidth.  Hence:
//   * no producer warp and no barrier: a packed unit (512 bytes, 16 columns) is one coalesced
//     16-byte asynchronous copy per lane into the lane's own slot of a shared-memory ring
//     (cp.async, a dozen units deep per warp: register loads cannot run that far ahead, a warp
//     has only a handful of scoreboards), and every warp issues its first ring-full as the first
//     thing the kernel does -- before the activations are staged and before the kernel ahead in
//     the stream has finished (the weights do not depend on it).  A lane reads back only what it
//     copied itself, so cp.async.wait_group is all the synchronisation the ring needs;
//   * one CTA owns whole column groups over the whole depth, its eight warps split the depth, so
//     a column's result never depends on the grid and nothing crosses CTAs;
//   * Q4, q4_direct_kernel: nibbles become exact f16 integers with one lop3 per pair, and are multiplied into
//     packed f16 sums over 8 depths (HFMA2, as the reference's SME kernel accumulates a K-block
//     in f16, csrc/gemm_f16f16_q4.h:236-341); every 32 depths the pair sums are widened and folded into
//     the f32 total with the block's scale.  Against the f32-accumulating oracle this differs by
//     f16 rounding of four-term partial sums and of their product with the scale, far inside the
//     1e-2 bar at the magnitudes activations have; but it is an f16 sum, which overflows beyond
//     65504 (a code of -8 times an activation above 8188) and is on f16's subnormal grid below
//     6e-5 -- calls that have f32 sums elsewhere (q4_mma_kernel) are not brought here for speed;
//   * 2-bit / 1-bit: the activation rows are quantised to int8 in shared memory by the CTA itself
//     (one or two rows; bit-exact quantize_row, src/kernels/lowbit/matmul.rs:354-371) or copied from
//     act_quant_kernel's output (more); codes are expanded in registers (2-bit: byte
//     permute of the 4-entry codebook, 1-bit: {0,1} bytes with sum = 2S - sum(q)), dot products
//     run on dp4a, exact int32 block sums meet in shared memory and one thread per output cell
//     folds them in K order with fmaf((float)sum, scale * sa, total) -- the reference's bits.
#include "epilogue.cuh"
#include "kernels.h"
#include "layout.h"

namespace smeg {
namespace {

constexpr int kDWarps = 8;
constexpr int kDThreads = 32 * kDWarps;

// Per-lane asynchronous copies global -> shared; a lane waits for its own groups only.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One packed Q4 word (8 nibbles, offset binary) -> the exact integer codes as f16 pairs:
// r[0] = column g (d, d+1), r[1] = column g+8 (d, d+1), r[2] = column g (d+2, d+3), r[3] = column g+8 (d+2, d+3).
__device__ __forceinline__ void q4_codes_h2(uint32_t w, __half2 (&r)[4]) {
    const uint32_t w8 = w >> 8;
    uint32_t lo0 = lop3_and_or(w, 0x000f000fu, 0x64006400u), hi0 = lop3_and_or(w, 0x00f000f0u, 0x64006400u);
    uint32_t lo1 = lop3_and_or(w8, 0x000f000fu, 0x64006400u), hi1 = lop3_and_or(w8, 0x00f000f0u, 0x64006400u);
    const __half2 off = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x6408));      // 1032
    const __half2 sc16 = __halves2half2(__ushort_as_half(0x2c00), __ushort_as_half(0x2c00));     // 1/16
    const __half2 off16 = __halves2half2(__ushort_as_half(0xd480), __ushort_as_half(0xd480));    // -72
    r[0] = __hsub2(*reinterpret_cast<__half2*>(&lo0), off);
    r[1] = __hsub2(*reinterpret_cast<__half2*>(&lo1), off);
    r[2] = __hfma2(*reinterpret_cast<__half2*>(&hi0), sc16, off16);
    r[3] = __hfma2(*reinterpret_cast<__half2*>(&hi1), sc16, off16);
}

__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

// ---------------------------------------------------------------------------------------------
// Q4, f16, M rows (1 or 2), K-blocks >= 32.
// Shared memory: ring [8 warps][PF][32 lanes] of {16 B codes} then {2 x 4 B scales} | A rows
// [M][kpad + 8] f16 | the cross-warp exchange [8 warps][CPC][M][16] f32.
// ---------------------------------------------------------------------------------------------
constexpr int kQ4PF = 8;                                           // units in flight per warp
constexpr size_t kQ4RingBytes = (size_t)kDWarps * kQ4PF * 32 * (16 + 8);

// Sum over the 256 threads of a CTA, in the order of the separate norm pass.
__device__ __forceinline__ float cta_sum(float v, float* sh) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();                       // sh may still be read from the previous call
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sh[w];
    return t;
}

// One activation row as the norm of an f32 row, in shared memory: the arithmetic and the order of norm_rows_kernel (the
// same bits), repeated by every CTA -- a row is a few KB out of L2 against a launch of its own in front of the projection.
__device__ __noinline__ void stage_norm_row(uint16_t* dst, const float* xr, const float* weight, const float* bias, int dim, int kpad, float eps,
                                            int rms, float* sh) {
    constexpr int KEEP = kNormInMost / kDThreads;              // values a thread keeps in registers between the passes
    const int tid = threadIdx.x;
    float x[KEEP];
#pragma unroll
    for (int i = 0; i < KEEP; ++i) x[i] = tid + i * kDThreads < dim ? xr[tid + i * kDThreads] : 0.0f;
    const float fdim = (float)dim;
    float mean = 0.0f;
    if (!rms) {
        float s = 0.0f;
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (tid + i * kDThreads < dim) s += x[i];
        mean = __fdiv_rn(cta_sum(s, sh), fdim);
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        if (tid + i * kDThreads < dim) {
            const float d = __fsub_rn(x[i], mean);
            ss = __fmaf_rn(d, d, ss);
        }
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(cta_sum(ss, sh), fdim), eps)));
    auto put = [&](int j, float v) {
        dst[j] = __half_as_ushort(__float2half_rn(__fadd_rn(__fmul_rn(__fmul_rn(__fsub_rn(v, mean), r), weight[j]), bias ? bias[j] : 0.0f)));
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        if (tid + i * kDThreads < dim) put(tid + i * kDThreads, x[i]);
    for (int j = dim + tid; j < kpad; j += kDThreads) dst[j] = 0;
}

// The warps' shares [8][cpc][M][16] in warp order, epilogue, store: `share` column groups (gated form: pairs of them) from `first`.
template <int M>
__device__ __forceinline__ void q4_store_cells(const Q4GemvArgs& p, const float* red, int CPC, int first, int share, int ncg) {
    const int tid = threadIdx.x;
    if (p.glu) {
        // a hidden unit's gate and up sums lie in neighbouring local groups: out = f16(act(f16(gate)) * f16(up)), the
        // arithmetic of the separate gate pass (glu, src/linear.rs:804-835) on the rounded projections
        const int hn = p.n >> 1;
        for (int o = tid; o < share * M * 16; o += kDThreads) {
            const int col16 = o & 15, r = (o >> 4) % M, ul = o / (16 * M);
            float ag = 0.0f, au = 0.0f;
#pragma unroll
            for (int w = 0; w < kDWarps; ++w) {
                ag += red[(((size_t)w * CPC + 2 * ul) * M + r) * 16 + col16];
                au += red[(((size_t)w * CPC + 2 * ul + 1) * M + r) * 16 + col16];
            }
            const float gv = __half2float(__float2half_rn(ag)), uv = __half2float(__float2half_rn(au));
            const int hcol = (first + ul) * 16 + col16;
            if (hcol < hn) p.c[(size_t)r * hn + hcol] = __half_as_ushort(__float2half_rn(__fmul_rn(glu_gate((uint32_t)p.glu, gv), uv)));
        }
        return;
    }
    for (int o = tid; o < ncg * M * 16; o += kDThreads) {
        const int col16 = o & 15, r = (o >> 4) % M, c = o / (16 * M);
        float acc = 0.0f;
#pragma unroll
        for (int w = 0; w < kDWarps; ++w) acc += red[(((size_t)w * CPC + c) * M + r) * 16 + col16];
        const int col = (first + c) * 16 + col16;
        if (col < p.n) {
            if (p.c32) p.c32[(size_t)r * p.n + col] = acc;
            else if (p.yacc) p.yacc[(size_t)r * p.n + col] = __fadd_rn(p.yacc[(size_t)r * p.n + col], __half2float(__float2half_rn(acc)));
            else if (p.kc && col >= p.q_len) {
                const int kv = col - p.q_len;
                const uint16_t v = __half_as_ushort(__float2half_rn(acc));
                if (kv < p.kv_len) p.kc[(size_t)r * p.kv_len + kv] = v;
                else p.vc[(size_t)r * p.kv_len + kv - p.kv_len] = v;
            }
            else p.c[(size_t)r * p.n + col] = ep_store_value<0>(p.ep, acc, (size_t)r, (size_t)col);
        }
    }
}

// GEN: the activations may be the norm of f32 rows (p.nx).
template <int M, int GEN>
__global__ void __launch_bounds__(kDThreads, 3) q4_direct_kernel(const __grid_constant__ Q4GemvArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int PF = kQ4PF;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int kpad = p.k64 * 64, a_stride = kpad + 8;
    uint4* ring_w = reinterpret_cast<uint4*>(smem_raw) + (size_t)warp * PF * 32 + lane;                     // + slot * 32
    uint32_t* ring_s = reinterpret_cast<uint32_t*>(smem_raw + (size_t)kDWarps * PF * 512) + (size_t)warp * PF * 64 + lane;   // + slot * 64 (+ 32)
    uint16_t* As = reinterpret_cast<uint16_t*>(smem_raw + kQ4RingBytes);
    float* red = reinterpret_cast<float*>(smem_raw + kQ4RingBytes + (size_t)M * a_stride * 2);
    const int CPC = p.cg;                                          // most column groups a CTA takes
    // this CTA's column groups: an equal share of all of them
    // (gated form: the share is counted in pairs of a gate group 4q + e and its up group 4q + 2 + e, e = 0, 1 -- the
    // matrix interleaves 32 gate and 32 up columns -- and the CTA walks gate, up, gate, up, ...)
    const int first = (int)blockIdx.x * p.dq + min((int)blockIdx.x, p.dr);
    const int share = p.dq + ((int)blockIdx.x < p.dr ? 1 : 0);
    const int ncg = p.glu ? 2 * share : share;
    auto group_of = [&](int c) -> int {
        if (!p.glu) return first + c;
        const int u = first + (c >> 1);
        return 4 * (u >> 1) + (u & 1) + 2 * (c & 1);
    };
    const int upw = p.dupw;                                        // units per warp: a contiguous run of the depth
    const int u_begin = min(warp * upw, p.k64), u_end = min(u_begin + upw, p.k64);
    const int total = ncg * (u_end - u_begin);                     // units this warp walks, column group by column group

    // load cursor: the unit's codes and the scale words of its two 32-deep halves (columns g, g + 8)
    const unsigned char* lp = p.codes + q4_unit_offset((size_t)group_of(0), (size_t)u_begin, p.k64) + lane * 16;
    const uint16_t* ls = p.scales + q4_scale_row((size_t)group_of(0), 0, p.nb) + 2 * g;
    int lu = u_begin, lc = 0;
    auto issue = [&](int slot) {
        cp_async16(ring_w + slot * 32, lp);
        cp_async4(ring_s + slot * 64, ls + (size_t)((lu * 64) >> p.log2_block) * 16);
        cp_async4(ring_s + slot * 64 + 32, ls + (size_t)((lu * 64 + 32) >> p.log2_block) * 16);
        lp += kUnitBytes;
        if (++lu == u_end) {
            lu = u_begin;
            const int cgn = group_of(++lc);                        // (one past the last group is never loaded from)
            lp = p.codes + q4_unit_offset((size_t)cgn, (size_t)u_begin, p.k64) + lane * 16;
            ls = p.scales + q4_scale_row((size_t)cgn, 0, p.nb) + 2 * g;
        }
    };
#pragma unroll
    for (int i = 0; i < PF; ++i) {
        if (i < total) issue(i);
        cp_async_commit();
    }
    pdl_launch_dependents();
    pdl_wait();                                                    // the activations may come from the kernel ahead

    // ---- stage the activation rows (zero past k) ----
    __shared__ float norm_sh[8];
    if (GEN && p.nx) {
        for (int r = 0; r < M; ++r) stage_norm_row(As + (size_t)r * a_stride, p.nx + (size_t)r * p.k, p.nw, p.nbias, p.k, kpad, p.neps, p.nrms, norm_sh);
    } else {
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll 2
            for (int d = tid * 8; d < kpad; d += kDThreads * 8)        // (k is a multiple of 8)
                *reinterpret_cast<uint4*>(As + (size_t)r * a_stride + d) =
                    d < p.k ? *reinterpret_cast<const uint4*>(p.a + (size_t)r * p.k + d) : make_uint4(0, 0, 0, 0);
    }
    __syncthreads();

    float tot[M][2];
#pragma unroll
    for (int r = 0; r < M; ++r) tot[r][0] = tot[r][1] = 0.0f;
    int cc = 0, cu = u_begin, slot = 0;                            // compute cursor
    const uint16_t* ap = As + cu * 64 + 8 * t;
    for (int j = 0; j < total; ++j) {
        cp_async_wait<PF - 1>();                                   // this lane's copies of unit j have landed
        const uint4 wv = ring_w[slot * 32];
        const uint32_t sw[2] = {ring_s[slot * 64], ring_s[slot * 64 + 32]};
        const uint32_t words[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            __half2 c0[4], c1[4];
            q4_codes_h2(words[2 * h], c0);
            q4_codes_h2(words[2 * h + 1], c1);
#pragma unroll
            for (int r = 0; r < M; ++r) {
                const uint4 av = *reinterpret_cast<const uint4*>(ap + (size_t)r * a_stride + 32 * h);
                __half2 s0 = __hmul2(c0[0], as_h2(av.x)), s1 = __hmul2(c0[1], as_h2(av.x));
                s0 = __hfma2(c0[2], as_h2(av.y), s0);
                s1 = __hfma2(c0[3], as_h2(av.y), s1);
                s0 = __hfma2(c1[0], as_h2(av.z), s0);
                s1 = __hfma2(c1[1], as_h2(av.z), s1);
                s0 = __hfma2(c1[2], as_h2(av.w), s0);
                s1 = __hfma2(c1[3], as_h2(av.w), s1);
                // (column g, column g + 8): the pair sums of 8 depths, times the block's scales, widened once
                const __half2 sum = __hadd2(__lows2half2(s0, s1), __highs2half2(s0, s1));
                const float2 f = __half22float2(__hmul2(sum, as_h2(sw[h])));
                tot[r][0] += f.x;
                tot[r][1] += f.y;
            }
        }
        if (j + PF < total) issue(slot);
        cp_async_commit();
        slot = slot + 1 == PF ? 0 : slot + 1;
        ap += 64;
        if (++cu == u_end) {
            // end of this warp's share of a column group: the four lanes of a column hold different depths
#pragma unroll
            for (int r = 0; r < M; ++r)
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    float v = tot[r][jj];
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if (t == 0) red[(((size_t)warp * CPC + cc) * M + r) * 16 + g + 8 * jj] = v;
                    tot[r][jj] = 0.0f;
                }
            cu = u_begin;
            ap = As + cu * 64 + 8 * t;
            ++cc;
        }
    }
    cp_async_wait<0>();
    if (total == 0) {
        // a warp with no depth of its own contributes zeros
        for (int o = lane; o < ncg * M * 16; o += 32) red[(size_t)warp * CPC * M * 16 + o] = 0.0f;
    }
    __syncthreads();
    q4_store_cells<M>(p, red, CPC, first, share, ncg);
}

// ---------------------------------------------------------------------------------------------
// Q4, f16, M rows (1 or 2), K-blocks >= 32, on warp-level tensor-core instructions: depths of eight stages and more.
//
// What q4_direct_kernel spends is instructions: 128 a unit of 1024 weights, of them 36 to make signed numbers of the codes, 32
// packed multiply-adds, 16 to widen and fold two K-blocks; 66 MB of a gate/up matrix were bound by them at 3.3 TB/s.  Here
//   * a code is not converted at all: four bits where they lie in a half word are the f16 subnormal u 2^-24 or u 2^-20 (u = code + 8),
//     one AND a pair; the products are exact in f32 and 8 sum(a) comes off through the accumulators' start values;
//   * mma.m16n8k16 has room for eight columns where there is one row, so the columns stand for K-blocks: a stage is four units,
//     lane (g, t) takes vectors of unit t, B is zero but where its column's K-block meets its depths, and after sixteen MMAs
//     the accumulators are the sums of eight K-blocks, folded at once (12 instructions instead of 128);
//   * the copies are coalesced a unit at a time and read back across the lanes, under an XOR of the unit's number.
// 61 warp instructions a unit (us, graph replays; q4_direct_kernel / this): 1 row, 28672 x 4096 17.8 / 12.3 (5.4 TB/s), 4096 x 14336
// 10.8 / 7.5, 4096 x 4096 3.95 / 3.25; 2 rows, 14336 x 4096 14.0 / 8.4 (but 1024 x 14336 7.9 / 8.5: rows that leave an SM room for one CTA).
// From 14336 to 28672 columns it adds 33 MB in 5.3 us, 6.2 TB/s: what is left is the time to the first byte and the last wave's end.
// Sums are f32 throughout (q4_direct_kernel: f16 over 8 depths): 2-norm of the error against 64 bits 2.1e-4 of the result, an exact
// product's f16 store, where q4_direct_kernel has 4.9e-4 (1 and 2 rows, 1024 to 14336 columns, 2048 to 14336 depths, blocks of 32 to 128).
// What a K-block's sum loses goes with 8 sum|a|, whatever its codes: columns of nothing but zero codes under nonzero scales are not
// exactly zero (up to 1.4e-6 with scales of 0.01 over 4096 normal activations, under the f16 store of any other column).
// Shared memory: ring [8 warps][PF] of a stage's codes and scale words | A rows [M][units * 72] f16 (a unit's 64 depths
// and 8 halves of padding) | the blocks' start values [stages][8 M] f32 | the cross-warp exchange [8 warps][CPC][M][16] f32.
// ---------------------------------------------------------------------------------------------
// Zeros where `bytes` is 0 (nothing is read then).
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4z(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16s(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4s(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
// D (16 weight columns x 8, f32) += A (16 x 16 f16) * B (16 x 8 f16)
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int kQ4StageUnits = 4;                                   // 256 depths
constexpr int kQ4AUnit = 72;                                       // halves from one unit of an activation row to the next
__host__ __device__ constexpr int q4_slot_bytes(int m) { return kQ4StageUnits * 512 + 256 * m; }
__host__ __device__ constexpr int q4_stages(int k64) { return (k64 + kQ4StageUnits - 1) / kQ4StageUnits; }
__host__ __device__ constexpr size_t q4_rows_bytes(int m, int stages) { return (size_t)m * stages * (kQ4StageUnits * kQ4AUnit * 2 + 32); }
// Where depth d lies in a staged row: the second and third pair of each run of eight change places, so that the pairs of one
// MMA's B operand are neighbours.
__device__ __forceinline__ int q4_a_index(int d) { return (d >> 6) * kQ4AUnit + (d & 57) + ((d & 2) << 1) + ((d & 4) >> 1); }

// Rows with an infinity or a NaN among their activations (bits of `rows`), again: the kernel's sums would carry them to columns
// whose code there is zero or make a NaN of them (it multiplies code + 8 and takes 8 times the row's sum off).  A thread a column,
// code by code; f32 sums of a K-block, folded with its scale.
template <int M>
__device__ __noinline__ void q4_exact_cells(const Q4GemvArgs& p, const uint16_t* As, int a_stride, float* red, int cpc, int ncg, int first, int rows) {
    for (int o = threadIdx.x; o < ncg * M * 16; o += kDThreads) {
        const int col16 = o & 15, r = (o >> 4) % M, c = o / (16 * M);
        if (!((rows >> r) & 1)) continue;                          // (a finite row's result does not depend on its neighbour's)
        const int u0 = first + (c >> 1);
        const int cg = p.glu ? 4 * (u0 >> 1) + (u0 & 1) + 2 * (c & 1) : first + c;
        float tot = 0.0f;
        for (int d0 = 0; d0 < p.k64 * 64; d0 += 32) {
            float part = 0.0f;
            for (int d = d0; d < d0 + 32; ++d) {
                size_t at;
                int nib;
                q4_locate((size_t)d, (size_t)cg * 16 + col16, (size_t)p.k64, &at, &nib);
                const int code = (int)((*reinterpret_cast<const uint32_t*>(p.codes + at) >> (4 * nib)) & 15u) - 8;
                if (d < p.k) part = fmaf((float)code, __half2float(__ushort_as_half(As[(size_t)r * a_stride + q4_a_index(d)])), part);
            }
            const uint16_t s = p.scales[q4_scale_row((size_t)cg, (size_t)(d0 >> p.log2_block), p.nb) + scale_slot(col16)];
            if (d0 < p.k) tot = fmaf(part, __half2float(__ushort_as_half(s)), tot);
        }
        for (int w = 0; w < kDWarps; ++w) red[((size_t)w * cpc + c) * M * 16 + r * 16 + col16] = w ? 0.0f : tot;
    }
}

// PF: ring slots per warp, a stage in work and the others on their way.
template <int M, int PF>
__global__ void __launch_bounds__(kDThreads, PF > 3 ? 2 : 3) q4_stage_kernel(const __grid_constant__ Q4GemvArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int SLOT = q4_slot_bytes(M), NC = M;              // NC accumulator pairs
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int ns = q4_stages(p.k64), a_stride = ns * kQ4StageUnits * kQ4AUnit;
    const uint32_t ring = smem_u32(smem_raw) + (uint32_t)(warp * PF * SLOT);
    uint16_t* As = reinterpret_cast<uint16_t*>(smem_raw + (size_t)kDWarps * PF * SLOT);
    float* start = reinterpret_cast<float*>(As + (size_t)M * a_stride);     // [stage][8 M]
    float* red = start + (size_t)ns * 8 * M;
    const int CPC = p.cg;                                          // most column groups a CTA takes
    // this CTA's column groups: an equal share of all of them
    // (gated form: the share is counted in pairs of a gate group 4q + e and its up group 4q + 2 + e, e = 0, 1 -- the
    // matrix interleaves 32 gate and 32 up columns -- and the CTA walks gate, up, gate, up, ...)
    const int first = (int)blockIdx.x * p.dq + min((int)blockIdx.x, p.dr);
    const int share = p.dq + ((int)blockIdx.x < p.dr ? 1 : 0);
    const int ncg = p.glu ? 2 * share : share;
    auto group_of = [&](int c) -> int {
        if (!p.glu) return first + c;
        const int u = first + (c >> 1);
        return 4 * (u >> 1) + (u & 1) + 2 * (c & 1);
    };
    // the eight warps split the depth: by the depth alone, so that a column's sum does not depend on the call's form
    const int s_begin = (warp * ns) >> 3, s_end = ((warp + 1) * ns) >> 3, mine = s_end - s_begin;
    const int total = ncg * mine;                                  // stages this warp walks

    // K-blocks (of the stage's eight) whose scales this lane folds: see below
    const int blk_a = M == 1 ? 4 * (t & 1) + (t >> 1) : 4 * (t & 1);
    // load cursor
    int ls = s_begin, lc = 0;
    const unsigned char* lp = p.codes;
    const unsigned char* lsc = p.codes;
    const uint32_t cg_codes = (uint32_t)p.k64 * kUnitBytes, cg_scales = (uint32_t)p.nb * 32, sc_shift = (uint32_t)p.log2_block - 5;
    auto load_from = [&](int c) {
        const uint32_t cg = (uint32_t)group_of(c);
        lp = p.codes + (uint64_t)cg * cg_codes + (uint32_t)(s_begin * kQ4StageUnits * kUnitBytes + lane * 16);
        lsc = reinterpret_cast<const unsigned char*>(p.scales) + (uint64_t)cg * cg_scales + (uint32_t)(4 * g);
    };
    const uint32_t wr = (uint32_t)(g * 64), wx = (uint32_t)(t << 4);
    auto issue = [&](uint32_t sb) {
        const uint32_t ss = sb + kQ4StageUnits * 512 + (uint32_t)(lane * 8 * M), sw = sb + wr;
        const uint32_t blk = (uint32_t)(ls * 8 + blk_a);           // counted in 32 depths
        if (ls * kQ4StageUnits + kQ4StageUnits <= p.k64) {
#pragma unroll
            for (int j = 0; j < kQ4StageUnits; ++j) cp_async16s(sw + (wx ^ (uint32_t)(j << 4)) + j * 512, lp + j * kUnitBytes);
#pragma unroll
            for (int e = 0; e < 2 * M; ++e) cp_async4s(ss + 4 * e, lsc + (((blk + (M == 1 ? 2 : 1) * e) >> sc_shift) << 5));
        } else {                                                   // the last stage of a depth that is no whole number of them: zeros
            const int left = p.k64 - ls * kQ4StageUnits;
#pragma unroll
            for (int j = 0; j < kQ4StageUnits; ++j)
                cp_async16z(sw + (wx ^ (uint32_t)(j << 4)) + j * 512, j < left ? lp + j * kUnitBytes : lp, j < left ? 16u : 0u);
#pragma unroll
            for (int e = 0; e < 2 * M; ++e) {
                const uint32_t be = blk + (M == 1 ? 2 : 1) * e;
                const bool in = be < (uint32_t)p.k64 * 2;
                cp_async4z(ss + 4 * e, in ? lsc + ((be >> sc_shift) << 5) : lsc, in ? 4u : 0u);
            }
        }
        lp += kQ4StageUnits * kUnitBytes;
        if (++ls == s_end) {
            ls = s_begin;
            if (++lc < ncg) load_from(lc);
        }
    };
    if (total) load_from(0);
#pragma unroll
    for (int i = 0; i < PF - 1; ++i) {
        if (i < total) issue(ring + (uint32_t)(i * SLOT));
        cp_async_commit();
    }
    pdl_launch_dependents();
    pdl_wait();                                                    // the activations may come from the kernel ahead

    // ---- stage the activation rows (zero past k), a warp a stage of 256 depths, and the blocks' start values: what the
    // products with code + 8 have too much, -8 sum(a) 2^-24 ----
    int bad = 0;
#pragma unroll
    for (int r = 0; r < M; ++r)
        for (int st0 = warp; st0 < ns; st0 += kDWarps * 4) {       // four loads on their way
            uint4 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int st = st0 + e * kDWarps, d = st * 256 + lane * 8;
                v[e] = make_uint4(0, 0, 0, 0);
                if (st < ns && d < p.k) v[e] = *reinterpret_cast<const uint4*>(p.a + (size_t)r * p.k + d);        // (k is a multiple of 8)
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int st = st0 + e * kDWarps, d = st * 256 + lane * 8;
                if (st >= ns) break;                               // (the same in all lanes)
                *reinterpret_cast<uint4*>(As + (size_t)r * a_stride + q4_a_index(d)) = make_uint4(v[e].x, v[e].z, v[e].y, v[e].w);
                const float2 f0 = __half22float2(as_h2(v[e].x)), f1 = __half22float2(as_h2(v[e].y)), f2 = __half22float2(as_h2(v[e].z)), f3 = __half22float2(as_h2(v[e].w));
                float sum = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                bad |= (int)!(fabsf(sum) <= 3.0e38f) << r;         // 32 finite f16 values sum to 2.1e6 at most
                // block 2 tb + h of the stage is column h * 4 + tb of the products (one row), r * 4 + tb of those of half h (two)
                const int tb = lane >> 3, h = (lane >> 2) & 1;
                if (t == 0) start[(size_t)st * 8 * M + (M == 1 ? h * 4 + tb : h * 8 + r * 4 + tb)] = sum * -4.76837158203125e-07f;
            }
        }
    __syncthreads();

    // ---- the products ----
    // Lane (g, t) multiplies the codes of unit t of the stage (of the lanes (g, 0..3) of that unit in turn), so the depths of
    // an MMA are those of four units, and column n of its B operand is zero but for the unit (and half, or row) n stands for:
    // an accumulator's column is one K-block's sum, and eight blocks are folded at once.
    const uint32_t a_base = smem_u32(As) + (uint32_t)(((M == 1 ? t * kQ4AUnit + (g >> 2) * 32 : (g >> 2) * a_stride + t * kQ4AUnit)) * 2);
    const bool on0 = (g & 3) == t && (M == 2 || g < 4), on1 = (g & 3) == t && (M == 2 || g >= 4);
    const uint32_t s_base = smem_u32(start) + (uint32_t)(8 * t);
    uint32_t rd[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) rd[i] = (uint32_t)(t * 512 + g * 64) + (wx ^ (uint32_t)(i << 4));
    uint4 b0[2], b1[2];                                            // (zero in the lanes that never load them)
    b0[0] = b0[1] = b1[0] = b1[1] = make_uint4(0, 0, 0, 0);
    float tot0 = 0.0f, tot1 = 0.0f;
    int cc = 0, cs = s_begin;                                     // compute cursor
    const uint32_t ring_end = ring + PF * SLOT;
    uint32_t sb = ring, fill = ring_end - SLOT;                    // the slot in work and the one before it
    uint32_t aa = a_base + (uint32_t)(s_begin * kQ4StageUnits * kQ4AUnit * 2), sa = s_base + (uint32_t)(s_begin * M * 32);
    for (int j = 0; j < total; ++j) {
        cp_async_wait<PF - 2>();
        __syncwarp();                                              // every lane's copies of the stage have landed, and the slot before is read
        if (j + PF - 1 < total) issue(fill);
        cp_async_commit();
        float lo[NC][4], hi[NC][4];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const uint2 s = lds64(sa + (uint32_t)(c * 32));
            lo[c][0] = lo[c][2] = __uint_as_float(s.x);
            lo[c][1] = lo[c][3] = __uint_as_float(s.y);
#pragma unroll
            for (int q = 0; q < 4; ++q) hi[c][q] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 wv = lds128(sb + rd[i]);
            if (on0) b0[i & 1] = lds128(aa + 16 * i);
            if (on1) b1[i & 1] = lds128(aa + (M == 1 ? 0 : 64) + 16 * i);
            // a nibble where it lies is the f16 subnormal u 2^-24 (low ones) or u 2^-20
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t w0 = h ? wv.z : wv.x, w1 = h ? wv.w : wv.y, v0 = w0 >> 8, v1 = w1 >> 8;
                const uint4& b = h ? b1[i & 1] : b0[i & 1];
                const int c = M == 1 ? 0 : h;
                mma_f16(lo[c], w0 & 0x000f000fu, v0 & 0x000f000fu, w1 & 0x000f000fu, v1 & 0x000f000fu, b.x, b.y);
                mma_f16(hi[c], w0 & 0x00f000f0u, v0 & 0x00f000f0u, w1 & 0x00f000f0u, v1 & 0x00f000f0u, b.z, b.w);
            }
        }
        uint32_t sw[2 * M];
        const uint32_t ss = sb + kQ4StageUnits * 512 + (uint32_t)(lane * 8 * M);
        if (M == 1) {
            const uint2 v = lds64(ss);
            sw[0] = v.x; sw[1] = v.y;
        } else {
            const uint4 v = lds128(ss);
            sw[0] = v.x; sw[2 * M - 2] = v.z; sw[1] = v.y; sw[2 * M - 1] = v.w;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            // columns 2t, 2t + 1 of the products: blocks blk_a and blk_a + 2 (one row); of half c: blk_a + c and blk_a + 2 + c (two)
            const float2 fa = __half22float2(as_h2(M == 1 ? sw[0] : sw[c])), fc = __half22float2(as_h2(M == 1 ? sw[1] : sw[(2 + c) % (2 * M)]));
            tot0 = fmaf(fmaf(hi[c][0], 0.0625f, lo[c][0]), fa.x, tot0);
            tot1 = fmaf(fmaf(hi[c][2], 0.0625f, lo[c][2]), fa.y, tot1);
            tot0 = fmaf(fmaf(hi[c][1], 0.0625f, lo[c][1]), fc.x, tot0);
            tot1 = fmaf(fmaf(hi[c][3], 0.0625f, lo[c][3]), fc.y, tot1);
        }
        fill = sb;
        sb = sb + SLOT == ring_end ? ring : sb + SLOT;
        aa += kQ4StageUnits * kQ4AUnit * 2;
        sa += M * 32;
        if (++cs == s_end) {
            // end of this warp's share of a column group: the lanes of a column (and row) hold different blocks
            tot0 += __shfl_xor_sync(0xffffffffu, tot0, 1);
            tot1 += __shfl_xor_sync(0xffffffffu, tot1, 1);
            if (M == 1) {
                tot0 += __shfl_xor_sync(0xffffffffu, tot0, 2);
                tot1 += __shfl_xor_sync(0xffffffffu, tot1, 2);
            }
            if ((t & (M == 1 ? 3 : 1)) == 0) {
                float* to = red + ((warp * CPC + cc) * M + (M == 1 ? 0 : t >> 1)) * 16;
                to[g] = tot0 * 16777216.0f;
                to[g + 8] = tot1 * 16777216.0f;
            }
            tot0 = tot1 = 0.0f;
            aa -= (uint32_t)(mine * kQ4StageUnits * kQ4AUnit * 2);
            sa -= (uint32_t)(mine * M * 32);
            cs = s_begin;
            ++cc;
        }
    }
    cp_async_wait<0>();
    if (__syncthreads_or(bad)) {
        int rows = 0;
#pragma unroll
        for (int r = 0; r < M; ++r) rows |= __syncthreads_or((bad >> r) & 1) ? 1 << r : 0;
        q4_exact_cells<M>(p, As, a_stride, red, CPC, ncg, first, rows);
        __syncthreads();
    }
    q4_store_cells<M>(p, red, CPC, first, share, ncg);
}

// ---------------------------------------------------------------------------------------------
// 2-bit / 1-bit weights x int8 activations, M rows (1..4).
// Shared memory: ring [8 warps][PF][32 lanes] of 16 B codes | Qs [M][kq + 16] int8 | SAs [M][nb] f32 |
//                QSs [M][nb] i32 | AMX [M][nb] i32 | sums [2][nb][M][16] i32 | staged scale rows.
// ---------------------------------------------------------------------------------------------
constexpr int kLbPF = 8;                                           // units in flight per warp
constexpr size_t kLbRingBytes = (size_t)kDWarps * kLbPF * 512;

__device__ __forceinline__ uint32_t prmt_lut(uint32_t lut, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(lut), "r"(0u), "r"(sel));
    return d;
}

template <int BITS, int M, int BIGBLK>
__global__ void __launch_bounds__(kDThreads, 3) lowbit_direct_kernel(const __grid_constant__ LowbitGemvArgs p) {
    constexpr int UD = BITS == 2 ? kQ2UnitDepth : kQ1UnitDepth;
    constexpr int STEPS = UD / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int kq = p.kq, q_stride = kq + 16, nb = p.nb;
    const int CPC = p.gpt;
    uint4* ring_w = reinterpret_cast<uint4*>(smem_raw) + (size_t)warp * kLbPF * 32 + lane;                  // + slot * 32
    int8_t* Qs = reinterpret_cast<int8_t*>(smem_raw + kLbRingBytes);
    float* SAs = reinterpret_cast<float*>(smem_raw + kLbRingBytes + (size_t)M * q_stride);
    int* QSs = reinterpret_cast<int*>(SAs + (size_t)M * nb);
    int* AMX = QSs + (size_t)M * nb;
    int* sums = AMX + (size_t)M * nb;
    // [ncg][nb][16] when p.dsc; 16-byte aligned for the asynchronous copies
    uint16_t* SCs = reinterpret_cast<uint16_t*>((reinterpret_cast<uintptr_t>(sums + (size_t)2 * nb * M * 16) + 15) & ~(uintptr_t)15);
    const int cg_first = (int)blockIdx.x * p.dq + min((int)blockIdx.x, p.dr);
    const int ncg = p.dq + ((int)blockIdx.x < p.dr ? 1 : 0);
    const int upw = p.dupw;
    const int u_begin = min(warp * upw, p.ku), u_end = min(u_begin + upw, p.ku);
    const int total = ncg * (u_end - u_begin);                     // units this warp walks, column group by column group
    const int block = 1 << p.log2_block;

    constexpr int PF = kLbPF;
    const unsigned char* lp = p.codes + ((size_t)cg_first * p.ku + (size_t)u_begin) * kUnitBytes + lane * 16;   // load cursor
    int lu = u_begin;
    auto issue = [&](int slot) {
        cp_async16(ring_w + slot * 32, lp);
        lp += kUnitBytes;
        if (++lu == u_end) {
            lu = u_begin;
            lp += (size_t)(p.ku - (u_end - u_begin)) * kUnitBytes;
        }
    };
    // the CTA's scale rows ride along with the first units
    if (p.dsc) {
        const uint16_t* src = p.scales + (size_t)cg_first * nb * 16;
        for (int ch = tid; ch < ncg * nb * 2; ch += kDThreads) cp_async16(SCs + ch * 8, src + (size_t)ch * 8);
    }
#pragma unroll
    for (int i = 0; i < PF; ++i) {
        if (i < total) issue(i);
        cp_async_commit();
    }
    pdl_launch_dependents();
    for (int idx = tid; idx < 2 * nb * M * 16; idx += kDThreads) sums[idx] = 0;
    for (int idx = tid; idx < M * nb; idx += kDThreads) { AMX[idx] = 0; QSs[idx] = 0; SAs[idx] = 0.0f; }
    pdl_wait();

    if (p.a != nullptr) {
        // ---- quantize_row (src/kernels/lowbit/matmul.rs:354-371) over the rows, in shared memory ----
        // An item is eight consecutive depths of one row; a thread keeps its items in registers between the
        // two passes (block maxima, then codes), QI items at a time.
        __syncthreads();
        const int nvec = kq / 8;                                   // items per row
        constexpr int QI = 4;
        // eight consecutive depths of one row as f16 bits (zero past k)
        auto load8 = [&](int r, int d) -> uint4 {
            if (p.a_vec_ok && d + 8 <= p.k) return *reinterpret_cast<const uint4*>(p.a + (size_t)r * p.k + d);
            __align__(16) uint16_t h[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) h[e] = d + e < p.k ? p.a[(size_t)r * p.k + d + e] : (uint16_t)0;
            return *reinterpret_cast<uint4*>(h);
        };
        // rows longer than QI * 256 items go in several rounds; a K-block must then lie inside one round
        // (the host only takes this path when it does)
        for (int v0 = 0; v0 < nvec; v0 += QI * kDThreads) {
#pragma unroll
            for (int r = 0; r < M; ++r) {
                uint4 hv[QI];
#pragma unroll
                for (int i = 0; i < QI; ++i) {
                    const int d = (v0 + tid + i * kDThreads) * 8;
                    hv[i] = make_uint4(0, 0, 0, 0);
                    if (d < p.k) hv[i] = load8(r, d);
                }
#pragma unroll
                for (int i = 0; i < QI; ++i) {
                    const int d = (v0 + tid + i * kDThreads) * 8;
                    const uint32_t hw[4] = {hv[i].x, hv[i].y, hv[i].z, hv[i].w};
                    int mx = 0;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        // |x| as integer bits: ordered like the values, and every NaN is above infinity (padding is 0)
                        const float2 f = __half22float2(as_h2(hw[e] & 0x7fff7fffu));
                        mx = max(mx, max(__float_as_int(f.x), __float_as_int(f.y)));
                    }
                    if (block >= 256) {
                        // a warp's 32 items are 256 consecutive depths: one K-block
                        mx = __reduce_max_sync(0xffffffffu, mx);
                        if (lane == 0 && mx != 0) atomicMax(&AMX[r * nb + (d >> p.log2_block)], mx);
                    } else if (d < p.k) {
                        atomicMax(&AMX[r * nb + (d >> p.log2_block)], mx);
                    }
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < QI; ++i) {
                    const int d = (v0 + tid + i * kDThreads) * 8;
                    if (d >= kq) continue;
                    uint32_t lo = 0, hi = 0;
                    if (d < p.k) {
                        const int bl = d >> p.log2_block;
                        const int bits = AMX[r * nb + bl];
                        const float amax = bits > 0x7f800000 ? __int_as_float(0x7fc00000) : __int_as_float(bits);
                        const float inv = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
                        if ((d & (block - 1)) == 0) {
                            const float sa = __fdiv_rn(amax, 127.0f);
                            SAs[r * nb + bl] = sa;
                            if (p.sa_out && blockIdx.x == 0) p.sa_out[(size_t)r * p.nb_real + bl] = sa;
                        }
                        const uint32_t hw[4] = {hv[i].x, hv[i].y, hv[i].z, hv[i].w};
                        int q[8];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = __half22float2(as_h2(hw[e]));
                            // round to nearest even, NaN -> 0, then saturate: round_ties_even(x) as i8 (padding is 0)
                            q[2 * e] = max(-128, min(127, __float2int_rn(__fmul_rn(f.x, inv))));
                            q[2 * e + 1] = max(-128, min(127, __float2int_rn(__fmul_rn(f.y, inv))));
                        }
                        lo = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
                        hi = __byte_perm(__byte_perm(q[4], q[5], 0x0040), __byte_perm(q[6], q[7], 0x0040), 0x5410);
                        if (BITS == 1) {
                            const int sq = __dp4a((int)lo, 0x01010101, __dp4a((int)hi, 0x01010101, 0));
                            if (sq != 0) atomicAdd(&QSs[r * nb + bl], sq);
                        }
                        if (p.q_out && blockIdx.x == 0) {
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                if (d + e < p.k) p.q_out[(size_t)r * p.k + d + e] = (int8_t)q[e];
                        }
                    }
                    *reinterpret_cast<uint2*>(Qs + (size_t)r * q_stride + d) = make_uint2(lo, hi);
                }
            }
        }
    } else {
#pragma unroll
        for (int r = 0; r < M; ++r)
            for (int v = tid; v < kq / 16; v += kDThreads)
                *reinterpret_cast<uint4*>(Qs + (size_t)r * q_stride + v * 16) = *reinterpret_cast<const uint4*>(p.q + (size_t)r * kq + v * 16);
        for (int idx = tid; idx < M * nb; idx += kDThreads) {
            SAs[idx] = p.sa[idx];
            QSs[idx] = p.qsum ? p.qsum[idx] : 0;
        }
    }
    __syncthreads();

    // ---- block sums ----
    int acc[M][2];
#pragma unroll
    for (int r = 0; r < M; ++r) acc[r][0] = acc[r][1] = 0;
    int cu = u_begin;                                              // compute cursor
    int* sb = sums;                                                // the column group's block sums
    // flush: the lanes of a column holding the same block add into one cell
    auto flush = [&](int bl) {
#pragma unroll
        for (int r = 0; r < M; ++r)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                int v = acc[r][j];
                acc[r][j] = 0;
                if (block >= 32) {
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if (t == 0 && v != 0) atomicAdd(&sb[((size_t)bl * M + r) * 16 + g + 8 * j], v);
                } else if (v != 0) {
                    atomicAdd(&sb[((size_t)bl * M + r) * 16 + g + 8 * j], v);
                }
            }
    };
    // One column group at a time: its block sums meet in one of two buffers; when every warp has added its share the
    // cells' owners fold them (and clear the buffer) while the other warps go on with the next column group.
    int slot = 0, j = 0;
    for (int c = 0; c < ncg; ++c) {
        sb = sums + (size_t)(c & 1) * nb * M * 16;
        for (cu = u_begin; cu < u_end; ++cu, ++j) {
            cp_async_wait<PF - 1>();                               // this lane's copy of unit j has landed
            const uint4 wv = ring_w[slot * 32];
            const uint32_t words[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const int d = cu * UD + 32 * s + 8 * t;            // this lane's 8 depths
                const uint32_t w = words[BITS == 2 ? s : (s >> 1)];
                uint32_t af[4];
                if (BITS == 2) {
                    const uint32_t e = w & 0x33333333u, o = (w >> 2) & 0x33333333u;
                    af[0] = prmt_lut(p.lut, e);
                    af[1] = prmt_lut(p.lut, o);
                    af[2] = prmt_lut(p.lut, e >> 16);
                    af[3] = prmt_lut(p.lut, o >> 16);
                } else {
                    const int sh = 4 * (s & 1);
                    af[0] = (w >> (sh + 0)) & 0x01010101u;
                    af[1] = (w >> (sh + 1)) & 0x01010101u;
                    af[2] = (w >> (sh + 2)) & 0x01010101u;
                    af[3] = (w >> (sh + 3)) & 0x01010101u;
                }
#pragma unroll
                for (int r = 0; r < M; ++r) {
                    const uint2 aq = *reinterpret_cast<const uint2*>(Qs + (size_t)r * q_stride + d);
                    acc[r][0] = __dp4a((int)af[0], (int)aq.x, acc[r][0]);
                    acc[r][0] = __dp4a((int)af[2], (int)aq.y, acc[r][0]);
                    acc[r][1] = __dp4a((int)af[1], (int)aq.x, acc[r][1]);
                    acc[r][1] = __dp4a((int)af[3], (int)aq.y, acc[r][1]);
                }
                // end of a K-block for this lane's depths (blocks of 16: lanes t < 2 and t >= 2 differ),
                // or of this warp's share of the column group
                if (!BIGBLK && (((d + 32) >> p.log2_block) != (d >> p.log2_block) || (s == STEPS - 1 && cu == u_end - 1))) flush(d >> p.log2_block);
            }
            // blocks of a whole unit or more: one test per unit
            if (BIGBLK && ((((cu + 1) * UD) & (block - 1)) == 0 || cu == u_end - 1)) flush((cu * UD) >> p.log2_block);
            if (j + PF < total) issue(slot);
            cp_async_commit();
            slot = slot + 1 == PF ? 0 : slot + 1;
        }
        if (c == 0) cp_async_wait<0>();                            // the staged scale rows (first group of copies) as well
        __syncthreads();
        // ---- ordered fold of the column group's cells, epilogue, store ----
        if (tid < M * 16) {
            const int col16 = tid & 15, r = tid >> 4;
            const int col = (cg_first + c) * 16 + col16;
            const uint16_t* sc = (p.dsc ? SCs + (size_t)c * nb * 16 : p.scales + ((size_t)(cg_first + c) * nb) * 16) + scale_slot(col16);
            int* cell = sb + (size_t)r * 16 + col16;
            float tot = 0.0f;
#pragma unroll 4
            for (int bl = 0; bl < p.nb_real; ++bl) {
                int sum = cell[(size_t)bl * M * 16];
                cell[(size_t)bl * M * 16] = 0;
                if (BITS == 1) sum = 2 * sum - QSs[r * nb + bl];
                if (p.sums_out && col < p.n) p.sums_out[((size_t)r * p.n + col) * p.nb_real + bl] = sum;
                const float scale = __half2float(__ushort_as_half(sc[(size_t)bl * 16]));
                tot = fmaf((float)sum, __fmul_rn(scale, SAs[r * nb + bl]), tot);
            }
            if (col < p.n) p.c[(size_t)r * p.n + col] = ep_store_value<0>(p.ep, tot, (size_t)r, (size_t)col);
        }
    }
    cp_async_wait<0>();
}

template <typename K>
cudaError_t opt_in_smem(K kern, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

// Grid of the one-wave kernels: per_sm CTAs per SM when there are that many column groups, more when a
// CTA would otherwise take more than max_groups of them; *cpc = most column groups of one CTA.
int direct_grid(int n16, int sm_count, int max_groups, int* cpc, int per_sm) {
    int grid = n16 < per_sm * sm_count ? n16 : per_sm * sm_count;
    if ((n16 + grid - 1) / grid > max_groups) grid = (n16 + max_groups - 1) / max_groups;
    if (grid < 1) grid = 1;
    *cpc = (n16 + grid - 1) / grid;
    return grid;
}

}  // namespace

// ---- Q4 ----
bool q4_direct_supported(const Q4GemvArgs& a, int bf16) {
    if (bf16 || a.m < 1 || a.m > 2 || a.log2_block < 5 || a.k64 < 1) return false;
    if (a.k % 8 != 0 || !a.a_vec_ok) return false;                // 128-bit activation loads
    const size_t smem = kQ4RingBytes + (size_t)a.m * ((size_t)a.k64 * 64 + 8) * 2;
    return smem <= 100 * 1024;
}

cudaError_t q4_direct_launch(Q4GemvArgs a, int sm_count, cudaStream_t stream) {
    const int n16 = (a.n + 15) / 16, ns = q4_stages(a.k64);
    a.n16 = n16;
    // three CTAs per SM when the matrix gives every SM that many, else two (and then never three on one SM
    // while another has one: the shared-memory request is padded past a third of an SM's)
    int per_sm = n16 > 2 * sm_count ? 3 : 2;
    int grid_x;
    auto split = [&]() {
        if (a.glu) {
            // shares are (gate group, up group) pairs: n16 / 2 of them, at most 8 (16 groups) per CTA
            const int pairs = n16 / 2;
            int cpp = 1;
            grid_x = direct_grid(pairs, sm_count, 8, &cpp, per_sm);
            a.cg = 2 * cpp;
            a.dq = pairs / grid_x; a.dr = pairs % grid_x;
        } else {
            grid_x = direct_grid(n16, sm_count, 16, &a.cg, per_sm);
            a.dq = n16 / grid_x; a.dr = n16 % grid_x;
        }
    };
    split();
    cudaError_t e;
    if (ns >= kDWarps && !a.nx) {
        // At least a stage of 256 depths for each warp.  (Shorter depths stay with the kernel below, whose warps have a unit each
        // where a stage would have one warp in work: us, this / that, 1 row: 1536 x 384 2.06 / 1.72, 4096 x 1024 2.40 / 2.06,
        // 3072 x 2048 2.57 / 2.58, 1024 x 4096 2.7 / 3.2.)
        // As many CTAs per SM as have room with three slots (of 228 KB, each with 1 KB of the system's): one more would be the half wave
        // behind (us, three or two whatever their size / this: 2 rows 28672 x 4096 18.2 / 13.4, 5120 x 5120 8.4 / 5.7, 1 row 5120 x 13824
        // 12.6 / 9.4, 28672 x 8192 26.4 / 21.5).
        // Ring: three slots where three CTAs share an SM; of two, each takes what its rows leave of half an SM, up to five.
        const size_t slot = (size_t)kDWarps * q4_slot_bytes(a.m);
        auto rest_bytes = [&]() { return q4_rows_bytes(a.m, ns) + (size_t)kDWarps * a.cg * a.m * 16 * sizeof(float); };
        while (per_sm > 1 && 3 * slot + rest_bytes() > (per_sm == 3 ? 75 : 113) * (size_t)1024) {
            --per_sm;
            split();
        }
        const size_t rest = rest_bytes();
        const int pf = per_sm > 2 ? 3 : 5 * slot + rest <= 112 * 1024 ? 5 : 4 * slot + rest <= 112 * 1024 ? 4 : 3;
        size_t bytes = pf * slot + rest;
        if (per_sm == 2 && bytes < 80 * 1024) bytes = 80 * 1024;
#define SMEG_QS(MM, PP)                                                               \
    if (a.m == MM && pf == PP) {                                                      \
        e = opt_in_smem(q4_stage_kernel<MM, PP>, bytes);                              \
        return e != cudaSuccess ? e : launch_pdl(q4_stage_kernel<MM, PP>, dim3(grid_x), dim3(kDThreads), bytes, stream, a); \
    }
        SMEG_QS(1, 3) SMEG_QS(1, 4) SMEG_QS(1, 5) SMEG_QS(2, 3) SMEG_QS(2, 4) SMEG_QS(2, 5)
#undef SMEG_QS
    }
    a.dupw = (a.k64 + kDWarps - 1) / kDWarps;
    size_t smem = kQ4RingBytes + (size_t)a.m * ((size_t)a.k64 * 64 + 8) * 2 + (size_t)kDWarps * a.cg * a.m * 16 * sizeof(float);
    if (per_sm == 2 && smem < 80 * 1024) smem = 80 * 1024;
    // A narrow layer's projections all take the form that can norm: a step through such a layer is launches of 2 us, and going
    // from one kernel's code to another's costs a fetch of it each time (six 384-wide layers 96 us a step, 111 with two kernels)
    const bool gen = a.nx || (size_t)n16 * a.k64 <= 4096;
    const dim3 grid(grid_x);
#define SMEG_QD(MM)                                                                   \
    case MM:                                                                          \
        e = gen ? opt_in_smem(q4_direct_kernel<MM, 1>, smem) : opt_in_smem(q4_direct_kernel<MM, 0>, smem); \
        if (e != cudaSuccess) return e;                                               \
        if (gen) return launch_pdl(q4_direct_kernel<MM, 1>, grid, dim3(kDThreads), smem, stream, a); \
        return launch_pdl(q4_direct_kernel<MM, 0>, grid, dim3(kDThreads), smem, stream, a);
    switch (a.m) {
        SMEG_QD(1) SMEG_QD(2)
    default: return cudaErrorInvalidValue;
    }
#undef SMEG_QD
}

// ---- 2-bit / 1-bit ----
static bool lowbit_scales_staged(const LowbitGemvArgs& a, int cpc) { return (size_t)cpc * a.nb * 32 <= 16 * 1024; }
static size_t lowbit_direct_smem(const LowbitGemvArgs& a, int cpc) {
    return kLbRingBytes + (size_t)a.m * (a.kq + 16) + (size_t)3 * a.m * a.nb * 4 + (size_t)2 * a.nb * a.m * 16 * 4 +
           (lowbit_scales_staged(a, cpc) ? (size_t)cpc * a.nb * 32 + 16 : 0);
}

bool lowbit_direct_supported(const LowbitGemvArgs& a, bool fused) {
    if (a.m < 1 || a.m > 4 || a.ku < 1 || a.k < 1) return false;
    if (a.m > 2 && a.log2_block > 4) return false;               // (lowbit_rows_kernel has room for whatever this kernel has)
    if (fused && a.m > 2) return false;                          // every CTA repeats the quantisation
    // in-kernel quantisation walks a row in rounds of 8192 depths: a K-block must lie inside one round
    if (fused && a.kq > 8192 && ((1 << a.log2_block) > 8192 || 8192 % (1 << a.log2_block) != 0)) return false;
    return lowbit_direct_smem(a, 1) <= 110 * 1024;
}

// lowbit_rows_kernel reads K-blocks above 256 twice before its products, and sixteen warps that hand parts of a depth on have little to do
// on short ones.  us, there / here: blocks of 512, 1-bit, 1 row 2048 x 512 3.3 / 2.7, 8192 x 1024 5.9 / 5.1, 1024 x 6144 2.8 / 2.6 (but 4096 x
// 4096 4.3 / 4.8), 2-bit 2 rows 512 x 256 4.0 / 3.3; blocks of 256, 2-bit, 1 row 2048 x 512 3.0 / 2.7 (3072 x 512 3.3 / 3.3), 1-bit 2 rows 1024 x 512
// 3.8 / 3.5; blocks of 128, 2-bit, 2 rows 512 x 256 3.4 / 3.1 (2048 x 512 4.1 / 4.2; 1-bit 3.3 / 4.1); blocks of 64, 2-bit, 1 row 1024 x 512 2.8 / 2.7.
bool lowbit_direct_shorter(const LowbitGemvArgs& a, int bits, int sm_count) {
    if (a.m > 2 || !lowbit_direct_supported(a, true)) return false;
    const bool one_group = a.n16 <= sm_count;                      // of columns a CTA of that kernel
    if (a.log2_block > 8) return one_group ? (size_t)a.m * a.k <= 12288 : a.n16 <= 3 * sm_count && a.k <= 4096 - 1024 * a.m;
    return one_group && a.k > 256 && (a.log2_block == 8 ? a.k <= 2048 : bits == 2 && a.log2_block >= 6 && a.k <= 1024);
}

cudaError_t lowbit_direct_launch(LowbitGemvArgs a, int bits, int sm_count, cudaStream_t stream) {
    int cpc = 1, maxg = 16;
    int grid_x = direct_grid(a.n16, sm_count, maxg, &cpc, 3);
    while (maxg > 1 && lowbit_direct_smem(a, cpc) > 110 * 1024) grid_x = direct_grid(a.n16, sm_count, --maxg, &cpc, 3);
    a.gpt = cpc;
    a.dq = a.n16 / grid_x; a.dr = a.n16 % grid_x; a.dupw = (a.ku + kDWarps - 1) / kDWarps;
    a.dsc = lowbit_scales_staged(a, cpc) ? 1 : 0;
    const size_t smem = lowbit_direct_smem(a, cpc);
    const dim3 grid(grid_x);
    cudaError_t e;
    const int ud = bits == 2 ? kQ2UnitDepth : kQ1UnitDepth;
    const bool big = (1 << a.log2_block) >= ud;
#define SMEG_LD(BB, MM, GG)                                                               \
    if (bits == BB && a.m == MM && big == (GG == 1)) {                                    \
        e = opt_in_smem(lowbit_direct_kernel<BB, MM, GG>, smem);                          \
        if (e != cudaSuccess) return e;                                                   \
        return launch_pdl(lowbit_direct_kernel<BB, MM, GG>, grid, dim3(kDThreads), smem, stream, a); \
    }
    // (three and four rows come here under K-blocks of 16 alone)
    SMEG_LD(2, 1, 0) SMEG_LD(2, 2, 0) SMEG_LD(2, 3, 0) SMEG_LD(2, 4, 0) SMEG_LD(2, 1, 1) SMEG_LD(2, 2, 1)
    SMEG_LD(1, 1, 0) SMEG_LD(1, 2, 0) SMEG_LD(1, 3, 0) SMEG_LD(1, 4, 0) SMEG_LD(1, 1, 1) SMEG_LD(1, 2, 1)
#undef SMEG_LD
    return cudaErrorInvalidValue;
}

}  // namespace smeg
