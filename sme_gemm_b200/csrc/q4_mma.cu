// Q4 GEMM for a handful of rows on warp-level tensor-core instructions, straight from global memory (sm_100a):
//   q4_mma_kernel   C[m][n] = ep( A[m][k] @ dequant(W) ), f16 or bf16, K-blocks of 32 and up
//                   DENSE: C = ep( T(beta * (A @ W)) ) on K-major 16-bit weights, whose 16-byte pieces are fragments as they lie
//
// Replaces the reference's SME Q4 GEMV (run_q4_gemv1 / run_q4_gemv, csrc/gemm_f16f16_q4.h:236-431, and the bf16 twin
// csrc/gemm_b16b16_q4.h:171-268) above the rows of gemv_direct.cu's kernels, and for bf16 from one row.
//
// Laid out like q4_direct_kernel: a packed unit (16 columns x 64 depths) is one 16-byte asynchronous copy per lane into
// the lane's own slot of a ring, a lane reads back only what it copied itself, so the loop has no barrier and no producer;
// the eight warps of a CTA split the depth.  A lane's 16 bytes are the A fragments of four mma.m16n8k16 as they lie
// (weight columns = M, activation rows = N), and its B fragments are 16-byte pieces of the activation rows, which ride in
// the same ring: nothing limits the depth, and a pass over CG column groups shares one read of them.  Codes become exact
// f16 / bf16 integers (one lop3 per pair and a subtraction), the tensor core sums 32 depths in f32 and the block's f32
// scale folds the sum into the total: no weight is rounded on the way, for bf16 either.
//
// What bounds it: instruction issue (109 warp instructions a unit at eight bf16 rows, 44 of them the expansion, issue slots 58 % busy; with the
// copies' addresses formed from indexes for each unit 135: 8 x 4096 x 14336 13.5 us, now 12.1, 16 rows 16.7 and 15.6, f16 12.0 and 11.4).
// Against the ring-staged kernel that ran these calls before (us): bf16 8 x 4096 x 14336 28.0 -> 12.1 (2.8 TB/s), 16 rows 67 -> 15.6; bf16 4096 x 4096 1 row 15.8 -> 4.9, 16 rows 28.5 -> 6.3; f16 8 rows 9.8 -> 4.6, 16 rows 14.0 -> 6.2; against
// q4_direct_kernel at 4 rows 8.5 -> 4.5 (one and two rows stay with the kernels of gemv_direct.cu: 3.4 and 4.1).
#include <atomic>

#include "epilogue.cuh"
#include "kernels.h"
#include "layout.h"

namespace smeg {
namespace {

constexpr int kMWarps = 8;
constexpr int kMThreads = 32 * kMWarps;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// `bytes` bytes (0 to 16) and zeros behind them: nothing past them is read
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

template <int BF16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
    if (BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// One packed word (8 nibbles, offset binary) -> the four A registers: a[0] = column g (d, d+1), a[1] = column g+8 (d, d+1),
// a[2] = column g (d+2, d+3), a[3] = column g+8 (d+2, d+3), exact integers in T.
template <int BF16>
__device__ __forceinline__ void word_codes(uint32_t w, uint32_t (&a)[4]) {
    if (BF16) {
        // 128 + u is a bf16 number whose last place is 1
        const uint32_t x[4] = {w, w >> 8, w >> 4, w >> 12};
        const __nv_bfloat162 off = __halves2bfloat162(__ushort_as_bfloat16(0x4308), __ushort_as_bfloat16(0x4308));   // 136
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t v = lop3_and_or(x[i], 0x000f000fu, 0x43004300u);
            const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v), off);
            a[i] = *reinterpret_cast<const uint32_t*>(&r);
        }
        return;
    }
    const uint32_t w8 = w >> 8;
    const uint32_t lo0 = lop3_and_or(w, 0x000f000fu, 0x64006400u), hi0 = lop3_and_or(w, 0x00f000f0u, 0x64006400u);
    const uint32_t lo1 = lop3_and_or(w8, 0x000f000fu, 0x64006400u), hi1 = lop3_and_or(w8, 0x00f000f0u, 0x64006400u);
    const __half2 off = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x6408));      // 1032
    const __half2 sc16 = __halves2half2(__ushort_as_half(0x2c00), __ushort_as_half(0x2c00));     // 1/16
    const __half2 off16 = __halves2half2(__ushort_as_half(0xd480), __ushort_as_half(0xd480));    // -72
    const __half2 r0 = __hsub2(*reinterpret_cast<const __half2*>(&lo0), off), r1 = __hsub2(*reinterpret_cast<const __half2*>(&lo1), off);
    const __half2 r2 = __hfma2(*reinterpret_cast<const __half2*>(&hi0), sc16, off16), r3 = __hfma2(*reinterpret_cast<const __half2*>(&hi1), sc16, off16);
    a[0] = *reinterpret_cast<const uint32_t*>(&r0); a[1] = *reinterpret_cast<const uint32_t*>(&r1);
    a[2] = *reinterpret_cast<const uint32_t*>(&r2); a[3] = *reinterpret_cast<const uint32_t*>(&r3);
}

// Ring slot of a warp: [CG] codes (dense: [CG][column g, g + 8][2 halves] pieces of weights), [2 NT] activation pieces (none where
// the rows are staged, rows = 0), 16 bytes a lane each, then [CG][2 halves] scale words.
constexpr int mma_w_bytes(int dense) { return dense ? 2048 : 512; }
constexpr int mma_slot_bytes(int rows, int cg, int dense) { return mma_w_bytes(dense) * cg + 1024 * rows + (dense ? 0 : 256 * cg); }
// As deep as two CTAs per SM leave room for.
constexpr int mma_ring_slots(int nt, int cg, int dense) { return dense ? (nt == 1 ? 4 : 3) : (nt == 1 ? (cg == 1 ? 6 : 4) : (cg == 1 ? 4 : 3)); }
constexpr size_t mma_smem(int nt, int cg, int dense, int staged) {
    return (size_t)kMWarps * mma_ring_slots(nt, cg, dense) * mma_slot_bytes(staged ? 0 : nt, cg, dense) + (size_t)kMWarps * cg * nt * 512;
}
constexpr size_t kMmaStagedMost = 56 * 1024;
inline size_t mma_staged_bytes(int m, int k64) { return (size_t)m * ((size_t)k64 * 64 + 8) * 2; }

// A row to shared memory (16-byte aligned) in pieces as wide as its start allows, eight on their way a thread, and zeros behind
// it up to kpad.
template <typename T>
__device__ __forceinline__ int stage_pieces(uint16_t* dst, const uint16_t* src, int k) {
    constexpr int per = sizeof(T) / 2;
    const int n = k / per;
    for (int d0 = threadIdx.x; d0 < n; d0 += kMThreads * 8) {
        T v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (d0 + e * kMThreads < n) v[e] = reinterpret_cast<const T*>(src)[d0 + e * kMThreads];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (d0 + e * kMThreads < n) reinterpret_cast<T*>(dst)[d0 + e * kMThreads] = v[e];
    }
    return n * per;
}
__device__ __noinline__ void stage_row(uint16_t* dst, const uint16_t* src, int k, int kpad) {
    const unsigned at = (unsigned)(uintptr_t)src;
    const int done = (at & 15) == 0 ? stage_pieces<uint4>(dst, src, k) : (at & 7) == 0 ? stage_pieces<uint2>(dst, src, k)
                     : (at & 3) == 0 ? stage_pieces<uint32_t>(dst, src, k) : stage_pieces<uint16_t>(dst, src, k);
    for (int d = done + (int)threadIdx.x; d < kpad; d += kMThreads) dst[d] = d < k ? src[d] : (uint16_t)0;
}

// NT = tiles of eight rows per CTA, CG = column groups of a pass.  Grid: (CTAs over the passes, row tiles of 8 NT).  STAGED: a few
// rows that are no whole 16-byte words, copied to shared memory by every CTA instead of a padded copy in
// front of the call (us on the device, with the copy / staged: 5001 x 4097 1 row 8.8 / 6.9, 2 rows 8.7 / 7.8, 4096 x 8190 2 rows
// 9.7 / 8.8, 14336 x 4092 15.2 / 13.5; a pass from the host, 2051 x 1500 2 rows, 8.7 / 5.3; 700 x 8191 at 3 rows 6.6 / 7.1).
template <int BF16, int NT, int CG, int DENSE, int STAGED>
__global__ void __launch_bounds__(kMThreads, 2) q4_mma_kernel(const __grid_constant__ Q4GemvArgs p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int PF = mma_ring_slots(NT, CG, DENSE), RB = STAGED ? 0 : 1024 * NT, SLOT = mma_slot_bytes(STAGED ? 0 : NT, CG, DENSE);
    constexpr int WB = mma_w_bytes(DENSE), PER = CG * NT * 128;
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t ring = smem_u32(smem_raw) + (uint32_t)(warp * PF * SLOT);
    float* red = reinterpret_cast<float*>(smem_raw + (size_t)kMWarps * PF * SLOT);       // [8 warps][CG][NT][4][32 lanes]
    uint16_t* rows_s = reinterpret_cast<uint16_t*>(red + kMWarps * PER);                 // STAGED: [m][k64 * 64 + 8]
    const int rows_ld = p.k64 * 64 + 8;
    // this CTA's passes: an equal share of all of them
    const int first = (int)blockIdx.x * p.dq + min((int)blockIdx.x, p.dr);
    const int passes = p.dq + ((int)blockIdx.x < p.dr ? 1 : 0);
    const int row0 = (int)blockIdx.y * 8 * NT;
    // column group c of a pass (gated form: a gate group 4q + e and its up group 4q + 2 + e)
    auto group_of = [&](int pass, int c) -> int {
        if (CG == 2 && p.glu) return 4 * (pass >> 1) + (pass & 1) + 2 * c;
        return CG * pass + c;
    };
    const int upw = p.dupw;                                        // units per warp: a contiguous run of the depth
    const int u_begin = min(warp * upw, p.k64), u_end = min(u_begin + upw, p.k64), nu = u_end - u_begin;
    const int total = passes * nu;

    // load cursor: where the unit's codes and scales (dense: pieces of weights) and its rows start, as pointers that a unit moves on.
    // (Formed from the indexes for each unit they were a third of the loop's instructions.)
    int lu = u_begin, lpass = first;
    // (Dense weights and passes of one column group on sixteen rows keep the indexes: 64 x 2048 x 2048 dense with pointers 7.0 us, without
    // 6.84, 16 x 4096 x 4096 6.13 and 5.99.)
    constexpr bool PTR = !DENSE && !(NT == 2 && CG == 1);
    const unsigned char *wp[CG], *sp[CG];
    const uint32_t sc_shift = DENSE ? 0u : (uint32_t)p.log2_block - 5;
    auto weights_from = [&](int pass) {
        if (!PTR) return;
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            const uint32_t grp = (uint32_t)min(group_of(pass, c), p.n16 - 1);           // a tail pass may be one group short
            wp[c] = p.codes + (uint64_t)grp * (uint32_t)(p.k64 * kUnitBytes) + (uint32_t)(u_begin * kUnitBytes + lane * 16);
            sp[c] = reinterpret_cast<const unsigned char*>(p.scales) + (uint64_t)grp * (uint32_t)(p.nb * 32) + (uint32_t)(4 * g);
        }
    };
    auto issue_weights = [&](uint32_t slot, int u) {
        if (DENSE) {
            const int d = u * 64 + 8 * t;                          // (kd is a multiple of 8; columns past n and depths past kd are zeros)
#pragma unroll
            for (int c = 0; c < CG; ++c)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int col = group_of(lpass, c) * 16 + g + 8 * j;
                    const uint16_t* src = p.wdense + (size_t)min(col, p.n - 1) * p.kd + d;
                    const uint32_t lo = col < p.n && d < p.kd ? 16u : 0u, hi = col < p.n && d + 32 < p.kd ? 16u : 0u;
                    const uint32_t dst = slot + (uint32_t)(WB * c + 1024 * j + lane * 16);
                    cp_async16_zfill(dst, lo ? src : p.wdense, lo);
                    cp_async16_zfill(dst + 512, hi ? src + 32 : p.wdense, hi);
                }
            return;
        }
        if (!PTR) {
#pragma unroll
            for (int c = 0; c < CG; ++c) {
                const size_t grp = (size_t)min(group_of(lpass, c), p.n16 - 1);
                cp_async16(slot + (uint32_t)(512 * c + lane * 16), p.codes + q4_unit_offset(grp, (size_t)u, p.k64) + lane * 16);
                const uint16_t* s = p.scales + q4_scale_row(grp, 0, p.nb) + 2 * g;
                const uint32_t d = slot + (uint32_t)(512 * CG + RB + 256 * c + lane * 4);
                cp_async4(d, s + (size_t)((u * 64) >> p.log2_block) * 16);
                cp_async4(d + 128, s + (size_t)((u * 64 + 32) >> p.log2_block) * 16);
            }
            return;
        }
        const uint32_t ra = ((uint32_t)(2 * u) >> sc_shift) * 32, rb = ((uint32_t)(2 * u + 1) >> sc_shift) * 32;
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            cp_async16(slot + (uint32_t)(512 * c + lane * 16), wp[c]);
            wp[c] += kUnitBytes;
            const uint32_t d = slot + (uint32_t)(512 * CG + RB + 256 * c + lane * 4);
            cp_async4(d, sp[c] + ra);
            cp_async4(d + 128, sp[c] + rb);
        }
    };
    const uint16_t* arow[NT];
    int kend[NT];
    uint32_t a_sz[NT];                                             // rows past the batch are zeros, without a read
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        arow[nt] = p.a + (size_t)min(row0 + 8 * nt + g, p.m - 1) * p.k + (PTR ? u_begin * 64 : 0) + 8 * t;
        a_sz[nt] = row0 + 8 * nt + g < p.m ? 16u : 0u;
        kend[nt] = row0 + 8 * nt + g < p.m ? p.k : 0;
    }
    const int whole = p.k >> 6;                                    // units without a depth past the rows' end
    auto issue_rows = [&](uint32_t slot, int u) {
        if (STAGED) return;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const uint32_t dst = slot + (uint32_t)(WB * CG + 1024 * nt + lane * 16);
            if (!PTR) {
                const int d = u * 64;
                const uint32_t lo = d + 8 * t < kend[nt] ? 16u : 0u, hi = d + 32 + 8 * t < kend[nt] ? 16u : 0u;   // k is a multiple of 8
                cp_async16_zfill(dst, lo ? arow[nt] + d : p.a, lo);
                cp_async16_zfill(dst + 512, hi ? arow[nt] + d + 32 : p.a, hi);
                continue;
            }
            if (u < whole) {                                       // (a size of zero reads nothing)
                cp_async16_zfill(dst, arow[nt], a_sz[nt]);
                cp_async16_zfill(dst + 512, arow[nt] + 32, a_sz[nt]);
            } else {
                const uint32_t lo = u * 64 + 8 * t < p.k ? a_sz[nt] : 0u, hi = u * 64 + 32 + 8 * t < p.k ? a_sz[nt] : 0u;   // k is a multiple of 8
                cp_async16_zfill(dst, lo ? arow[nt] : p.a, lo);
                cp_async16_zfill(dst + 512, hi ? arow[nt] + 32 : p.a, hi);
            }
            arow[nt] += 64;
        }
    };
    auto rows_back = [&]() {
        if (!PTR) return;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) arow[nt] -= (size_t)nu * 64;
    };
    // the weights of the first ring-full do not depend on the kernel ahead in the stream; the activations may
    if (total > 0) weights_from(first);
    {
        const int ahead = total < PF - 1 ? total : PF - 1;
        for (int i = 0; i < ahead; ++i) {
            issue_weights(ring + (uint32_t)(i * SLOT), lu);
            if (++lu == u_end) {
                lu = u_begin;
                if (++lpass < first + passes) weights_from(lpass);
            }
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    {
        int ru = u_begin;
#pragma unroll
        for (int i = 0; i < PF - 1; ++i) {
            if (i < total) {
                issue_rows(ring + (uint32_t)(i * SLOT), ru);
                if (++ru == u_end) { ru = u_begin; rows_back(); }
            }
            cp_async_commit();
        }
    }
    if (STAGED) {
        for (int r = 0; r < p.m; ++r) stage_row(rows_s + (size_t)r * rows_ld, p.a + (size_t)r * p.k, p.k, p.k64 * 64);
        __syncthreads();
    }

    float tot[CG][NT][4];
#pragma unroll
    for (int c = 0; c < CG; ++c)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) tot[c][nt][r] = 0.0f;
    const float zero4[4] = {0.f, 0.f, 0.f, 0.f};
    int slot = 0;
    for (int ps = 0; ps < passes; ++ps) {
        for (int u = 0; u < nu; ++u) {
            cp_async_wait<PF - 2>();                               // this lane's copies of the unit have landed
            const uint32_t sb = ring + (uint32_t)(slot * SLOT);
            uint4 alo[NT], ahi[NT];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                if (STAGED) {
                    const uint16_t* ar = rows_s + (size_t)min(g, p.m - 1) * rows_ld + (u_begin + u) * 64 + 8 * t;
                    alo[nt] = g < p.m ? *reinterpret_cast<const uint4*>(ar) : make_uint4(0, 0, 0, 0);
                    ahi[nt] = g < p.m ? *reinterpret_cast<const uint4*>(ar + 32) : make_uint4(0, 0, 0, 0);
                    continue;
                }
                alo[nt] = lds128(sb + (uint32_t)(WB * CG + 1024 * nt + lane * 16));
                ahi[nt] = lds128(sb + (uint32_t)(WB * CG + 1024 * nt + 512 + lane * 16));
            }
            uint4 wv[CG][DENSE ? 4 : 1];                           // dense: column g low, high half, column g + 8 low, high
            uint32_t sw[CG][2];
#pragma unroll
            for (int c = 0; c < CG; ++c) {
#pragma unroll
                for (int j = 0; j < (DENSE ? 4 : 1); ++j) wv[c][j] = lds128(sb + (uint32_t)(WB * c + 512 * j + lane * 16));
                if (!DENSE) {
                    sw[c][0] = lds32(sb + (uint32_t)(512 * CG + RB + 256 * c + lane * 4));
                    sw[c][1] = lds32(sb + (uint32_t)(512 * CG + RB + 256 * c + 128 + lane * 4));
                }
            }
            // the slot read in the step before is free: the unit PF - 1 steps on goes there
            const int fill = slot == 0 ? PF - 1 : slot - 1;
            if (lpass < first + passes) {
                const uint32_t fb = ring + (uint32_t)(fill * SLOT);
                issue_weights(fb, lu);
                issue_rows(fb, lu);
                if (++lu == u_end) {
                    lu = u_begin;
                    rows_back();
                    if (++lpass < first + passes) weights_from(lpass);
                }
            }
            cp_async_commit();
            slot = slot + 1 == PF ? 0 : slot + 1;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < CG; ++c) {
                    if constexpr (DENSE) {
                        const uint4 lo = wv[c][h], hi = wv[c][2 + h];
                        const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            const uint4& av = h ? ahi[nt] : alo[nt];
                            mma16816<BF16>(tot[c][nt], a0, av.x, av.y, tot[c][nt]);
                            mma16816<BF16>(tot[c][nt], a1, av.z, av.w, tot[c][nt]);
                        }
                        continue;
                    }
                    uint32_t af0[4], af1[4];
                    word_codes<BF16>(h ? wv[c][0].z : wv[c][0].x, af0);
                    word_codes<BF16>(h ? wv[c][0].w : wv[c][0].y, af1);
                    const float2 sf = __half22float2(*reinterpret_cast<const __half2*>(&sw[c][h]));   // columns g, g + 8
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const uint4& av = h ? ahi[nt] : alo[nt];
                        float part[4];
                        mma16816<BF16>(part, af0, av.x, av.y, zero4);
                        mma16816<BF16>(part, af1, av.z, av.w, part);
                        tot[c][nt][0] = fmaf(part[0], sf.x, tot[c][nt][0]);
                        tot[c][nt][1] = fmaf(part[1], sf.x, tot[c][nt][1]);
                        tot[c][nt][2] = fmaf(part[2], sf.y, tot[c][nt][2]);
                        tot[c][nt][3] = fmaf(part[3], sf.y, tot[c][nt][3]);
                    }
                }
        }
        // ---- the warps' shares of the pass in warp order, epilogue, store ----
        float* rb = red;
        if (ps) __syncthreads();                                   // the pass before has been read
#pragma unroll
        for (int c = 0; c < CG; ++c)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    rb[warp * PER + ((c * NT + nt) * 4 + r) * 32 + lane] = tot[c][nt][r];
                    tot[c][nt][r] = 0.0f;
                }
        __syncthreads();
        const int pass = first + ps;
        if (CG == 2 && p.glu) {
            // out = f16(act(f16(gate)) * f16(up)), the arithmetic of the separate gate pass on the rounded projections
            const int hn = p.n >> 1;
            for (int o = tid; o < NT * 128; o += kMThreads) {
                float ag = 0.0f, au = 0.0f;
#pragma unroll
                for (int w = 0; w < kMWarps; ++w) {
                    ag += rb[w * PER + o];
                    au += rb[w * PER + NT * 128 + o];
                }
                const int ln = o & 31, r = (o >> 5) & 3, nt = o >> 7;
                const int hcol = pass * 16 + (ln >> 2) + 8 * (r >> 1), row = row0 + 8 * nt + 2 * (ln & 3) + (r & 1);
                const float gv = t_to_f32<BF16>(f32_to_t<BF16>(ag)), uv = t_to_f32<BF16>(f32_to_t<BF16>(au));
                if (hcol < hn && row < p.m) p.c[(size_t)row * hn + hcol] = f32_to_t<BF16>(__fmul_rn(glu_gate((uint32_t)p.glu, gv), uv));
            }
            continue;
        }
        for (int o = tid; o < PER; o += kMThreads) {
            float acc = 0.0f;
#pragma unroll
            for (int w = 0; w < kMWarps; ++w) acc += rb[w * PER + o];
            const int ln = o & 31, r = (o >> 5) & 3, nt = (o >> 7) % NT, c = o / (128 * NT);
            const int col = (CG * pass + c) * 16 + (ln >> 2) + 8 * (r >> 1), row = row0 + 8 * nt + 2 * (ln & 3) + (r & 1);
            if (col < p.n && row < p.m) {
                if (DENSE) {
                    if (p.beta != 1.0f) acc = __fmul_rn(p.beta, acc);
                    p.c[p.col_major ? (size_t)col * p.m + row : (size_t)row * p.n + col] = ep_store_value<BF16>(p.ep, acc, (size_t)row, (size_t)col);
                } else if (p.c32) p.c32[(size_t)row * p.n + col] = acc;
                else if (p.yacc) p.yacc[(size_t)row * p.n + col] = __fadd_rn(p.yacc[(size_t)row * p.n + col], t_to_f32<BF16>(f32_to_t<BF16>(acc)));
                else p.c[(size_t)row * p.n + col] = ep_store_value<BF16>(p.ep, acc, (size_t)row, (size_t)col);
            }
        }
    }
    cp_async_wait<0>();
}

template <int BF16, int NT, int CG, int DENSE, int STAGED = 0>
cudaError_t launch(const Q4GemvArgs& a, dim3 grid, cudaStream_t stream) {
    static std::atomic<int> attr_dev{-1};   // the opt-in is per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev.load(std::memory_order_acquire) != dev) {
        const cudaError_t e = cudaFuncSetAttribute(q4_mma_kernel<BF16, NT, CG, DENSE, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(mma_smem(NT, CG, DENSE, STAGED) + (STAGED ? kMmaStagedMost : 0)));
        if (e != cudaSuccess) return e;
        attr_dev.store(dev, std::memory_order_release);
    }
    const size_t smem = mma_smem(NT, CG, DENSE, STAGED) + (STAGED ? mma_staged_bytes(a.m, a.k64) : 0);
    return launch_pdl(q4_mma_kernel<BF16, NT, CG, DENSE, STAGED>, grid, dim3(kMThreads), smem, stream, a);
}

}  // namespace

// Rows that are no whole 16-byte words are taken up to two at a time, while they fit beside two CTAs' rings.
bool q4_mma_supported(const Q4GemvArgs& a) {
    return a.m >= 1 && a.log2_block >= 5 && a.k64 >= 1 && (a.a_vec_ok || (a.m <= 2 && mma_staged_bytes(a.m, a.k64) <= kMmaStagedMost));
}

cudaError_t q4_mma_launch(Q4GemvArgs a, int bf16, int sm_count, cudaStream_t stream) {
    const int n16 = (a.n + 15) / 16;
    const int nt = a.m <= 8 ? 1 : 2;                               // (32 rows per CTA leave room for one CTA per SM: 17 rows of 4096 x 4096 15 us against 12)
    const int ytiles = (a.m + 8 * nt - 1) / (8 * nt);
    // One wave of CTAs.  Passes of two column groups share the reads of the activations; where that leaves CTA slots idle
    // (under 4 groups per SM) a pass is one group and twice as many CTAs run.
    const int cg = a.wdense ? 1 : a.glu || (long long)n16 * ytiles > 4ll * sm_count ? 2 : 1;
    const int passes = (n16 + cg - 1) / cg;                         // (gated form: n is a multiple of 64)
    const int ctas = 2 * sm_count / ytiles, slots = ctas > 0 ? ctas : 1;
    const int grid_x = passes < slots ? passes : slots;
    a.n16 = n16;
    a.dq = passes / grid_x; a.dr = passes % grid_x;
    a.dupw = (a.k64 + kMWarps - 1) / kMWarps;
    const dim3 grid(grid_x, ytiles);
    if (a.wdense) {
        if (bf16) return nt == 1 ? launch<1, 1, 1, 1>(a, grid, stream) : launch<1, 2, 1, 1>(a, grid, stream);
        return nt == 1 ? launch<0, 1, 1, 1>(a, grid, stream) : launch<0, 2, 1, 1>(a, grid, stream);
    }
    if (!a.a_vec_ok) {
        if (bf16) return cg == 2 ? launch<1, 1, 2, 0, 1>(a, grid, stream) : launch<1, 1, 1, 0, 1>(a, grid, stream);
        return cg == 2 ? launch<0, 1, 2, 0, 1>(a, grid, stream) : launch<0, 1, 1, 0, 1>(a, grid, stream);
    }
#define SMEG_QM(B, T)                                                                          \
    if (bf16 == B && nt == T) return cg == 2 ? launch<B, T, 2, 0>(a, grid, stream) : launch<B, T, 1, 0>(a, grid, stream);
    SMEG_QM(0, 1) SMEG_QM(0, 2)
    SMEG_QM(1, 1) SMEG_QM(1, 2)
#undef SMEG_QM
    return cudaErrorInvalidValue;
}

}  // namespace smeg
