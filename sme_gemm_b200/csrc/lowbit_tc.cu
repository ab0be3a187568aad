// 2-bit / 1-bit weights x int8-quantised activations on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory): matmul_q2 / matmul_q1 above a handful of rows, up to
// prefill-sized batches.
//
// Replaces the reference's SME kernel for these batch sizes (q2_core / run_q2_gemv / Q2_FOLD,
// csrc/gemm_q2.cc:180-204,300-404, which walks the rows in groups of five) and reproduces the bits
// of its portable statement (reference, src/kernels/lowbit/matmul.rs:376-398): every K-block's sum
// is an exact int32, and an output cell folds its blocks in K order with
// total = fmaf((float)sum, scale * sa, total).
//
// The block sums are integer dot products, formed EXACTLY on the f16 tensor-core path: the int8
// activation codes travel as f16 integers (act_quant_kernel writes them so), a weight travels as
// the f16 whose bit pattern is a small unsigned integer u (u * 2^-24: the sign bit itself for
// 1-bit weights, codebook value + 128 for 2-bit ones), products of such numbers are exact, and an
// f32 accumulator holds their sum exactly while it stays below 2^24 units -- which a run of at
// most 256 depths guarantees (255 * 128 * 256 < 2^24).  A K-block longer than that is accumulated
// in runs of 256 depths whose integer sums are added in the fold.  (tcgen05.mma.kind::i8 gives the
// same integers, and an earlier form of this kernel used it, but in it tcgen05's int8 kind
// sustained only ~135 TOP/s against ~1500 TFLOP/s for f16.)  The 1-bit form does not even move
// its sign bits: bit b of a half word is the f16 number 2^(b-24) for b < 12, so an operand register
// is the packed word under one mask, and act_quant_kernel leaves the codes of the matching depths
// in the matching order, scaled by the inverse power of two (2^8, 1, 2^6, 2^-2: still exact f16
// numbers); the sums of a lane's two columns then carry 2^-16 and 2^-15, which the fold undoes.
//
// One CTA owns 128 weight columns (the MMA's M dimension) x a tile of up to 128 activation rows (the
// MMA's N dimension) over the whole depth, walked in 64-deep stages.  Roles (640 threads):
//   warp 16 (rows)      one TMA tile load per stage of the activation codes (tensor map, 128-byte
//                       swizzle, rows past m read as zero).
//   warp 18 (weights)   the packed units of the CTA's 8 column groups, 512 depths per bulk copy.
//   warps 0-7 (expand)  four pairs taking the stages in turn, a warp four column groups of its
//                       stage: 2-bit codes through a byte-permute lookup of the offset codebook,
//                       sign bits as they are, widened to 16 bits and written as the K-major,
//                       128-byte-swizzled operand.
//   warp 17 (MMA)       one elected thread issues the stage's four K = 16 instructions.  A run's
//                       steps accumulate into one of a ring of accumulators in tensor memory
//                       (512 columns / row tile); the run's last step commits it to the fold warps.
//   warp 19 (scales)    per K-block the operands of the fold -- the rows' activation scales and code
//                       sums, the column groups' scale rows -- into a small ring, so that no fold
//                       warp ever waits for a global load.
//   warps 8-15 (fold)   thread = weight column: read a finished run per row (tcgen05.ld), release
//                       the accumulator, and at the end of a K-block fold the block's integer into
//                       the running f32 total with the block's scale; after the last block the
//                       epilogue graph runs on the f16-rounded product and C is stored.
// K-blocks of one run take lowbit_tc_block_kernel, further down.
// Every wait is bounded; a timed-out wait raises the status word and the kernel drains and exits.
#include <atomic>

#include "epilogue.cuh"
#include "kernels.h"
#include "layout.h"
#include "tc_common.cuh"

#include <type_traits>

namespace smeg {
namespace {

constexpr int kLtThreads = 32 * 20;
constexpr int kLtStage = 64;                     // depths per stage (one 128-byte swizzle row of f16)
constexpr int kLtATile = 128 * 128;              // expanded weights of a stage: 16 KB
constexpr int kLtNA = 6, kLtNB = 6, kLtNK = 3;   // ring depths: operand, rows, packed
constexpr int kLtSlotStages = 8;                 // stages of one packed-ring slot (512 depths)
constexpr int kLtNF = 8;                         // ring depth of the fold operands (K-blocks)
constexpr int kLtRun = 256;                      // most depths summed in one accumulator

__device__ __forceinline__ uint32_t prmt2(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// Four bytes -> four 16-bit values with zero high bytes (f16 bit patterns u * 2^-24).
__device__ __forceinline__ uint2 widen4(uint32_t v) { return make_uint2(prmt2(v, 0u, 0x4140u), prmt2(v, 0u, 0x4342u)); }
// TPW = rows one fold warp takes (16 or 32), DW = fold warps per lane quarter (1 or 2): the row
// tile of a CTA is TPW * DW rows.
// The general form: K-blocks of several runs (more than 256 depths), and the debug output of the block sums.
template <int BITS, int TPW, int DW>
__global__ void __launch_bounds__(kLtThreads, 1) lowbit_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ LowbitTcArgs p) {
    constexpr int NT = TPW * DW;                               // rows per CTA tile
    constexpr int ACC_STRIDE = NT < 32 ? 32 : NT;              // tensor-memory columns between accumulators
    constexpr int NACC = 512 / ACC_STRIDE;
    constexpr int NA = kLtNA, NB = kLtNB;                      // ring depths: operand, rows
    constexpr int UPS = BITS == 2 ? 4 : 2;                     // packed units per slot and column group (512 depths)
    constexpr int SPU = BITS == 2 ? 2 : 4;                     // stages per unit
    constexpr int KSLOT = 8 * UPS * kUnitBytes;                // bytes of a packed slot
    constexpr int BTILE = NT * 128;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem_raw = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;

    unsigned char* ring_a = smem_raw;                                          // [NA][16 KB]
    unsigned char* ring_b = ring_a + (size_t)NA * kLtATile;                 // [NB][BTILE], tiles 1024-byte aligned
    constexpr int BSLOT = (BTILE + 1023) / 1024 * 1024;
    unsigned char* ring_k = ring_b + (size_t)NB * BSLOT;                    // [NK][KSLOT]
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring_k + (size_t)kLtNK * KSLOT);
    uint64_t* a_full = bars;                      // [NA] operand written (the stage's two expand warps)
    uint64_t* a_empty = a_full + NA;           // [NA] the stage's MMAs retired
    uint64_t* b_full = a_empty + NA;           // [NB] row tile landed
    uint64_t* b_empty = b_full + NB;           // [NB] the stage's MMAs retired
    uint64_t* k_full = b_empty + NB;           // [NK] packed units landed
    uint64_t* k_empty = k_full + kLtNK;           // [NK] every stage of the slot has been expanded
    uint64_t* acc_full = k_empty + kLtNK;         // [NACC] a K-block's sums are complete
    uint64_t* acc_empty = acc_full + NACC;        // [NACC] ... and read by every fold warp
    uint64_t* f_full = acc_empty + NACC;          // [NF] fold operands of a K-block landed
    uint64_t* f_empty = f_full + kLtNF;           // [NF] ... and read by every fold warp
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(f_empty + kLtNF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    // fold-operand ring: per K-block [NT f32 activation scales][NT i32 code sums][8 column groups x 16 f16 scales]
    constexpr int FSLOT = NT * 8 + 256;
    unsigned char* ring_f = reinterpret_cast<unsigned char*>(bars) + 1024;

    const int col0 = blockIdx.x * 128, cg0 = blockIdx.x * 8;
    const int tok0 = blockIdx.y * NT;
    const int block = 1 << p.log2_block;
    const int log2_run = min(p.log2_block, 8);                 // an accumulator sums a run of min(block, 256) depths
    const int run = 1 << log2_run;
    // depths that belong to a real K-block and are staged (>= k: what lies past k multiplies zero activations)
    const int k_end = (int)min((long long)p.nb_real << p.log2_block, (long long)p.kq);
    const int stages = (k_end + kLtStage - 1) / kLtStage;
    const int slots = (stages + kLtSlotStages - 1) / kLtSlotStages;

    if (tid == 0) {
        for (int s = 0; s < NA; ++s) { mbar_init(&a_full[s], 2); mbar_init(&a_empty[s], 1); }
        for (int s = 0; s < NB; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
        for (int s = 0; s < kLtNK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 2 * kLtSlotStages); }
        for (int s = 0; s < NACC; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4 * DW); }
        for (int s = 0; s < kLtNF; ++s) { mbar_init(&f_full[s], 1); mbar_init(&f_empty[s], 4 * DW); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 17) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    if (warp == 16 && lane == 0) tma_prefetch_desc(&tmap_q);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 16) {
        // ===================== row producer =====================
        if (lane == 0) {
            for (int i = 0; i < stages; ++i) {
                const int slot = i % NB;
                if (i >= NB && !mbar_wait_poll(&b_empty[slot], ((i / NB) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT)) break;
                mbar_expect_tx(&b_full[slot], (unsigned)BTILE);
                tma_load_2d(ring_b + (size_t)slot * BSLOT, &tmap_q, i * kLtStage, tok0, &b_full[slot]);   // x in f16 elements
            }
        }
    } else if (warp == 18) {
        // ===================== packed-weight producer: lane c = column group c of the CTA =====================
        for (int gq = 0; gq < slots; ++gq) {
            const int slot = gq % kLtNK;
            if (gq >= kLtNK && !__all_sync(0xffffffffu, mbar_wait_poll(&k_empty[slot], ((gq / kLtNK) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            const int u0 = gq * UPS;
            const int units = min(UPS, p.ku - u0);
            if (lane == 0) mbar_expect_tx(&k_full[slot], (unsigned)(8 * units * kUnitBytes));
            __syncwarp();
            if (lane < 8) {
                const size_t cgi = (size_t)min(cg0 + lane, p.n16 - 1);         // a tail group re-reads the last one
                bulk_g2s(ring_k + (size_t)slot * KSLOT + (size_t)lane * UPS * kUnitBytes,
                         p.codes + (cgi * p.ku + (size_t)u0) * kUnitBytes, units * kUnitBytes, &k_full[slot]);
            }
            __syncwarp();
        }
    } else if (warp == 19) {
        // ===================== fold-operand producer: lane 0 the rows' scales, lane 1 their code sums, lanes 2-9 a column group's scale row =====================
        for (int blk = 0; blk < p.nb_real; ++blk) {
            const int fs = blk % kLtNF;
            if (blk >= kLtNF && !__all_sync(0xffffffffu, mbar_wait_poll(&f_empty[fs], ((blk / kLtNF) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            unsigned char* dst = ring_f + (size_t)fs * FSLOT;
            if (lane == 0) mbar_expect_tx(&f_full[fs], (unsigned)(NT * 8 + 8 * 32));
            __syncwarp();
            if (lane == 0) bulk_g2s(dst, p.sa_t + (size_t)blk * p.mpad + tok0, NT * 4, &f_full[fs]);
            else if (lane == 1) bulk_g2s(dst + NT * 4, p.qsum_t + (size_t)blk * p.mpad + tok0, NT * 4, &f_full[fs]);
            else if (lane >= 2 && lane < 10) {
                const size_t cgi = (size_t)min(cg0 + lane - 2, p.n16 - 1);
                bulk_g2s(dst + NT * 8 + (lane - 2) * 32, p.scales + (cgi * p.nb + (size_t)blk) * 16, 32, &f_full[fs]);
            }
            __syncwarp();
        }
    } else if (warp == 17) {
        // ===================== MMA issuer =====================
        const uint32_t idesc = umma_idesc(0, 128, NT);
        for (int i = 0; i < stages; ++i) {
            const int as = i % NA, bs = i % NB;
            if (!__all_sync(0xffffffffu, mbar_wait_poll(&b_full[bs], (i / NB) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            if (!__all_sync(0xffffffffu, mbar_wait_poll(&a_full[as], (i / NA) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            tc_fence_after();
            const uint64_t a_desc0 = umma_desc_sw128(smem_u32(ring_a + (size_t)as * kLtATile));
            const uint64_t b_desc0 = umma_desc_sw128(smem_u32(ring_b + (size_t)bs * BSLOT));
            // the runs that begin in this stage take the next accumulators of the ring once the fold warps have read
            // their last use: wait for those first, then issue the whole stage from one thread
            bool ok = true;
#pragma unroll
            for (int ks = 0; ks < kLtStage / 16; ++ks) {
                const int depth = i * kLtStage + 16 * ks;
                const int ri = depth >> log2_run;
                if (depth < k_end && (depth & (run - 1)) == 0 && ri >= NACC && ok)
                    ok = __all_sync(0xffffffffu, mbar_wait_poll(&acc_empty[ri % NACC], ((ri / NACC) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            }
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < kLtStage / 16; ++ks) {
                    const int depth = i * kLtStage + 16 * ks;
                    if (depth >= k_end) break;                             // padding past the last real K-block
                    const int buf = (depth >> log2_run) % NACC;             // the accumulator of the depth's run
                    const bool first = (depth & (run - 1)) == 0;
                    const bool last = ((depth + 16) & (run - 1)) == 0 || depth + 16 >= k_end;
                    umma_f16(tmem_base + (uint32_t)(buf * ACC_STRIDE), a_desc0 + 2 * ks, b_desc0 + 2 * ks, idesc, first ? 0u : 1u);
                    if (last) umma_commit(&acc_full[buf]);
                }
                umma_commit(&a_empty[as]);
                umma_commit(&b_empty[bs]);
            }
            __syncwarp();
        }
    } else if (warp < 8) {
        // ===================== expand warps: four pairs of warps take the stages in turn =====================
        // A warp's trip through one stage (waits, loads, expansion, stores, fence, arrival) is a chain of
        // latencies several hundred cycles long however little it computes, so a stage is not spread over
        // all eight warps: pair (stage % 4) expands it, each warp four column groups with independent
        // instruction chains, and four stages are in flight at once.
        const int g = lane >> 2, t = lane & 3;
        const int pair = warp >> 1, half = warp & 1;
        for (int i = pair; i < stages; i += 4) {
            const int gq = i / kLtSlotStages, si = i % kLtSlotStages, ks_slot = gq % kLtNK, as = i % NA;
            if (i >= NA && !__all_sync(0xffffffffu, mbar_wait_poll(&a_empty[as], ((i / NA) - 1) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            if (!__all_sync(0xffffffffu, mbar_wait_poll(&k_full[ks_slot], (gq / kLtNK) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            unsigned char* at = ring_a + (size_t)as * kLtATile;
            const int h = si % SPU;                                            // 64-deep part of the unit
            const unsigned char* pk = ring_k + (size_t)ks_slot * KSLOT + (si / SPU) * kUnitBytes + lane * 16;
            uint4 wv[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) wv[cc] = *reinterpret_cast<const uint4*>(pk + (size_t)(4 * half + cc) * UPS * kUnitBytes);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                const int row_lo = 16 * (4 * half + cc) + g, row_hi = row_lo + 8;
                // 8 depths (16 bytes) of a 32-deep step land in chunk 4 * step + t of the row
                const uint32_t off_lo = (uint32_t)((row_lo >> 3) * 1024 + (row_lo & 7) * 128);
                const uint32_t off_hi = (uint32_t)((row_hi >> 3) * 1024 + (row_hi & 7) * 128);
                const uint32_t sw_lo = (uint32_t)(row_lo & 7), sw_hi = (uint32_t)(row_hi & 7);
                // 2-bit: words 2 h, 2 h + 1 (32 depths each); 1-bit: word h (its two 4-bit halves are the two steps)
                const uint32_t w0 = BITS == 2 ? (h ? wv[cc].z : wv[cc].x) : (h == 0 ? wv[cc].x : (h == 1 ? wv[cc].y : (h == 2 ? wv[cc].z : wv[cc].w)));
                const uint32_t w1 = h ? wv[cc].w : wv[cc].y;
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    // 32-deep step s of the stage: depths 8 t .. 8 t + 7 of columns g (lo) and g + 8 (hi)
                    uint32_t lo03 = 0, lo47 = 0, hi03 = 0, hi47 = 0;           // 2-bit: four bytes each: u of depths +0..3 / +4..7
                    if (BITS == 2) {
                        const uint32_t w = s ? w1 : w0;
                        const uint32_t e = w & 0x33333333u, o = (w >> 2) & 0x33333333u;
                        lo03 = prmt2(p.lut, 0u, e); lo47 = prmt2(p.lut, 0u, e >> 16);
                        hi03 = prmt2(p.lut, 0u, o); hi47 = prmt2(p.lut, 0u, o >> 16);
                    }
                    const uint32_t chunk = (uint32_t)(4 * s + t);
                    if (BITS == 1) {
                        // A sign bit stays where it lies in its half word: bit b of an f16 is the number 2^(b-24) for
                        // b < 12, and act_quant_kernel has left the codes of a run of eight depths in the order
                        // 0 2 1 3 4 6 5 7, scaled by 2^8 2^8 1 1 2^6 2^6 2^-2 2^-2: every product of column g is
                        // u q 2^-16 and of column g + 8 (one bit higher) u q 2^-15.  One AND per register.
                        const uint32_t v = w0 >> (4 * s);
                        *reinterpret_cast<uint4*>(at + off_lo + ((chunk ^ sw_lo) << 4)) =
                            make_uint4(v & 0x00010001u, v & 0x01000100u, v & 0x00040004u, v & 0x04000400u);
                        *reinterpret_cast<uint4*>(at + off_hi + ((chunk ^ sw_hi) << 4)) =
                            make_uint4(v & 0x00020002u, v & 0x02000200u, v & 0x00080008u, v & 0x08000800u);
                        continue;
                    }
                    const uint2 l0 = widen4(lo03), l1 = widen4(lo47), h0 = widen4(hi03), h1 = widen4(hi47);
                    *reinterpret_cast<uint4*>(at + off_lo + ((chunk ^ sw_lo) << 4)) = make_uint4(l0.x, l0.y, l1.x, l1.y);
                    *reinterpret_cast<uint4*>(at + off_hi + ((chunk ^ sw_hi) << 4)) = make_uint4(h0.x, h0.y, h1.x, h1.y);
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&a_full[as]);
                mbar_arrive(&k_empty[ks_slot]);        // one arrival per warp and stage: a full slot collects 16
            }
        }
    } else if (warp < 16) {
        // ===================== fold warps: thread = weight column, registers = rows =====================
        const int dw = warp - 8, q = dw & 3, part = dw >> 2;
        if (part < DW) {
            const int cl = 32 * q + lane;                                   // column within the CTA tile
            const int col = col0 + cl;
            const uint32_t lane_base = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(part * TPW);
            const int row0 = tok0 + part * TPW;                             // first activation row of this warp
            const int sc_off = NT * 8 + (cl >> 4) * 32 + scale_slot(cl & 15) * 2;   // this column's scale inside a fold slot
            // what turns an accumulator into S = sum u q: 2-bit sums are scaled by 2^-24, 1-bit by 2^-16 (columns g of a
            // column group) or 2^-15 (columns g + 8)
            const float unscale = BITS == 2 ? 16777216.0f : ((cl & 8) ? 32768.0f : 65536.0f);
            float tot[TPW];
#pragma unroll
            for (int j = 0; j < TPW; ++j) tot[j] = 0.0f;
            bool ok = true;
            const int rpb = block >> log2_run;                              // runs per K-block
            int ri = 0;                                                     // run counter
            for (int blk = 0; blk < p.nb_real && ok; ++blk) {
                const int fs = blk % kLtNF;
                int sblk[TPW];                                              // the block's integer sums
#pragma unroll
                for (int j = 0; j < TPW; ++j) sblk[j] = 0;
                // runs of this block that hold staged depths
                const int runs = min(rpb, (k_end - (blk << p.log2_block) + run - 1) >> log2_run);
                for (int rr = 0; rr < runs; ++rr, ++ri) {
                    const int buf = ri % NACC;
                    ok = mbar_wait_poll(&acc_full[buf], (ri / NACC) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT);
                    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int j0 = 0; j0 < TPW; j0 += 8) {
                        uint32_t r[8];
                        tmem_ld8(lane_base + (uint32_t)(buf * ACC_STRIDE + j0), r);
                        tmem_ld_wait();
                        // the accumulator holds (sum of u * q) / unscale exactly
#pragma unroll
                        for (int j = 0; j < 8; ++j) sblk[j0 + j] += __float2int_rn(__uint_as_float(r[j]) * unscale);
                    }
                    // the accumulator is in registers: hand it back to the MMA warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[buf]);
                }
                if (!ok) break;
                ok = mbar_wait_poll(&f_full[fs], (blk / kLtNF) & 1, abort_flag, p.status, STATUS_TMEM_TIMEOUT);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                const unsigned char* fo = ring_f + (size_t)fs * FSLOT;
                const float scale = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t*>(fo + sc_off)));
                const float* sa = reinterpret_cast<const float*>(fo) + part * TPW;
                const float* qs = reinterpret_cast<const float*>(fo + NT * 4) + part * TPW;
#pragma unroll
                for (int j0 = 0; j0 < TPW; j0 += 4) {
                    const float4 s0 = *reinterpret_cast<const float4*>(sa + j0);
                    const float4 q0 = *reinterpret_cast<const float4*>(qs + j0);
                    const float sv[4] = {s0.x, s0.y, s0.z, s0.w};
                    const int qv[4] = {__float2int_rn(q0.x), __float2int_rn(q0.y), __float2int_rn(q0.z), __float2int_rn(q0.w)};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        // 1-bit: u is the sign bit, value = 2 u - 1; 2-bit: u = value + 128
                        const int sum = BITS == 1 ? 2 * sblk[j0 + j] - qv[j] : sblk[j0 + j] - 128 * qv[j];
                        if (p.sums_out && col < p.n && row0 + j0 + j < p.m)
                            p.sums_out[((size_t)(row0 + j0 + j) * p.n + col) * p.nb_real + blk] = sum;
                        tot[j0 + j] = fmaf((float)sum, __fmul_rn(scale, sv[j]), tot[j0 + j]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&f_empty[fs]);
            }
            if (ok && col < p.n) {
#pragma unroll
                for (int j = 0; j < TPW; ++j) {
                    const int row = row0 + j;
                    if (row < p.m) p.c[(size_t)row * p.n + col] = ep_store_value<0>(p.ep, tot[j], (size_t)row, (size_t)col);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------------------------
// K-blocks of one run (16 to 256 depths), the form every model's call takes.  The roles are those above; what differs:
//   * a stage is 128 depths and its operands share one pair of barriers; accumulators change hands in groups (a wait and an
//     arrival of every fold warp cost ~0.6 us of a K-block whatever its depth) and are asked for only where one begins;
//   * the expanded weights go to tensor memory (A operand of the MMA; thread = weight column, 128 depths = 64 columns, four
//     slots), not to shared memory, whose 128 bytes a cycle bound the kernel: written and read there they were half of a
//     stage's traffic at 128 rows;
//   * a weight is its value as an f16 number (1-bit: +-1, the packed bit shifted to the sign; 2-bit: a byte-permute lookup of the
//     codebook's f16 halves), so the accumulator is the K-block's integer itself (|sum| < 2^23, exact) and the fold reads one
//     operand per row, its activation scale: every lane of 16 warps reads each of them, and with the code sums beside them
//     these broadcasts were the other half;
//   * 16 fold warps, four per lane quarter, NT / 4 rows each, totals in registers, two rows per instruction (f32x2).
// NT rows per CTA are chosen by the launcher.  1-bit 512 x 4096 x 14336: 219 us with 64-deep stages in shared memory, 110 now (0.55
// PFLOP/s; the tensor pipe is busy a quarter of the time, two thirds of the issue slots are taken).
constexpr int kLbThreads = 32 * 28;
constexpr int kLbNK = 3, kLbNF = 6;               // ring depths: packed slots (two units a column group), fold operands
constexpr int kLbKSlot = 8 * 2 * kUnitBytes;
constexpr int kLbNS = 4;                          // stages in flight: row tiles in shared memory, weights in tensor memory
constexpr uint32_t kLbACol = 256;                 // tensor memory: two groups of accumulators below, the weights of the stages from here
__host__ __device__ constexpr int lb_group(int nt) { return nt >= 96 ? 1 : 128 / nt; }
__host__ __device__ constexpr size_t lb_smem(int nt) {
    return 1024 + (size_t)kLbNS * nt * 256 + (size_t)kLbNK * kLbKSlot + 1024 + (size_t)kLbNF * lb_group(nt) * (nt * 4 + 256);
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack_f32x2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul_f32x2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

struct LbRing {
    int slot = 0;
    unsigned phase = 0;
    bool wrapped = false;
    __device__ __forceinline__ void next(int n) {
        if (++slot == n) { slot = 0; phase ^= 1u; wrapped = true; }
    }
};

// Tensor maps of the four streams, one tiled copy per stage, packed slot or group of K-blocks each (ten bulk copies of 32 to 512
// bytes per K-block took their warp ~1000 cycles to issue, more than everything else did in that time):
//   rows    activation codes as f16 [m][kq], 64 depths x NT rows       codes   packed units [n16][ku x 512 B], two units of 8 groups
//   sa      activation scales [nb][mpad], NT rows of G blocks      scales  [n16][nb x 32 B], G blocks of 8 groups
struct LbMaps { CUtensorMap rows, codes, sa, scales; };

template <int BITS, int NT>
__global__ void __launch_bounds__(kLbThreads, 1) lowbit_tc_block_kernel(const __grid_constant__ LbMaps maps, const __grid_constant__ LowbitTcArgs p) {
    constexpr int NS = kLbNS, G = lb_group(NT), ACC_STRIDE = 128 / G;
    constexpr int TPW = NT / 4;                                // rows of a fold warp
    constexpr int BTILE = NT * 128;                            // row tile of 64 depths
    constexpr int SLOT = 2 * BTILE;
    constexpr int SPK = BITS == 2 ? 2 : 4;                     // stages per packed slot
    constexpr int FSLOT = G * (NT * 4 + 256);                  // [G][NT] row scales, then [8 column groups][G][16 f16 scales]
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    unsigned char* ring_k = smem + (size_t)NS * SLOT;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring_k + (size_t)kLbNK * kLbKSlot);
    unsigned char* ring_f = reinterpret_cast<unsigned char*>(bars) + 1024;
    uint64_t *full = bars, *empty = full + NS, *k_full = empty + NS, *k_empty = k_full + kLbNK, *acc_full = k_empty + kLbNK, *acc_empty = acc_full + 2,
             *f_full = acc_empty + 2, *f_empty = f_full + kLbNF;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(f_empty + kLbNF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int col0 = blockIdx.x * 128, cg0 = blockIdx.x * 8, tok0 = blockIdx.y * NT;
    // depths that belong to a real K-block and are staged (>= k: what lies past k multiplies zero activations)
    const int k_end = (int)min((long long)p.nb_real << p.log2_block, (long long)p.kq);
    const int stages = (k_end + 127) >> 7;

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) { mbar_init(&full[s], 5); mbar_init(&empty[s], 1); }
        for (int s = 0; s < kLbNK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 4 * SPK); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 16); }
        for (int s = 0; s < kLbNF; ++s) { mbar_init(&f_full[s], 1); mbar_init(&f_empty[s], 16); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    pdl_wait();                                                // (before the allocation: the kernel ahead may still hold tensor memory)
    if (warp == 25) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = *tmem_slot;

    if (warp == 24) {                                          // ---- row tiles ----
        if (lane == 0) {
            tma_prefetch_desc(&maps.rows);
            LbRing r;
            for (int i = 0; i < stages; ++i, r.next(NS)) {
                if (r.wrapped && !mbar_wait(&empty[r.slot], r.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT)) break;
                unsigned char* b = smem + (size_t)r.slot * SLOT;
                mbar_expect_tx(&full[r.slot], 2 * BTILE);
                tma_load_2d(b, &maps.rows, i * 128, tok0, &full[r.slot]);
                tma_load_2d(b + BTILE, &maps.rows, i * 128 + 64, tok0, &full[r.slot]);
            }
        }
    } else if (warp == 26) {                                   // ---- packed weights ----
        if (lane == 0) {
            tma_prefetch_desc(&maps.codes);
            LbRing r;
            for (int u0 = 0; u0 * (BITS == 2 ? kQ2UnitDepth : kQ1UnitDepth) < k_end; u0 += 2, r.next(kLbNK)) {
                if (r.wrapped && !mbar_wait(&k_empty[r.slot], r.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT)) break;
                // whole boxes always: what lies past the last unit or column group arrives as zeros and is never used
                mbar_expect_tx(&k_full[r.slot], (unsigned)kLbKSlot);
                tma_load_2d(ring_k + (size_t)r.slot * kLbKSlot, &maps.codes, u0 * (kUnitBytes / 8), cg0, &k_full[r.slot]);
            }
        }
    } else if (warp == 27) {                                   // ---- fold operands ----
        if (lane == 0) {
            tma_prefetch_desc(&maps.sa);
            tma_prefetch_desc(&maps.scales);
            LbRing r;
            for (int blk0 = 0; blk0 < p.nb_real; blk0 += G, r.next(kLbNF)) {
                if (r.wrapped && !mbar_wait(&f_empty[r.slot], r.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT)) break;
                unsigned char* dst = ring_f + (size_t)r.slot * FSLOT;
                mbar_expect_tx(&f_full[r.slot], (unsigned)FSLOT);
                tma_load_2d(dst, &maps.sa, tok0, blk0, &f_full[r.slot]);
                tma_load_2d(dst + G * NT * 4, &maps.scales, blk0 * 4, cg0, &f_full[r.slot]);
            }
        }
    } else if (warp == 25) {                                   // ---- MMA ----
        const uint32_t idesc = umma_idesc(0, 128, NT);
        const uint64_t b_first = umma_desc_sw128(smem_u32(smem));
        LbRing r, acc;                                         // acc: group of accumulators; ga: the one in it
        int ga = 0;
        const int L = p.log2_block;
        if (L >= 7) {
            // one accumulator per 128 or 256 depths
            const int mask = (1 << (L - 7)) - 1;
            for (int i = 0; i < stages; ++i, r.next(NS)) {
                const bool first = (i & mask) == 0, last = ((i + 1) & mask) == 0 || i == stages - 1;
                if (ga == 0 && first && acc.wrapped && !__all_sync(0xffffffffu, mbar_wait(&acc_empty[acc.slot], acc.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
                if (!__all_sync(0xffffffffu, mbar_wait(&full[r.slot], r.phase, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
                tc_fence_after();
                const uint32_t at = tmem + kLbACol + 64u * (uint32_t)r.slot;
                const uint64_t bd = b_first + (uint64_t)(r.slot * (SLOT >> 4));
                const uint32_t d = tmem + (uint32_t)((acc.slot * G + ga) * ACC_STRIDE);
                const bool hand = last && (ga == G - 1 || i == stages - 1);
                if (elect_one()) {
                    if (k_end - i * 128 >= 128) {
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)
                            umma_f16_ts(d, at + 8 * ks, bd + (ks >> 2) * (BTILE >> 4) + 2 * (ks & 3), idesc, ks > 0 || !first);
                    } else {
                        for (int ks = 0; i * 128 + 16 * ks < k_end; ++ks)
                            umma_f16_ts(d, at + 8 * ks, bd + (ks >> 2) * (BTILE >> 4) + 2 * (ks & 3), idesc, ks > 0 || !first);
                    }
                    umma_commit(&empty[r.slot]);
                    if (hand) umma_commit(&acc_full[acc.slot]);
                }
                __syncwarp();
                if (hand) { ga = 0; acc.next(2); }
                else if (last) ++ga;
            }
        } else {
            // several runs per stage, an accumulator each; a group is asked for as its first run begins (the groups before it
            // are on their way to the fold warps by then)
            auto walk = [&](auto steps_c) {
                constexpr int STEPS = decltype(steps_c)::value;              // K = 16 steps of a run
                for (int i = 0; i < stages; ++i, r.next(NS)) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[r.slot], r.phase, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) return;
                    tc_fence_after();
                    const uint32_t at = tmem + kLbACol + 64u * (uint32_t)r.slot;
                    const uint64_t bd = b_first + (uint64_t)(r.slot * (SLOT >> 4));
                    const int left = min(8, (k_end - i * 128) >> 4);             // K = 16 steps of the stage
#pragma unroll
                    for (int k0 = 0; k0 < 8; k0 += STEPS) {
                        if (k0 >= left) break;
                        if (ga == 0 && acc.wrapped) {
                            if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[acc.slot], acc.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) return;
                            tc_fence_after();
                        }
                        const uint32_t d = tmem + (uint32_t)((acc.slot * G + ga) * ACC_STRIDE);
                        const bool end = k0 + STEPS >= left, hand = ga == G - 1 || (end && i == stages - 1);
                        if (elect_one()) {
#pragma unroll
                            for (int ks = k0; ks < k0 + STEPS; ++ks)
                                if (ks < left) umma_f16_ts(d, at + 8 * ks, bd + (ks >> 2) * (BTILE >> 4) + 2 * (ks & 3), idesc, ks > k0);
                            if (hand) umma_commit(&acc_full[acc.slot]);
                            if (end) umma_commit(&empty[r.slot]);
                        }
                        __syncwarp();
                        if (hand) { ga = 0; acc.next(2); }
                        else ++ga;
                    }
                }
            };
            if (L == 6) walk(std::integral_constant<int, 4>());
            else if (L == 5) walk(std::integral_constant<int, 2>());
            else walk(std::integral_constant<int, 1>());
        }
    } else if (warp < 8) {                                     // ---- expand ----
        // thread = weight column: group `group` of warps takes every other stage, warp w the lane quarter w % 4
        const int group = warp >> 2, q = warp & 3, cl = 32 * q + lane, g = cl & 7, hi = (cl >> 3) & 1;
        const uint32_t at = tmem + ((uint32_t)(32 * q) << 16) + kLbACol;
        // the column's depths lie in the 16-byte vectors of four lanes of its column group's units (packed for lane (g, t):
        // columns g and g + 8, runs of eight depths at 8 t)
        const uint32_t pk = smem_u32(ring_k) + (uint32_t)((cl >> 4) * 2 * kUnitBytes + g * 64);
        uint32_t lut_lo = 0, lut_hi = 0;                       // 2-bit: low and high bytes of the codebook's values as f16 numbers
        if (BITS == 2) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t h = __half_as_ushort(__int2half_rn((int)(int8_t)((p.lut ^ 0x80808080u) >> (8 * c))));
                lut_lo |= (h & 0xffu) << (8 * c);
                lut_hi |= (h >> 8) << (8 * c);
            }
        }
        LbRing r, kr;
        if (group) r.next(NS);
        for (int i = group; i < stages; i += 2, r.next(NS), r.next(NS)) {
            const int part = i & (SPK - 1);                    // stage within its packed slot
            if (i >= SPK && part == group) kr.next(kLbNK);
            if (!__all_sync(0xffffffffu, mbar_wait(&k_full[kr.slot], kr.phase, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            // 2-bit: a unit is the stage, word s its 32-deep step s; 1-bit: half a unit, a word two steps
            const uint32_t src = pk + (uint32_t)(kr.slot * kLbKSlot) + (uint32_t)(BITS == 2 ? part * kUnitBytes : (part >> 1) * kUnitBytes + (part & 1) * 8);
            uint32_t w[4][BITS == 2 ? 4 : 2];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if constexpr (BITS == 2)
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[t][0]), "=r"(w[t][1]), "=r"(w[t][2]), "=r"(w[t][3]) : "r"(src + 16 * t) : "memory");
                else
                    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(w[t][0]), "=r"(w[t][1]) : "r"(src + 16 * t) : "memory");
            }
            if (r.wrapped && !__all_sync(0xffffffffu, mbar_wait(&empty[r.slot], r.phase ^ 1u, abort_flag, p.status, STATUS_TMEM_TIMEOUT))) break;
            tc_fence_after();
#pragma unroll
            for (int s = 0; s < 4; ++s) {                      // 32-deep step: 16 tensor-memory columns
                uint32_t o[16];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (BITS == 1) {
                        // the bits of depths (0, 2), (1, 3), (4, 6), (5, 7) -- the order act_quant_kernel leaves the codes in --
                        // lie 16 apart: one shift brings a pair to the signs of two f16 ones (bit set = +1)
                        const uint32_t v = w[t][s >> 1] << (1 - hi);
                        const int up = 14 - 4 * (s & 1);
                        o[4 * t] = (~(v << up) & 0x80008000u) | 0x3c003c00u;
                        o[4 * t + 1] = (~(v << (up - 8)) & 0x80008000u) | 0x3c003c00u;
                        o[4 * t + 2] = (~(v << (up - 2)) & 0x80008000u) | 0x3c003c00u;
                        o[4 * t + 3] = (~(v << (up - 10)) & 0x80008000u) | 0x3c003c00u;
                    } else {
                        const uint32_t e = (w[t][s] >> (2 * hi)) & 0x33333333u;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {          // depths 0-3, 4-7
                            const uint32_t lo = prmt2(lut_lo, 0u, e >> (16 * h)), up = prmt2(lut_hi, 0u, e >> (16 * h));
                            o[4 * t + 2 * h] = prmt2(lo, up, 0x5140u);
                            o[4 * t + 2 * h + 1] = prmt2(lo, up, 0x7362u);
                        }
                    }
                }
                tmem_st16(at + (uint32_t)(64 * r.slot + 16 * s), o);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[r.slot]);
                mbar_arrive(&k_empty[kr.slot]);
            }
        }
    } else {                                                   // ---- fold: thread = weight column, registers = rows ----
        const int dw = warp - 8, q = dw & 3, part = dw >> 2;
        const int cl = 32 * q + lane, col = col0 + cl;
        const uint32_t acc_base = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(part * TPW);
        const int sc_off = G * NT * 4 + (cl >> 4) * (G * 32) + scale_slot(cl & 15) * 2;   // this column's first scale inside a fold slot
        f32x2 tot[TPW / 2];
#pragma unroll
        for (int j = 0; j < TPW / 2; ++j) tot[j] = 0ull;
        LbRing acc, fr;
        bool ok = true;
        for (int blk0 = 0; blk0 < p.nb_real; blk0 += G, acc.next(2), fr.next(kLbNF)) {
            ok = __all_sync(0xffffffffu, mbar_wait(&f_full[fr.slot], fr.phase, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (!ok) break;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc.slot], acc.phase, abort_flag, p.status, STATUS_TMEM_TIMEOUT));
            if (!ok) break;
            tc_fence_after();
            const int blocks = min(G, p.nb_real - blk0);
#pragma unroll
            for (int gi = 0; gi < G; ++gi) {
                if (gi >= blocks) break;
                const unsigned char* fo = ring_f + (size_t)fr.slot * FSLOT;
                const float scale = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t*>(fo + sc_off + gi * 32)));
                const f32x2 scale2 = pack_f32x2(scale, scale);
                const ulonglong2* sa = reinterpret_cast<const ulonglong2*>(fo + gi * NT * 4 + part * TPW * 4);
                // Eight rows at a time, the next eight on their way while these are folded: a warp takes its rows of every
                // block one block after the other, so the length of this chain is the time of a K-block.
                const uint32_t src = acc_base + (uint32_t)((acc.slot * G + gi) * ACC_STRIDE);
                uint32_t av[2][8];
                tmem_ld8(src, av[0]);
#pragma unroll
                for (int c = 0; c < TPW / 8; ++c) {
                    const ulonglong2 s0 = sa[2 * c], s1 = sa[2 * c + 1];
                    tmem_ld_wait();
                    if (c + 1 < TPW / 8) {
                        tmem_ld8(src + 8 * (c + 1), av[(c + 1) & 1]);
                    } else if (gi == blocks - 1) {
                        // the group has been read: hand it back to the MMA warp
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&acc_empty[acc.slot]);
                    }
                    // total = fmaf((float)sum, scale * sa, total), the reference's statement, two rows at a time
                    const uint32_t(&v)[8] = av[c & 1];
                    f32x2* to = tot + 4 * c;
                    to[0] = fma_f32x2(pack_f32x2(__uint_as_float(v[0]), __uint_as_float(v[1])), mul_f32x2(scale2, s0.x), to[0]);
                    to[1] = fma_f32x2(pack_f32x2(__uint_as_float(v[2]), __uint_as_float(v[3])), mul_f32x2(scale2, s0.y), to[1]);
                    to[2] = fma_f32x2(pack_f32x2(__uint_as_float(v[4]), __uint_as_float(v[5])), mul_f32x2(scale2, s1.x), to[2]);
                    to[3] = fma_f32x2(pack_f32x2(__uint_as_float(v[6]), __uint_as_float(v[7])), mul_f32x2(scale2, s1.y), to[3]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&f_empty[fr.slot]);
        }
        if (ok && col < p.n) {
#pragma unroll
            for (int j = 0; j < TPW; j += 2) {
                float a, b;
                unpack_f32x2(tot[j / 2], a, b);
                const int row = tok0 + part * TPW + j;
                if (row < p.m) p.c[(size_t)row * p.n + col] = ep_store_value<0>(p.ep, a, (size_t)row, (size_t)col);
                if (row + 1 < p.m) p.c[(size_t)(row + 1) * p.n + col] = ep_store_value<0>(p.ep, b, (size_t)(row + 1), (size_t)col);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 25) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int BITS, int TPW, int DW>
cudaError_t launch_lt(const CUtensorMap& tm, const LowbitTcArgs& a, dim3 grid, size_t smem, cudaStream_t stream) {
    auto kern = lowbit_tc_kernel<BITS, TPW, DW>;
    static std::atomic<int> attr_dev{-1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev.load(std::memory_order_acquire) != dev) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        attr_dev.store(dev, std::memory_order_release);
    }
    kern<<<grid, kLtThreads, smem, stream>>>(tm, a);
    return cudaGetLastError();
}

template <int BITS, int NT>
cudaError_t launch_lb(const CUtensorMap& rows, const LowbitTcArgs& a, dim3 grid, cudaStream_t stream) {
    constexpr int G = lb_group(NT);
    LbMaps maps;
    maps.rows = rows;
    const cuuint32_t estr[2] = {1, 1};
    const cuuint64_t cdim[2] = {(cuuint64_t)a.ku * (kUnitBytes / 8), (cuuint64_t)a.n16}, cstride[1] = {(cuuint64_t)a.ku * kUnitBytes};
    const cuuint32_t cbox[2] = {2 * kUnitBytes / 8, 8};
    const cuuint64_t qdim[2] = {(cuuint64_t)a.mpad, (cuuint64_t)a.nb}, qstride[1] = {(cuuint64_t)a.mpad * 4};
    const cuuint32_t qbox[2] = {NT, (cuuint32_t)G};
    const cuuint64_t sdim[2] = {(cuuint64_t)a.nb * 4, (cuuint64_t)a.n16}, sstride[1] = {(cuuint64_t)a.nb * 32};
    const cuuint32_t sbox[2] = {(cuuint32_t)(4 * G), 8};
    auto map = [&](CUtensorMap* m, CUtensorMapDataType type, const void* base, const cuuint64_t* dim, const cuuint64_t* stride, const cuuint32_t* box) {
        return tensor_map_encoder()(m, type, 2, (void*)base, dim, stride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!map(&maps.codes, CU_TENSOR_MAP_DATA_TYPE_UINT64, a.codes, cdim, cstride, cbox) ||
        !map(&maps.sa, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.sa_t, qdim, qstride, qbox) ||
        !map(&maps.scales, CU_TENSOR_MAP_DATA_TYPE_UINT64, a.scales, sdim, sstride, sbox))
        return cudaErrorInvalidValue;
    auto kern = lowbit_tc_block_kernel<BITS, NT>;
    static std::atomic<int> attr_dev{-1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (attr_dev.load(std::memory_order_acquire) != dev) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lb_smem(NT));
        if (e != cudaSuccess) return e;
        attr_dev.store(dev, std::memory_order_release);
    }
    return launch_pdl(kern, grid, dim3(kLbThreads), lb_smem(NT), stream, maps, a);
}

}  // namespace

bool lowbit_tc_supported(int bits, int m, int k, int log2_block) {
    if (bits != 1 && bits != 2) return false;
    if (m < 1 || k < 1 || log2_block < 4) return false;           // an MMA step is 16 deep: K-blocks of 16 and up
    if (log2_block > 16) return false;                             // a block's sum of activation codes travels as a float
    return tensor_map_encoder() != nullptr;
}

bool lowbit_tc_one_run(int log2_block, bool sums) { return log2_block <= 8 && !sums; }

cudaError_t lowbit_tc_launch(LowbitTcArgs a, int sm_count, cudaStream_t stream) {
    // blocks of one run and no debug output: the floating-point fold
    const bool one_run = lowbit_tc_one_run(a.log2_block, a.sums_out != nullptr);
    const int col_tiles = (a.n + 127) / 128;
    // an MMA of 128 weight columns takes 16 rows or more
    int nt = a.m <= 16 ? 16 : (a.m <= 32 ? 32 : 64);
    if (one_run) {
        // rows per CTA: the fewest (waves x time of a tile); a tile costs its expansion whatever its rows, about what 60
        // rows of fold cost
        long long best = 0;
        for (int t : {128, 96, 64, 32}) {
            const long long tiles = (long long)col_tiles * ((a.m + t - 1) / t), cost = (tiles + sm_count - 1) / sm_count * (60 + t);
            if (best == 0 || cost < best) { best = cost; nt = t; }
        }
    }
    CUtensorMap tm;
    const cuuint64_t gdim[2] = {(cuuint64_t)a.kq, (cuuint64_t)a.m};
    const cuuint64_t gstride[1] = {(cuuint64_t)a.kq * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kLtStage, (cuuint32_t)nt};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = tensor_map_encoder()(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)a.qh, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    const dim3 grid(col_tiles, (a.m + nt - 1) / nt);
    if (one_run) {
        if (a.bits == 2) {
            if (nt == 32) return launch_lb<2, 32>(tm, a, grid, stream);
            if (nt == 64) return launch_lb<2, 64>(tm, a, grid, stream);
            if (nt == 96) return launch_lb<2, 96>(tm, a, grid, stream);
            return launch_lb<2, 128>(tm, a, grid, stream);
        }
        if (nt == 32) return launch_lb<1, 32>(tm, a, grid, stream);
        if (nt == 64) return launch_lb<1, 64>(tm, a, grid, stream);
        if (nt == 96) return launch_lb<1, 96>(tm, a, grid, stream);
        return launch_lb<1, 128>(tm, a, grid, stream);
    }
    const int ups = a.bits == 2 ? 4 : 2;
    const int bslot = (nt * 128 + 1023) / 1024 * 1024;
    const size_t smem = 1024 + (size_t)kLtNA * kLtATile + (size_t)kLtNB * bslot + (size_t)kLtNK * 8 * ups * kUnitBytes +
                        1024 + (size_t)kLtNF * (nt * 8 + 256) + 64;
    if (a.bits == 2) {
        if (nt == 16) return launch_lt<2, 16, 1>(tm, a, grid, smem, stream);
        if (nt == 32) return launch_lt<2, 16, 2>(tm, a, grid, smem, stream);
        return launch_lt<2, 32, 2>(tm, a, grid, smem, stream);
    }
    if (nt == 16) return launch_lt<1, 16, 1>(tm, a, grid, smem, stream);
    if (nt == 32) return launch_lt<1, 16, 2>(tm, a, grid, smem, stream);
    return launch_lt<1, 32, 2>(tm, a, grid, smem, stream);
}

}  // namespace smeg
