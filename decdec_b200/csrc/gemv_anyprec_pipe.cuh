// Any-precision GEMV role for 3 to 8 bits, bulk-copy pipelined variant.
//
// In the tensor [plane][row][K/32] consecutive rows of one plane are contiguous, so a stage of R rows is one
// contiguous run per plane plus the R LUT rows.  A producer thread moves them with 1-D bulk asynchronous
// copies (cp.async.bulk, completion counted on an mbarrier) several stages ahead of the consumer warps;
// a warp's work item is (pair of rows of the stage, segment of their channels).
// Bound: the ALU pipe (half of the issue rate): about 1.7 logic and permute operations turn a 3-bit code into its 16-bit weight,
// 2.6 a 4-bit one.  Everything else is kept off that pipe:
//  * the products go through mma.m16n8k16 (16-bit factors, fp32 sums; common.cuh): every lane supplies four weights of either
//    row and its own four activations, lane (g, t) as rows g and g + 8 of A and column g of B, so that the diagonal entries
//    D[g][g] and D[g + 8][g] hold the sums of the quad's lanes for the two rows; the other entries mix lanes and are not used.
//    One instruction consumes eight weights per lane, and nothing is summed in 16 bits;
//  * the eight diagonal sums of a row are stored, not shuffled together: the fold at the end adds a row's slots, in a fixed order;
//  * the loop over a row's 1024-channel blocks is unrolled twice at 3 bits (28672 x 4096 23.1 -> 22.7 us; at 4 to 8 bits small layers
//    lose by it: 512 x 1792 at 8 bits 3.5 -> 3.8), and the last, shorter block has a body of its own, so that the masks it needs
//    are not paid for by the others.
// Measured, fp16, us per launch in a graph, against the same stages with packed 16-bit sums (3 bits) or two address operations and
// one mixed-precision multiply-add per weight (4 to 8 bits): on 28672 x 4096 3 bits 22.7 -> 22.7, 4 bits 37.6 -> 29.3, 5 bits
// 51.1 -> 33.1, 6 bits 52.4 -> 34.4, 8 bits 57.9 -> 53.4 (2.0, 2.0, 2.2, 2.6 and 2.5 TB/s of algorithmic bytes); on 4096 x 14336 16.1 -> 12.6, 25.5 -> 19.3, 37.0 -> 31.2; on
// 768 x 4096 3.6 -> 3.1, 4.9 -> 3.7, 6.5 -> 4.8.
// Two decoders.  3 bits: the row's table lives in registers and is looked up by byte permutes (lut_bytes.cuh), activations staged
// in the order in which the products take them.  4 to 8 bits: the plane words are regrouped into 4-bit fields, each code indexes the
// row's LUT in shared memory (a row of up to 64 entries spans at most 32 banks and equal entries broadcast, so a
// lookup is one wavefront).
// A CTA owns its rows completely (all of K) and folds them into y itself: GEMV-only launches use no global accumulator, ticket
// or fence.  Fused launches store the sums into the workspace accumulator and arrive on the tile's ticket, where they meet
// the compensation CTAs.
// Requirements: K % 128 == 0, K <= 32768.  Every mbarrier wait is bounded.
#pragma once
#include "gemv_anyprec.cuh"
#include "gemv_bcq_pipe.cuh"
#include "lut_bytes.cuh"

namespace dd {

constexpr int kApPipeThreads = 544;   // 16 consumer warps + 1 producer warp

struct ApPipeGeom {
    uint32_t rows_per_stage;   // R
    uint32_t segs;             // warps per pair of rows
    uint32_t seg_words;        // plane words (32 channels each) of a row that one warp takes: a multiple of 32
    uint32_t stages;           // pipeline depth
    uint32_t stage_bytes;
    uint32_t x_bytes;          // staged activations (rounded to 128)
    uint32_t rows_per_cta;     // even; a multiple of 32 beside a compensation role
    uint32_t part_bytes;       // partial sums of the CTA: fp32 [row][segment][8]
    uint32_t lut_off;          // where the warps keep their LUT rows at 4 to 7 bits (aligned to kApLutStride)
    uint32_t smem_bytes;
    uint32_t direct;           // 1: fold into y; 0: store into the accumulator and take the tile's ticket
    uint32_t wait_ns;          // limit of one mbarrier wait (DECDEC_PIPE_WAIT_NS)
};

constexpr int kApPipeHdr = 256;   // [abort, flag][full barriers 8][empty barriers 8]

// One plane-word position (32 channels) of one row through the lookup decoder: W[jj][i] = weights of channels 2i (low half) and
// 2i + 1 of group jj, beside the activations as they lie in memory.  `lut` is the window address of the row's LUT.  Even and odd
// nibble positions are moved into the bytes of two words (E and O).  Up to 7 bits such a byte holds the byte offset of an entry,
// 2 * code, and one byte permute puts it under the upper bytes of `lut`, which is aligned to kApLutStride.  At 8 bits it holds
// the code; a permute takes it out and `lut`, where the copy landed it, is added: 512 bytes per row are too much to move again in
// every warp (768 x 4096 7.5 us, 5.0 without).
constexpr uint32_t kApLutStride = 256;

template <int BITS>
__device__ __forceinline__ void ap_lookup_word(const uint32_t* q, uint32_t lut, uint32_t (&W)[4][4]) {
    constexpr int BH = BITS < 4 ? BITS : 4, BL = BITS - BH;
    uint32_t Mh[4], Ml[4] = {0u, 0u, 0u, 0u}, E[4], O[4];
    ap_merge<BH>(q, Mh);
    if constexpr (BL > 0) ap_merge<BL>(q + 4, Ml);
    constexpr uint32_t mh = 0x01010101u * (((1u << BH) - 1u) << (BITS <= 7 ? BL + 1 : BL)), ml = 0x01010101u * (((1u << BL) - 1u) << (BITS <= 7 ? 1 : 0));
#pragma unroll
    for (int ph = 0; ph < 4; ++ph) {
        const int rh = BH - 1 - ph + (BITS <= 7 ? BL + 1 : BL), rl = BL - 1 - ph + (BITS <= 7 ? 1 : 0);
        E[ph] = rotate_left(Mh[ph], rh) & mh;
        O[ph] = rotate_left(Mh[ph], rh - 4) & mh;
        if constexpr (BL > 0) {
            E[ph] |= rotate_left(Ml[ph], rl) & ml;
            O[ph] |= rotate_left(Ml[ph], rl - 4) & ml;
        }
    }
    auto entry = [&](int ph, int t) -> uint32_t {          // entry of the code at bit 4t + ph
        const uint32_t src = (t & 1) ? O[ph] : E[ph];
        const int b = t >> 1;
        uint32_t addr;
        if constexpr (BITS <= 7) addr = __byte_perm(src, lut, 0x7650u | (uint32_t)b);
        else addr = lut + 2u * __byte_perm(src, 0u, 0x4440u | (uint32_t)b);
        uint16_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
        return v;
    };
    // bit 31 - 8jj - r of the word is channel r of group jj
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
        for (int i = 0; i < 4; ++i) {                       // channels 2i, 2i + 1: bits 7 - 2i and 6 - 2i of the byte
            const int t = 2 * (3 - jj) + (i < 2 ? 1 : 0), ph = (i & 1) ? 1 : 3;
            W[jj][i] = entry(ph, t) | (entry(ph - 1, t) << 16);
        }
}

template <int DT, int BITS>
__device__ void ap_pipe_role(const ApParams& p, const FinParams& f, const ApPipeGeom& geo, uint32_t cta, unsigned char* sm) {
    constexpr bool LOOKUP = BITS > 3;
    constexpr uint32_t kLutRow = 2u << BITS;             // bytes of one row's LUT
    constexpr int NW = 16;                               // consumer warps; warp NW is the producer
    constexpr int NT = (NW + 1) * 32;
    using T = typename Tr<DT>::T;
    static_assert(DT != FP32, "any-precision kernels take fp16/bf16 only");
    volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(sm);
    unsigned* s_flag = reinterpret_cast<unsigned*>(sm + 4);
    const uint32_t bar_full = smem_u32(sm + 64);
    const uint32_t bar_empty = bar_full + 64;
    T* sx = reinterpret_cast<T*>(sm + kApPipeHdr);
    float* part = reinterpret_cast<float*>(sm + kApPipeHdr + geo.x_bytes);
    unsigned char* stage0 = sm + kApPipeHdr + geo.x_bytes + geo.part_bytes;      // the byte offsets are multiples of 128

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nwords = p.K / 32;
    const uint32_t rowbytes = nwords * 4;
    const uint32_t R = geo.rows_per_stage, S = geo.stages;
    const uint32_t r0 = cta * geo.rows_per_cta;
    const uint32_t r1 = min(p.N, r0 + geo.rows_per_cta);
    const uint32_t nst = (r1 - r0 + R - 1) / R;
    const uint32_t lut_off = BITS * R * rowbytes;       // LUT rows sit after the plane runs

    pdl_trigger();
    if (tid == 0) {
        *s_abort = 0u;
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == NW) {
        // ------------------------------ producer (one elected lane) -----------------------------
        if (lane == 0) {
            const size_t plane_stride = (size_t)p.N * nwords;
            const unsigned char* lutb = reinterpret_cast<const unsigned char*>(p.lut);
            uint32_t issued = 0;
            for (uint32_t i = 0; i < nst; ++i) {
                const uint32_t s = i % S, use = i / S;
                if (use > 0) {
                    // slots free only after the consumers' wait for the previous kernel: resolve the dependency before
                    // the first bounded wait (every slot is full by now, so no copy is delayed)
                    if (use == 1 && s == 0) pdl_wait();
                    if (!mbar_wait(bar_empty + 8 * s, (use - 1) & 1u, s_abort, geo.wait_ns)) break;
                }
                const uint32_t n0 = r0 + i * R;
                const uint32_t rows = min(R, r1 - n0);
                const uint32_t full = bar_full + 8 * s;
                mbar_expect_tx(full, rows * (BITS * rowbytes + kLutRow));
                const uint32_t dst = smem_u32(stage0 + (size_t)s * geo.stage_bytes);
#pragma unroll
                for (int pl = 0; pl < BITS; ++pl)
                    bulk_g2s(dst + pl * R * rowbytes, p.qweight + pl * plane_stride + (size_t)n0 * nwords, rows * rowbytes, full);
                bulk_g2s(dst + lut_off, lutb + (size_t)n0 * kLutRow, rows * kLutRow, full);
                issued = i + 1;
            }
            if (*s_abort) {
                const uint32_t first = issued > S ? issued - S : 0;
                for (uint32_t i = first; i < issued; ++i) {
                    volatile uint32_t never = 0;
                    mbar_wait(bar_full + 8 * (i % S), (i / S) & 1u, &never, 1000000000u);
                }
            }
        }
    } else {
        // ------------------------------ consumers ----------------------------------------------
        pdl_wait();     // weights are already streaming (producer warp); activations come from earlier kernels
        const T* x = reinterpret_cast<const T*>(p.x);
        const uint32_t tailE = nwords & 31u;              // words of the row's last, shorter block
        if constexpr (LOOKUP) {
            for (uint32_t k = tid; k < p.K; k += NW * 32) sx[k] = x[k];
        } else {
            // the byte-permute decoder delivers, for every ph, the channel pairs (7 - ph, 3 - ph) of the four groups of a word:
            // their activations are staged side by side, groups 3 to 0, where a group's eight channels lie in memory.  One load of
            // the main loop then holds both operand registers of two instructions, in the right order.
            const bool xvec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0u;
            for (uint32_t w = tid; w < nwords; w += NW * 32) {
                const uint32_t E = (w >> 5) == (nwords >> 5) ? tailE : 32u;
                const uint32_t at = (w & ~31u) * 32u + 8u * (w & 31u);
                union { uint4 v; unsigned short e[8]; } q[4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const unsigned short* src = reinterpret_cast<const unsigned short*>(x) + at + 8u * E * jj;
                    if (xvec) q[jj].v = *reinterpret_cast<const uint4*>(src);
                    else
#pragma unroll
                        for (int r = 0; r < 8; ++r) q[jj].e[r] = src[r];
                }
#pragma unroll
                for (int ph = 0; ph < 4; ++ph) {
                    uint32_t o[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[i] = (uint32_t)q[3 - i].e[7 - ph] | ((uint32_t)q[3 - i].e[3 - ph] << 16);
                    *reinterpret_cast<uint4*>(sx + at + 8u * E * ph) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NW * 32) : "memory");

        const uint32_t pair = warp / geo.segs, seg = warp % geo.segs;
        const uint32_t rowA = 2u * pair, rowB = min(rowA + 1u, R - 1u);   // a stage of one row: its sums are formed twice, used once
        const bool has_item = rowA < R;
        // step s of the segment: lane l takes plane word 32 * s + l of both rows, so that consecutive lanes read consecutive words
        // and consecutive 16-byte activation groups
        const uint32_t w0 = seg * geo.seg_words;
        const uint32_t nseg = w0 < nwords ? min(geo.seg_words, nwords - w0) : 0u;
        const uint32_t full = nseg / 32u;
        const uint32_t g = lane >> 2;
        const bool diag = (lane & 3u) == (g >> 1), odd = (g & 1u) != 0u;
        const uint32_t lut_mine = smem_u32(sm) + geo.lut_off + warp * 2u * kApLutStride;       // 4 to 7 bits
        uint32_t* lut_own = reinterpret_cast<uint32_t*>(sm + geo.lut_off + (size_t)warp * 2u * kApLutStride);

        for (uint32_t i = 0; i < nst; ++i) {
            const uint32_t s = i % S;
            if (!mbar_wait(bar_full + 8 * s, (i / S) & 1u, s_abort, geo.wait_ns)) break;
            const unsigned char* st = stage0 + (size_t)s * geo.stage_bytes;
            const uint32_t o = i * R + rowA;                  // first row of the pair, from r0
            float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            if (has_item && r0 + o < r1) {
                const uint32_t* pA = reinterpret_cast<const uint32_t*>(st + (size_t)rowA * rowbytes) + w0 + lane;
                const uint32_t row_gap = (rowB - rowA) * nwords, plane_gap = R * nwords;
                LutBytes<3> tA, tB;
                if constexpr (!LOOKUP) {
                    const uint4 a = *reinterpret_cast<const uint4*>(st + lut_off + rowA * kLutRow);
                    const uint4 b = *reinterpret_cast<const uint4*>(st + lut_off + rowB * kLutRow);
                    tA.fill_pairs(&a.x);
                    tB.fill_pairs(&b.x);
                } else if constexpr (BITS <= 7) {
                    // the pair's LUT rows to the warp's own, aligned place
                    __syncwarp();
                    const uint32_t* lw = reinterpret_cast<const uint32_t*>(st + lut_off + rowA * kLutRow);
                    constexpr uint32_t half = kLutRow / 4u;
                    const uint32_t n_lw = rowB > rowA ? 2u * half : half;
                    for (uint32_t at = lane; at < n_lw; at += 32u) lut_own[at < half ? at : at - half + kApLutStride / 4u] = lw[at];
                    __syncwarp();
                }
                const uint32_t lutA = BITS <= 7 ? lut_mine : smem_u32(st) + lut_off + rowA * kLutRow;
                const uint32_t lutB = BITS <= 7 ? lut_mine + kApLutStride : lutA + (rowB - rowA) * kLutRow;
                // RAGGED: the last step of a segment that is not a whole number of 32 words.  Lanes without one add zero
                // weights, not table entries that zero activations might turn into NaN.
                auto step = [&](uint32_t u, auto RAGGED) {
                    const bool ok = !RAGGED.value || 32u * u + lane < nseg;
                    const uint32_t blk = (w0 >> 5) + u;
                    const uint32_t E = RAGGED.value ? tailE : 32u;
                    uint32_t qA[BITS], qB[BITS];
                    const uint32_t* at = ok ? pA + 32u * u : pA - lane;        // the segment's first word stands in for one that is not there
#pragma unroll
                    for (int pl = 0; pl < BITS; ++pl) { qA[pl] = at[pl * plane_gap]; qB[pl] = at[pl * plane_gap + row_gap]; }
                    const T* xb = sx + blk * 1024u + (ok ? 8u * lane : 0u);
                    uint4 X[4];
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) X[jj] = *reinterpret_cast<const uint4*>(xb + 8u * E * jj);
                    const uint32_t m = ok ? 0xffffffffu : 0u;
                    if constexpr (RAGGED.value) {
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) { X[jj].x &= m; X[jj].y &= m; X[jj].z &= m; X[jj].w &= m; }
                    }
                    if constexpr (LOOKUP) {
                        uint32_t WA[4][4], WB[4][4];
                        ap_lookup_word<BITS>(qA, lutA, WA);
                        ap_lookup_word<BITS>(qB, lutB, WB);
                        if constexpr (RAGGED.value) {
#pragma unroll
                            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                                for (int e = 0; e < 4; ++e) { WA[jj][e] &= m; WB[jj][e] &= m; }
                        }
                        __syncwarp();
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) {
                            mma_16816<DT>(acc[0], WA[jj][0], WB[jj][0], WA[jj][1], WB[jj][1], X[jj].x, X[jj].y);
                            mma_16816<DT>(acc[1], WA[jj][2], WB[jj][2], WA[jj][3], WB[jj][3], X[jj].z, X[jj].w);
                        }
                    } else {
                        if constexpr (RAGGED.value) {
#pragma unroll
                            for (int e = 0; e < 2; ++e) { tA.lo[e] &= m; tA.hi[e] &= m; tB.lo[e] &= m; tB.hi[e] &= m; }
                        }
                        uint32_t VA[4], VB[4];
                        ap_fields<3>(qA, VA);
                        ap_fields<3>(qB, VB);
#pragma unroll
                        for (int ph = 0; ph < 4; ++ph) {
                            uint32_t a3, a2, a1, a0, b3, b2, b1, b0;
                            tA.lookup(VA[ph], a3, a2);
                            tA.lookup(VA[ph] >> 16, a1, a0);
                            tB.lookup(VB[ph], b3, b2);
                            tB.lookup(VB[ph] >> 16, b1, b0);
                            mma_16816<DT>(acc[0], a3, b3, a2, b2, X[ph].x, X[ph].y);
                            mma_16816<DT>(acc[1], a1, b1, a0, b0, X[ph].z, X[ph].w);
                        }
                    }
                };
#pragma unroll (LOOKUP ? 1 : 2)
                for (uint32_t u = 0; u < full; ++u) step(u, IsRagged<false>{});
                if (full * 32u < nseg) step(full, IsRagged<true>{});
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * s);      // the stage (plane words and LUT rows) is no longer read
            if (diag && has_item && r0 + o < r1) {
                float* slot = part + ((size_t)o * geo.segs + seg) * 8u + g;
                slot[0] = odd ? acc[0][1] + acc[1][1] : acc[0][0] + acc[1][0];
                if (rowA + 1u < R && r0 + o + 1u < r1) slot[geo.segs * 8u] = odd ? acc[0][3] + acc[1][3] : acc[0][2] + acc[1][2];
            }
        }
    }
    if (warp == NW) pdl_wait();     // the producer warp touches the accumulator and y only from here on
    // fold the CTA's rows: a row's slots in order, one output per thread; y is read before the barrier so that the load
    // overlaps the last warps' work
    T* y = reinterpret_cast<T*>(f.y);
    const uint32_t nrows = r1 - r0;
    float y0 = 0.0f;
    if (geo.direct && (uint32_t)tid < nrows) y0 = Tr<DT>::to_f(y[r0 + tid]);
    __syncthreads();
    if (*s_abort && tid == 0) raise_error(f.err, 1u);
    if (geo.direct && *s_abort) return;      // an unfinished launch leaves y alone
    for (uint32_t i = tid; i < nrows; i += NT) {
        const float4* slots = reinterpret_cast<const float4*>(part + (size_t)i * geo.segs * 8u);
        float v = 0.0f;
        for (uint32_t e = 0; e < 2u * geo.segs; ++e) { const float4 q = slots[e]; v += (q.x + q.y) + (q.z + q.w); }
        if (geo.direct) y[r0 + i] = Tr<DT>::from_f((i == (uint32_t)tid ? y0 : Tr<DT>::to_f(y[r0 + i])) + v);
        else __stcg(f.acc + r0 + i, *s_abort ? 0.0f : v);
    }
    if (geo.direct) return;
    // fused launch: the sums went to the accumulator (this CTA is their only GEMV writer) and the CTA arrives on its
    // tile even after a failed wait, so that the workspace stays consistent
    arrive_and_finalize<DT>(f, cta, cta + 1, s_flag, NT);
}

}  // namespace dd
