// SqueezeLLM GEMV role for 16-bit layers: pair tables in shared memory, products on the tensor cores.
//
// Bound: shared-memory wavefronts.  A byte of a 4-bit word (6 bits of a 3-bit string) names the weights of two neighbouring
// channels, so a table of the 2^(2 bits) possible PAIRS per column turns two weights into one lookup.  Entry e of table slot s
// sits at byte e * 256 + s * 4: with 64 columns per tile the lookup address is one byte permute of the word (4 bits) or a
// shift and a logic operation (3 bits), and the 32 lanes of a warp, which each own a slot, always hit 32 different banks.
// The products go through mma.m16n8k16 (16-bit factors, fp32 sums): lane (g, t) = (lane / 4, lane % 4) owns columns 2 * lane and
// 2 * lane + 1 of the tile; its pairs are k positions {2t, 2t+1, 2t+8, 2t+9} of rows g and g + 8 of A, and column t' of B
// holds the activations at the k positions of t = t' and zero elsewhere (the lanes with g == t carry them, the others carry
// zeros), so that D[g][t'] is the sum of the column that lane (g, t') owns.  One instruction consumes eight weights per lane;
// fp32 multiply-adds would need eight, and eight conversions.  A zero of B times an infinite or NaN weight would
// spread to the quad's other columns: a tile whose tables hold such a value is summed with fp32 multiply-adds instead.
//
// Split of the work.  The (64-column tile, 32-channel group) units are one line that is cut evenly over the thread blocks.  Where it
// pays their number is a multiple of the tiles' (host.cu:sqllm_pair_blocks), so that a thread block has one part and one table to
// build.  A thread block has at most two cut parts, its first and its last: a cut part's sums go to a place of their own in the workspace, and
// the part takes a ticket of the tile with the number of groups it covered; whoever brings the tickets to K / 32 adds the
// parts in the order of their channels, so that equal calls give equal bits.  The sums of a tile are then added to y, or, beside a
// compensation role, stored in the accumulator with one arrival on the tile (common.cuh).
// The launch may become resident while the previous kernel of the stream drains, but reads nothing before that one has
// completed: codes and centroids may come from it.  (Tables and first words ahead of the wait were worth 1.0 to 1.6 us per launch.)
//
// Measured, 4 bits, fp16, us per launch in a graph, against one lookup, one conversion and one fp32 multiply-add per weight: 28672 x 4096
// 35.6 -> 25.1, 4096 x 14336 32.4 -> 14.3, and the eight linears of two 8B blocks 187 -> 115.6 (125 with the even cut).  What is left over the wavefronts (20 000 cycles of a 28672 x 4096 launch) is the latency of a part's start (tables, first words) and end
// (sums of the warps): two thread blocks per SM overlap them (180 us with one).
#pragma once
#include "common.cuh"
#include "gemv_sqllm.cuh"

namespace dd {

constexpr int kSqPairThreads = 384;                       // two thread blocks per SM, 80 registers
constexpr uint32_t kSqTileN = 64;                         // columns per tile = 4-byte slots of a 256-byte table row
constexpr uint32_t kSqPartBytes = (kSqPairThreads / 32) * kSqTileN * 4;

__host__ __device__ inline uint32_t sq_pair_table_bytes(uint32_t bits) { return 256u << (2u * bits); }
// tables, activations of the longest part, partial sums of the warps, flag
__host__ __device__ inline uint32_t sq_pair_smem(uint32_t part_groups, uint32_t bits) {
    return sq_pair_table_bytes(bits) + part_groups * 64u + kSqPartBytes + 16u;
}
// groups of the longest part when `units` are cut over n_cta thread blocks
inline uint32_t sq_pair_part_groups(uint64_t units, uint32_t n_cta, uint32_t groups) {
    const uint64_t share = (units + n_cta - 1u) / n_cta;
    return share < groups ? (uint32_t)share : groups;
}

__device__ __forceinline__ uint2 ldg_stream(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
// Tables start where dynamic shared memory does: kSqTableBase bytes into the shared window (checked), so that the offset of an
// entry is its address but for a constant that the load instruction adds.
constexpr uint32_t kSqTableBase = 1024;
__device__ __forceinline__ uint32_t sq_table_at(uint32_t off) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(off), "n"(kSqTableBase));
    return v;
}

// the words of a 32-channel group of the two columns a lane owns
template <int WR>
__device__ __forceinline__ void sq_pair_load(const uint32_t* __restrict__ col, uint32_t N, uint32_t g, uint2 (&w)[WR]) {
    const uint32_t* at = col + (size_t)(WR * g) * N;
#pragma unroll
    for (int i = 0; i < WR; ++i) w[i] = ldg_stream(reinterpret_cast<const uint2*>(at + (size_t)i * N));
}

// sums of the two columns a lane owns over the groups [g0 + warp, g1) in steps of the warp count; w0 and w1 hold the first two
// FINITE: tensor-core form (see above); the sums of a quad end in its lanes t = 0 and 1.
template <int DT, int BITS, bool FINITE>
__device__ __forceinline__ void sq_pair_sums(const uint32_t* __restrict__ col, uint32_t N, uint32_t g0, uint32_t g1,
                                             const unsigned char* sx, uint2 (&w0)[BITS], uint2 (&w1)[BITS], float (&acc)[2][4]) {
    constexpr uint32_t NW = kSqPairThreads / 32;
    constexpr int WR = BITS;                                // word rows per 32-channel group
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t own = (lane >> 2) == (lane & 3) ? 0xffffffffu : 0u;
    const uint32_t slotA = lane * 4, slotB = slotA + 128;           // column 2 * lane in slot lane, the other in slot lane + 32
    auto load = [&](uint32_t g, uint2 (&w)[WR]) { sq_pair_load<WR>(col, N, g, w); };
    // table entry of pair p (channels 2p, 2p + 1) of a group's words
    auto entry = [&](const uint32_t* w, int p, uint32_t slot) -> uint32_t {
        uint32_t off;
        if constexpr (BITS == 4) {
            off = __byte_perm(w[p >> 2], slot, 0x5504u | ((uint32_t)(p & 3) << 4));
        } else {
            const int bit = 6 * p;                          // of the 96-bit string; the six bits move to bits 8..13
            const int wi = bit >> 5, r = bit & 31;
            uint32_t v;
            if (r + 6 > 32) v = __funnelshift_r(w[wi], w[wi + 1], r) << 8;
            else v = r >= 8 ? w[wi] >> (r - 8) : w[wi] << (8 - r);
            off = (v & 0x3f00u) | slot;
        }
        return sq_table_at(off);
    };
    auto consume = [&](uint32_t g, const uint2 (&w)[WR]) {
        uint32_t wA[WR], wB[WR];
#pragma unroll
        for (int i = 0; i < WR; ++i) { wA[i] = w[i].x; wB[i] = w[i].y; }
        const uint4* xg = reinterpret_cast<const uint4*>(sx + (g - g0) * 64u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {                       // eight channels; one address for the warp: one wavefront
            const uint4 X = xg[i];
            const uint32_t x[4] = {X.x, X.y, X.z, X.w};
#pragma unroll
            for (int h = 0; h < 2; ++h) {                   // four channels
                const int p = 4 * i + 2 * h;
                const uint32_t a0 = entry(wA, p, slotA), a1 = entry(wB, p, slotB);
                const uint32_t a2 = entry(wA, p + 1, slotA), a3 = entry(wB, p + 1, slotB);
                if constexpr (FINITE) {
                    mma_16816<DT>(acc[h], a0, a1, a2, a3, x[2 * h] & own, x[2 * h + 1] & own);
                } else {
                    const float2 x0 = unpack2<DT>(x[2 * h]), x1 = unpack2<DT>(x[2 * h + 1]);
                    const float2 p0 = unpack2<DT>(a0), p1 = unpack2<DT>(a1), p2 = unpack2<DT>(a2), p3 = unpack2<DT>(a3);
                    acc[0][0] = fmaf(p2.y, x1.y, fmaf(p2.x, x1.x, fmaf(p0.y, x0.y, fmaf(p0.x, x0.x, acc[0][0]))));
                    acc[0][1] = fmaf(p3.y, x1.y, fmaf(p3.x, x1.x, fmaf(p1.y, x0.y, fmaf(p1.x, x0.x, acc[0][1]))));
                }
            }
        }
    };
    // a group's words are asked for again as soon as they are used up: one to two groups (0.75 to 2 KB) in flight per warp
    uint32_t g = g0 + warp;
#pragma unroll 1
    for (; g + NW < g1; g += 2 * NW) {
        consume(g, w0);
        if (g + 2 * NW < g1) load(g + 2 * NW, w0);
        consume(g + NW, w1);
        if (g + 3 * NW < g1) load(g + 3 * NW, w1);
    }
    if (g < g1) consume(g, w0);
}

// Sums of the 64 columns of a tile whose parts lie in the workspace, in the order of the channels: v of thread tid < 64.
// Thread block c covers units [units * c / n_cta, units * (c + 1) / n_cta); its first part is at slot 2 c, a last part that starts
// with a tile of its own at slot 2 c + 1.
__device__ __forceinline__ float sq_pair_join(const SqParams& p, uint32_t tile, uint32_t groups, uint64_t units) {
    const uint64_t u0 = (uint64_t)tile * groups;
    const uint32_t c0 = (uint32_t)(((u0 + 1) * p.n_cta - 1) / units), c1 = (uint32_t)(((u0 + groups) * p.n_cta - 1) / units);
    const float* at = p.parts + (size_t)c0 * 2u * kSqTileN + (units * c0 / p.n_cta == u0 ? 0u : kSqTileN) + threadIdx.x;
    float v = __ldcg(at);
    at = p.parts + threadIdx.x;
    constexpr uint32_t U = 4;                               // loads in flight
    for (uint32_t c = c0 + 1; c <= c1; c += U) {
        float q[U];
#pragma unroll
        for (uint32_t i = 0; i < U; ++i) q[i] = c + i <= c1 ? __ldcg(at + (size_t)(c + i) * 2u * kSqTileN) : 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < U; ++i) if (c + i <= c1) v += q[i];
    }
    return v;
}

template <int DT, int BITS>
__device__ void sq_pair_role(const SqParams& p, const FinParams& f, uint32_t cta, unsigned char* sm) {
    using T = typename Tr<DT>::T;
    static_assert(DT != FP32, "16-bit layers");
    constexpr uint32_t NC = 1u << BITS;                     // centroids per column
    constexpr uint32_t NW = kSqPairThreads / 32;
    const uint32_t tbytes = sq_pair_table_bytes(BITS);
    T* sx = reinterpret_cast<T*>(sm + tbytes);
    float* part = reinterpret_cast<float*>(sm + tbytes + p.part_groups * 64u);
    unsigned* s_flag = reinterpret_cast<unsigned*>(reinterpret_cast<unsigned char*>(part) + kSqPartBytes);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t groups = p.K / 32;
    const T* x = reinterpret_cast<const T*>(p.x);
    T* y = reinterpret_cast<T*>(f.y);

    const uint64_t units = (uint64_t)f.n_tiles * groups;
    const uint64_t ubegin = units * cta / p.n_cta;
    uint64_t u = ubegin;
    const uint64_t uend = units * (cta + 1) / p.n_cta;
    pdl_trigger();
    if ((uint32_t)__cvta_generic_to_shared(sm) != kSqTableBase) {     // not the layout the launch was made for: nothing is computed
        if (tid == 0) raise_error(f.err, 2u);
        return;
    }
    pdl_wait();
    while (u < uend) {
        const uint32_t tile = (uint32_t)(u / groups), g0 = (uint32_t)(u % groups);
        const uint32_t g1 = (uint32_t)(uend - (uint64_t)tile * groups < groups ? uend - (uint64_t)tile * groups : groups);
        const uint32_t n0 = tile * kSqTileN;
        // the first words are on their way while the tables are built
        const uint32_t n = n0 + 2u * lane;
        const uint32_t* col = p.qweight + min(n, p.N - 2u);     // a lane beyond the last column reads that one; its table is zero
        uint2 w0[BITS], w1[BITS];
        if (g0 + warp < g1) sq_pair_load<BITS>(col, p.N, g0 + warp, w0);
        if (g0 + warp + NW < g1) sq_pair_load<BITS>(col, p.N, g0 + warp + NW, w1);
        // ---- pair tables of the tile: thread -> slot (columns 2 * slot of the first 32, 2 * slot + 1 of the others), every
        // sixth high code
        bool bad = false;
        {
            const uint32_t slot = tid & 63u;
            const uint32_t c = 2u * (slot & 31u) + (slot >> 5);
            uint32_t pr[NC / 2];                            // the column's centroids, two per register
            const bool ok = n0 + c < p.N;
            const uint4* row = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.lut) + (size_t)(n0 + c) * NC);
#pragma unroll
            for (uint32_t i = 0; i < NC / 8; ++i) {
                const uint4 r = ok ? __ldg(row + i) : make_uint4(0u, 0u, 0u, 0u);
                pr[4 * i] = r.x; pr[4 * i + 1] = r.y; pr[4 * i + 2] = r.z; pr[4 * i + 3] = r.w;
            }
            constexpr uint32_t kExp = DT == FP16 ? 0x7c00u : 0x7f80u;
#pragma unroll
            for (uint32_t i = 0; i < NC / 2; ++i) bad |= (pr[i] & kExp) == kExp || ((pr[i] >> 16) & kExp) == kExp;
            uint32_t* dst = reinterpret_cast<uint32_t*>(sm) + slot;
#pragma unroll
            for (uint32_t hi = 0; hi < NC; ++hi) {
                if (hi % (kSqPairThreads / 64) != tid / 64u) continue;
                const uint32_t hv = (hi & 1u) ? pr[hi / 2] >> 16 : pr[hi / 2] & 0xffffu;
#pragma unroll
                for (uint32_t lo = 0; lo < NC; ++lo)
                    dst[(hi * NC + lo) * 64u] = __byte_perm(pr[lo / 2], hv, (lo & 1u) ? 0x5432u : 0x5410u);
            }
        }
        for (uint32_t k = tid; k < (g1 - g0) * 32u; k += kSqPairThreads) sx[k] = x[g0 * 32u + k];
        const bool finite = !__syncthreads_or(bad);

        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        if (finite) {
            sq_pair_sums<DT, BITS, true>(col, p.N, g0, g1, sm + tbytes, w0, w1, acc);
            if ((lane & 3u) < 2u) {
                // lane (g, t): D columns 2t and 2t + 1 = the sums of lanes 4g + 2t and 4g + 2t + 1
                const uint32_t L = (lane & ~3u) + 2u * (lane & 3u);
                *reinterpret_cast<float4*>(part + warp * kSqTileN + 2u * L) =
                    make_float4(acc[0][0] + acc[1][0], acc[0][2] + acc[1][2], acc[0][1] + acc[1][1], acc[0][3] + acc[1][3]);
            }
        } else {
            sq_pair_sums<DT, BITS, false>(col, p.N, g0, g1, sm + tbytes, w0, w1, acc);
            *reinterpret_cast<float2*>(part + warp * kSqTileN + 2u * lane) = make_float2(acc[0][0], acc[0][1]);
        }
        __syncthreads();
        const bool whole = g1 - g0 == groups, mine = tid < kSqTileN && n0 + tid < p.N;
        float v = 0.0f;
        if (tid < kSqTileN) {
#pragma unroll
            for (uint32_t w = 0; w < NW; ++w) v += part[w * kSqTileN + tid];
        }
        bool joined = whole;
        if (!whole) {
            if (tid < kSqTileN) __stcg(p.parts + (2u * cta + (u == ubegin ? 0u : 1u)) * kSqTileN + tid, v);
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                const bool last = atomicAdd(p.part_tickets + tile, g1 - g0) + (g1 - g0) == groups;
                if (last) p.part_tickets[tile] = 0u;
                *s_flag = last;
            }
            __syncthreads();
            joined = *s_flag != 0u;
            if (joined && tid < kSqTileN) {
                __threadfence();
                v = sq_pair_join(p, tile, groups, units);
            }
        }
        if (joined) {
            if (p.direct) {
                if (mine) y[n0 + tid] = Tr<DT>::from_f(Tr<DT>::to_f(y[n0 + tid]) + v);
            } else {
                if (mine) __stcg(f.acc + n0 + tid, v);
                arrive_and_finalize<DT>(f, tile, tile + 1, s_flag, kSqPairThreads);
            }
        }
        u = (uint64_t)tile * groups + g1;
    }
}

}  // namespace dd
