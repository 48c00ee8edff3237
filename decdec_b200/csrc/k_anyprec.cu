// Any-precision launches (entry points `anyprec_gemv`, `dec_anyprec`, `anyprec_dequant`).
#include "internal.h"
#include <cstdlib>
#include "dec_role.cuh"
#include "gemv_anyprec_pipe.cuh"

namespace dd {

template <int DT, bool FAST3>
__global__ void __launch_bounds__(kThreads)
k_anyprec(const __grid_constant__ ApParams g, const __grid_constant__ DecParams d, const __grid_constant__ FinParams f) {
    extern __shared__ __align__(128) unsigned char sm[];
    if (blockIdx.x < d.n_cta) dec_role<DT>(d, f, blockIdx.x, sm);
    else if constexpr (FAST3) ap3_role<DT>(g, f, blockIdx.x - d.n_cta, sm);
    else apg_role<DT>(g, f, blockIdx.x - d.n_cta, sm);
}

size_t anyprec_smem(uint32_t K, bool fast3) {
    const size_t xb = ((size_t)K * 2 + 15) & ~(size_t)15;
    return fast3 ? xb + 16 : xb + 8 * 256 * 2 + 16;
}

template <int DT, bool FAST3>
static cudaError_t go(const ApParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    size_t smem = anyprec_smem(g.K, FAST3);
    if (d.n_cta && smem < (size_t)DecSmem::kBytes) smem = DecSmem::kBytes;
    static size_t configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > 48 * 1024 && dev < 64 && configured[dev] < smem) {
        cudaError_t e = cudaFuncSetAttribute(k_anyprec<DT, FAST3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured[dev] = smem;
    }
    k_anyprec<DT, FAST3><<<d.n_cta + g.n_cta, kThreads, smem, s>>>(g, d, f);
    return cudaGetLastError();
}

cudaError_t launch_anyprec(int dt, const ApParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    const bool fast3 = g.bits == 3 && (g.K % 128u) == 0u;
    if (dt == FP16) return fast3 ? go<FP16, true>(g, d, f, s) : go<FP16, false>(g, d, f, s);
    return fast3 ? go<BF16, true>(g, d, f, s) : go<BF16, false>(g, d, f, s);
}

template <int DT, int BITS>
__global__ void __launch_bounds__(kApPipeThreads, 1)
k_anyprec_pipe(const __grid_constant__ ApParams g, const __grid_constant__ DecParams d, const __grid_constant__ FinParams f,
               const __grid_constant__ ApPipeGeom geo) {
    extern __shared__ __align__(256) unsigned char sm[];     // the warps' LUT rows are aligned to kApLutStride
    if (blockIdx.x < d.n_cta) dec_role<DT>(d, f, blockIdx.x, sm);
    else ap_pipe_role<DT, BITS>(g, f, geo, blockIdx.x - d.n_cta, sm);
}

// Stage geometry of the pipelined kernel (3 to 8 bits); false if the shape is not eligible.  A CTA's rows are a whole
// number of 32-output finalizer tiles when a compensation role may share the launch; a GEMV-only launch (no config)
// has no finalizer and cuts the rows in pairs, which fills the SMs evenly (us at 3 bits, rows in multiples of 16 -> in pairs:
// 768 x 4096 3.94 -> 3.31, 1000 x 2176 4.00 -> 3.28, 4096 x 14336 14.65 -> 13.52, 28672 x 4096 23.53 -> 23.36).
bool anyprec_pipe_geometry(uint32_t N, uint32_t K, uint32_t bits, ApPipeGeom* geo, uint32_t sm_budget, bool gemv_only) {
    if (bits < 3 || bits > 8 || K % 128u || K > 32768u || N == 0) return false;
    const uint32_t rowbytes = K / 8;
    const uint32_t per_row = bits * rowbytes + (2u << bits);      // plane words and the LUT row
    geo->x_bytes = (K * 2 + 127u) & ~127u;
    if (sm_budget == 0) sm_budget = 1;
    uint32_t rows = (N + sm_budget - 1) / sm_budget;
    const uint32_t gran = gemv_only ? 2u : 32u;
    rows = ((rows + gran - 1) / gran) * gran;
    geo->rows_per_cta = rows;
    const bool own_luts = bits > 3 && bits < 8;
    const uint32_t lut_bytes = own_luts ? 16u * 2u * kApLutStride + kApLutStride : 0u;   // 16 warps, and room for the alignment
    // Cut of a stage over the 16 warps: rows in pairs, a row's 1024-channel blocks in `segs` segments.  A stage costs its
    // warps the blocks of a segment plus about 0.8 of a block for the wait, the tables and the sums; long segments spread
    // that best, short ones fill the warps when the CTA has few rows (and leave room for two stages of wide rows).
    const uint32_t nblk = (K + 1023u) / 1024u;
    uint32_t best = 0xffffffffu;
    for (uint32_t want = 1; want <= 16; ++want) {
        const uint32_t blocks = (nblk + want - 1) / want, segs = (nblk + blocks - 1) / blocks;
        const uint32_t part = (rows * segs * 32u + 127u) & ~127u;
        const uint32_t fixed = kApPipeHdr + geo->x_bytes + part + lut_bytes;
        if (segs > 16 || fixed >= 227u * 1024u) continue;
        const uint32_t budget = 227u * 1024u - fixed;
        uint32_t R = 2u * (16u / segs);
        while (R & (R - 1)) R &= R - 1;
        while (R > 2 && R / 2 >= rows) R >>= 1;
        // wide rows: fewer rows per stage until two stages fit (some consumer warps then have no work item)
        while (R > 1 && 2u * ((R * per_row + 127u) & ~127u) > budget) R >>= 1;
        const uint32_t stage = (R * per_row + 127u) & ~127u;
        if (2u * stage > budget) continue;
        const uint32_t nst = (rows + R - 1) / R;
        const uint32_t cost = nst * (10u * blocks + 8u);
        if (cost >= best) continue;
        best = cost;
        uint32_t smax = budget / stage;
        if (smax > 8) smax = 8;
        geo->segs = segs;
        geo->seg_words = 32u * blocks;
        geo->part_bytes = part;
        geo->rows_per_stage = R;
        geo->stage_bytes = stage;
        geo->stages = nst < smax ? nst : smax;
        const uint32_t end = kApPipeHdr + geo->x_bytes + part + geo->stages * stage;
        geo->lut_off = (end + kApLutStride - 1u) & ~(kApLutStride - 1u);
        geo->smem_bytes = own_luts ? geo->lut_off + 16u * 2u * kApLutStride : end;
    }
    if (best == 0xffffffffu) return false;
    geo->direct = 0;        // set by the caller
    {
        const char* w = getenv("DECDEC_PIPE_WAIT_NS");
        geo->wait_ns = (w && *w) ? (uint32_t)strtoul(w, nullptr, 10) : 50u * 1000u * 1000u;
    }
    if (geo->smem_bytes < (uint32_t)DecSmem::kBytes) geo->smem_bytes = DecSmem::kBytes;
    return true;
}

template <int DT, int BITS>
static cudaError_t go_pipe(const ApParams& g, const DecParams& d, const FinParams& f, const ApPipeGeom& geo, cudaStream_t s) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_anyprec_pipe<DT, BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    // programmatic dependent launch: thread blocks may become resident (and prefetch weights) while the
    // previous kernel of the stream drains; the kernel waits for it before touching activations or outputs
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.n_cta + g.n_cta);
    cfg.blockDim = dim3(kApPipeThreads);
    cfg.dynamicSmemBytes = geo.smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    const char* e = getenv("DECDEC_PDL");
    attr[0].val.programmaticStreamSerializationAllowed = (e && *e == '0') ? 0 : 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_anyprec_pipe<DT, BITS>, g, d, f, geo);
}

template <int DT>
static cudaError_t pipe_by_bits(const ApParams& g, const DecParams& d, const FinParams& f, const ApPipeGeom& geo, cudaStream_t s) {
    switch (g.bits) {
        case 3: return go_pipe<DT, 3>(g, d, f, geo, s);
        case 4: return go_pipe<DT, 4>(g, d, f, geo, s);
        case 5: return go_pipe<DT, 5>(g, d, f, geo, s);
        case 6: return go_pipe<DT, 6>(g, d, f, geo, s);
        case 7: return go_pipe<DT, 7>(g, d, f, geo, s);
        case 8: return go_pipe<DT, 8>(g, d, f, geo, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_anyprec_pipe(int dt, const ApParams& g, const DecParams& d, const FinParams& f, const ApPipeGeom& geo, cudaStream_t s) {
    return dt == FP16 ? pipe_by_bits<FP16>(g, d, f, geo, s) : pipe_by_bits<BF16>(g, d, f, geo, s);
}

template <int DT, int BITS>
static void dequant_bits(int blocks, const uint32_t* qweight, const void* lut, void* out, uint32_t N, uint32_t K, cudaStream_t s) {
    if constexpr (BITS <= 4) {
        if ((reinterpret_cast<uintptr_t>(lut) & 15u) == 0u) {        // the table rows are read with 16-byte loads
            ap_dequant_kernel<DT, BITS, true><<<blocks, kThreads, 0, s>>>(qweight, lut, out, N, K);
            return;
        }
    }
    ap_dequant_kernel<DT, BITS, false><<<blocks, kThreads, 0, s>>>(qweight, lut, out, N, K);
}

template <int DT>
static void dequant_dt(int blocks, const uint32_t* qweight, const void* lut, void* out, uint32_t N, uint32_t K, uint32_t bits, cudaStream_t s) {
    switch (bits) {
        case 3: dequant_bits<DT, 3>(blocks, qweight, lut, out, N, K, s); break;
        case 4: dequant_bits<DT, 4>(blocks, qweight, lut, out, N, K, s); break;
        case 5: dequant_bits<DT, 5>(blocks, qweight, lut, out, N, K, s); break;
        case 6: dequant_bits<DT, 6>(blocks, qweight, lut, out, N, K, s); break;
        case 7: dequant_bits<DT, 7>(blocks, qweight, lut, out, N, K, s); break;
        default: dequant_bits<DT, 8>(blocks, qweight, lut, out, N, K, s); break;
    }
}

cudaError_t launch_ap_dequant(int dt, const uint32_t* qweight, const void* lut, void* out, uint32_t N, uint32_t K,
                              uint32_t bits, cudaStream_t s) {
    const size_t total = (size_t)N * (K / 32);
    const int blocks = (int)((total + kThreads - 1) / kThreads < 148 * 16 ? (total + kThreads - 1) / kThreads : 148 * 16);
    if (blocks == 0) return cudaSuccess;
    if (dt == FP16) dequant_dt<FP16>(blocks, qweight, lut, out, N, K, bits, s);
    else dequant_dt<BF16>(blocks, qweight, lut, out, N, K, bits, s);
    return cudaGetLastError();
}

}  // namespace dd
