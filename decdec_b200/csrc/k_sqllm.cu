// SqueezeLLM launches (entry points `sqllm_gemv`, `dec_sqllm`).
#include "internal.h"
#include <cstdlib>
#include "dec_role.cuh"
#include "gemv_sqllm_pair.cuh"

namespace dd {

template <int DT>
__global__ void __launch_bounds__(kThreads, 3)
k_sqllm(const __grid_constant__ SqParams g, const __grid_constant__ DecParams d, const __grid_constant__ FinParams f) {
    extern __shared__ __align__(128) unsigned char sm[];
    if (blockIdx.x < d.n_cta) dec_role<DT>(d, f, blockIdx.x, sm);
    else sq_role<DT>(g, f, blockIdx.x - d.n_cta, sm);
}

size_t sqllm_smem(uint32_t K) { return (((size_t)K * 4 + 15) & ~(size_t)15) + (16 * 32 + 8 * 32) * 4 + 16; }

template <int DT>
static cudaError_t go(const SqParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    size_t smem = sqllm_smem(g.K);
    if (d.n_cta && smem < (size_t)DecSmem::kBytes) smem = DecSmem::kBytes;
    static size_t configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (smem > 48 * 1024 && dev < 64 && configured[dev] < smem) {
        cudaError_t e = cudaFuncSetAttribute(k_sqllm<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        configured[dev] = smem;
    }
    k_sqllm<DT><<<d.n_cta + g.n_cta, kThreads, smem, s>>>(g, d, f);
    return cudaGetLastError();
}

cudaError_t launch_sqllm(int dt, const SqParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    switch (dt) {
        case FP32: return go<FP32>(g, d, f, s);
        case FP16: return go<FP16>(g, d, f, s);
        default: return go<BF16>(g, d, f, s);
    }
}

// DEC: the launch has a compensation role (its register needs would otherwise be paid for by every launch)
template <int DT, int BITS, bool DEC>
__global__ void __launch_bounds__(kSqPairThreads, 2)
k_sqllm_pair(const __grid_constant__ SqParams g, const __grid_constant__ DecParams d, const __grid_constant__ FinParams f) {
    extern __shared__ __align__(128) unsigned char sm[];
    if (DEC && blockIdx.x < d.n_cta) dec_role<DT>(d, f, blockIdx.x, sm);
    else sq_pair_role<DT, BITS>(g, f, blockIdx.x - d.n_cta, sm);
}

template <int DT, int BITS, bool DEC>
static cudaError_t go_pair_dec(const SqParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    size_t smem = sq_pair_smem(g.part_groups, g.bits);
    if (DEC && smem < (size_t)DecSmem::kBytes) smem = DecSmem::kBytes;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_sqllm_pair<DT, BITS, DEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    // programmatic dependent launch: the thread blocks become resident while the previous kernel of the stream drains
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.n_cta + g.n_cta);
    cfg.blockDim = dim3(kSqPairThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    const char* e = getenv("DECDEC_PDL");
    attr[0].val.programmaticStreamSerializationAllowed = (e && (*e == '0' || (*e == '1' && DEC))) ? 0 : 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_sqllm_pair<DT, BITS, DEC>, g, d, f);
}

template <int DT, int BITS>
static cudaError_t go_pair(const SqParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    return d.n_cta ? go_pair_dec<DT, BITS, true>(g, d, f, s) : go_pair_dec<DT, BITS, false>(g, d, f, s);
}

// (shared memory: the 50 000 channels that run_sqllm takes need 166 KB in one part)
bool sqllm_pair_eligible(const void* qweight, const void* lut, uint32_t N, int dt) {
    int dev = 0, reserved = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess) { cudaGetLastError(); return false; }
    return (uint32_t)reserved == kSqTableBase && dt != FP32 && N % 2u == 0u && (reinterpret_cast<uintptr_t>(qweight) & 7u) == 0u &&
           (reinterpret_cast<uintptr_t>(lut) & 15u) == 0u;
}

cudaError_t launch_sqllm_pair(int dt, const SqParams& g, const DecParams& d, const FinParams& f, cudaStream_t s) {
    if (g.bits == 4) return dt == FP16 ? go_pair<FP16, 4>(g, d, f, s) : go_pair<BF16, 4>(g, d, f, s);
    return dt == FP16 ? go_pair<FP16, 3>(g, d, f, s) : go_pair<BF16, 3>(g, d, f, s);
}

}  // namespace dd
