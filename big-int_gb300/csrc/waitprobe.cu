// waitprobe.cu -- what a wait that runs out does, for the tests: the kernels with
// bounded waits on a barrier that never completes, so that their own limit ends
// them.  Nothing else about them differs; the device stays usable.
#include "multc.cuh"

namespace bi {

struct HeldItem {
    const uint64_t *pa, *pb;
    uint64_t* pr;
    uint32_t L, out_limbs;
    __device__ __forceinline__ uint64_t a(uint32_t x) const { return pa[x]; }
    __device__ __forceinline__ uint64_t b(uint32_t x) const { return pb[x]; }
    __device__ __forceinline__ void store(uint32_t x, uint64_t v) const { pr[x] = v; }
};

__global__ void __launch_bounds__(TcShape<32>::THREADS, 1)
held_products_kernel(const uint64_t* a, const uint64_t* b, uint64_t* r, uint32_t m, uint64_t n, TcGeom g,
                     uint32_t* gave_up) {
    extern __shared__ __align__(128) uint8_t smem_tc[];
    tc_products<32, 1>(g, smem_tc, blockIdx.x, gridDim.x, n, gave_up, [&](uint64_t i) {
        return HeldItem{a + i * m, b + i * m, r + i * 2 * m, m, 2 * m};
    });
}

static bi_status held_products(const uint64_t* a, const uint64_t* b, uint64_t* r, uint32_t m, uint64_t n,
                               uint32_t* gave_up, cudaStream_t st) {
    TcGeom g = {};
    tc_geometry_add<32>(g, m, 2 * m);
    g.NA = 2;
    const size_t smem = TcSmem<32>(g).total;
    cudaError_t e = smem_opt_in((const void*)held_products_kernel, smem);
    if (e != cudaSuccess) return set_error(BI_ECUDA, "held wait: %s", cudaGetErrorString(e));
    held_products_kernel<<<2, TcShape<32>::THREADS, smem, st>>>(a, b, r, m, n, g, gave_up);
    return check_launch("held products kernel");
}

}  // namespace bi

using namespace bi;

extern "C" bi_status bi_probe_held_wait(int kind, const uint64_t* a, const uint64_t* b, uint64_t* r, uint8_t* status,
                                        uint32_t m, uint64_t n, bi_stream s) {
    if (!a || !b || !r || n < 2 || n > 64 || m < 1 || m > 128) return set_error(BI_EINVAL, "held wait: bad arguments");
    BI_RETURN_IF(waits_ok());
    uint32_t* gave_up;
    BI_RETURN_IF(gave_up_word(&gave_up));
    if (kind == 0) return held_products(a, b, r, m, n, gave_up, (cudaStream_t)s);
    if (kind == 1) {
        if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)r) % 16) return set_error(BI_EINVAL, "held wait: buffers off a 16-byte boundary");
        return ragged_held(a, b, r, status, m, n, gave_up, (cudaStream_t)s);
    }
    if (kind == 2) return div_held(a, b, r, r + 2 * m * n, status, 2 * m, m, n, gave_up, (cudaStream_t)s);
    return set_error(BI_EINVAL, "held wait: no kind %d", kind);
}
