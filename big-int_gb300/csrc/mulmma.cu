// mulmma.cu -- uniform batches of medium products on one warp an instance
// (mulmma.cuh); mul.cu decides which products come here.
#include "mulmma.cuh"

namespace bi {

struct MmRow {                         // an instance of a uniform batch, 64-bit limbs or 32-bit words
    const void *pa, *pb;
    void* pr;
    uint32_t m, out, L, out_limbs;
    bool w32, vec;                     // vec: 64-bit limbs, an even count, 16-byte aligned
    __device__ __forceinline__ uint64_t limb(const void* p, uint32_t x) const {
        if (!w32) return static_cast<const uint64_t*>(p)[x];
        const uint32_t* w = static_cast<const uint32_t*>(p);
        return w[2 * x] | (2 * x + 1 < m ? (uint64_t)w[2 * x + 1] << 32 : 0ull);
    }
    __device__ __forceinline__ uint64_t a(uint32_t x) const { return limb(pa, x); }
    __device__ __forceinline__ uint64_t b(uint32_t x) const { return limb(pb, x); }
    __device__ __forceinline__ ulonglong2 a2(uint32_t x) const { return *reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(pa) + x); }
    __device__ __forceinline__ ulonglong2 b2(uint32_t x) const { return *reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(pb) + x); }
    __device__ __forceinline__ void store2(uint32_t x, uint64_t v, uint64_t w) const {
        *reinterpret_cast<ulonglong2*>(static_cast<uint64_t*>(pr) + x) = make_ulonglong2(v, w);
    }
    __device__ __forceinline__ void store(uint32_t x, uint64_t v) const {
        if (!w32) {
            static_cast<uint64_t*>(pr)[x] = v;
            return;
        }
        uint32_t* w = static_cast<uint32_t*>(pr);
        if (2 * x < out) w[2 * x] = (uint32_t)v;
        if (2 * x + 1 < out) w[2 * x + 1] = (uint32_t)(v >> 32);
    }
};

template <int LT, bool FULL>
__global__ void __launch_bounds__(MM_CTA)
mul_mma_kernel(const void* a, const void* b, void* r, uint64_t n, uint32_t m, bool w32, bool vec) {
    extern __shared__ __align__(16) uint32_t smem_mm[];
    using S = MmShape<LT, FULL>;
    uint32_t* sw = smem_mm + (threadIdx.x >> 5) * S::WORDS;
    const uint32_t out = FULL ? 2 * m : m, wb = w32 ? 4 : 8;
    const uint32_t L = w32 ? (m + 1) / 2 : m, ol = w32 ? (out + 1) / 2 : out;
    const uint64_t warps = (uint64_t)gridDim.x * (MM_CTA / 32);
    auto row = [&](uint64_t i) {
        return MmRow{static_cast<const uint8_t*>(a) + i * m * wb, static_cast<const uint8_t*>(b) + i * m * wb,
                     static_cast<uint8_t*>(r) + i * out * wb, m, out, L, ol, w32, vec};
    };
    uint64_t i = (uint64_t)blockIdx.x * (MM_CTA / 32) + (threadIdx.x >> 5);
    if (i >= n) return;
    MmLimbs<S::E> cur;
    cur.load(row(i));
    if constexpr (S::E <= 4) {         // the next instance's limbs load under this one's product
        for (;;) {
            MmLimbs<S::E> next;
            const uint64_t j = i + warps;
            next.load(row(j < n ? j : i));
            mm_product<LT, FULL>(row(i), cur, sw);
            if (j >= n) break;
            i = j;
            cur = next;
        }
    } else {
        for (;;) {
            mm_product<LT, FULL>(row(i), cur, sw);
            i += warps;
            if (i >= n) break;
            cur.load(row(i));
        }
    }
}

template <int LT, bool FULL>
static bi_status launch(const void* a, const void* b, void* r, uint32_t m, uint64_t n, bool w32, cudaStream_t st) {
    const size_t smem = MmShape<LT, FULL>::WORDS * 4 * (MM_CTA / 32);
    auto kern = mul_mma_kernel<LT, FULL>;
    static const int occ = [&] {
        int o = 0;
        if (smem_opt_in((const void*)kern, smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, MM_CTA, smem) != cudaSuccess) {
            cudaGetLastError();                // not the launch's error: grid one CTA an SM
            o = 1;
        }
        return o > 0 ? o : 1;
    }();
    cudaError_t e = smem_opt_in((const void*)kern, smem);
    if (e != cudaSuccess) return set_error(BI_ECUDA, "mul: %s", cudaGetErrorString(e));
    const uint64_t tiles = (n + MM_CTA / 32 - 1) / (MM_CTA / 32), cap = (uint64_t)num_sms() * occ;
    const bool vec = !w32 && m % 2 == 0 && ((uintptr_t)a | (uintptr_t)b | (uintptr_t)r) % 16 == 0;
    kern<<<(unsigned)(tiles < cap ? tiles : cap), MM_CTA, smem, st>>>(a, b, r, n, m, w32, vec);
    return check_launch("mul matrix kernel");
}

bi_status mul_mma(const void* a, const void* b, void* r, uint32_t m, uint64_t n, bool w32, bool full, cudaStream_t st) {
    const uint32_t L = w32 ? (m + 1) / 2 : m;
    switch (full ? 100 + (L + 15) / 16 : (L + 15) / 16) {
#define BI_MM(LT, FULL) case (FULL ? 100 : 0) + LT: return launch<LT, FULL>(a, b, r, m, n, w32, st);
    BI_MM(1, true) BI_MM(2, true) BI_MM(3, true) BI_MM(4, true) BI_MM(5, true) BI_MM(6, true) BI_MM(7, true) BI_MM(8, true)
    BI_MM(9, true) BI_MM(10, true)
    BI_MM(1, false) BI_MM(2, false) BI_MM(3, false) BI_MM(4, false) BI_MM(5, false) BI_MM(6, false) BI_MM(7, false) BI_MM(8, false) BI_MM(9, false)
    BI_MM(10, false) BI_MM(11, false) BI_MM(12, false) BI_MM(13, false) BI_MM(14, false) BI_MM(15, false)
    BI_MM(16, false)
#undef BI_MM
    default: return set_error(BI_EUNSUPPORTED, "mul matrix kernel: m=%u outside its sizes", m);
    }
}

}  // namespace bi
