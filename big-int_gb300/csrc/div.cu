// div.cu -- batched division (quotient and remainder) by a shifted inverse.
//
// The reference defines division only as a sequential C prototype
// (prototypes/div.c:427-467, div_shinv) and an unvalidated Futhark version
// (futhark/div.fut:150-167): q = floor(u * shinv_h(v) / B^h) + delta with the
// shifted inverse shinv_h(v) ~ B^h / v refined by Newton steps that use
// shorter iterates and prefixes of the divisor (refine3, div.c:333-349), then
// the remainder r = u - v*q and a final correction (div.c:457-463).  This
// kernel computes the same quantities on the GPU, one instance per CTA, all
// operands in shared memory, on 64-bit limbs:
//
//   1. normalise: shift u and v left by s bits so v's top limb has its top
//      bit set (K = limbs of v, H = limbs of the shifted u);
//   2. shifted inverse Y ~ B^(K+P) / v with P = H-K+2 limbs of precision:
//      start from floor((B^2-1)/v_top) (one correct limb) and apply Newton
//      steps y' = y + y(1 - x y) at growing precision p -> p' <= 2p-2, each
//      using only the top p'+1 limbs of v (divisor prefix) and a p+1-limb
//      iterate (shorter iterate); the error term 1 - x y is recovered from
//      the low p'+2 limbs of the product, as div.c's powerdiff recovers
//      B^h - v*w from a truncated product (div.c:246-280);
//   3. q = floor(u * Y / B^(K+P)); r = u - q*v from the low K+1 limbs of q*v;
//      while r < 0: q--, r += v; while r >= v: q++, r -= v (the reference's
//      delta step, div.c:459-463, made two-sided and bounded);
//   4. r is shifted back right by s bits.
// The estimate is exact or one short in every case tested; a bound of
// DIV_MAX_CORRECTIONS steps on each side turns anything else into status 2.
//
// Small and medium divisors take another route to the same unique (q, r):
// schoolbook long division (divsmall.cuh) on one thread per instance up to
// DIV_THREAD_MAX_MV 64-bit limbs and on one warp per instance up to
// DIV_WARP_MAX_MV, where its K (MU - K + 1) limb products and no barriers
// cost less than a CTA running the steps above (div_use_long holds the
// measured crossover, which depends on the batch size too).  Medium and large
// divisors go by blocks of quotient limbs to the tensor cores (divtc.cuh) where
// div_use_tc says so, and the two routes above keep the rest.
#include <type_traits>

#include "divblock.cuh"
#include "divtc.cuh"
#include "divcore.cuh"
#include "divsmall.cuh"

namespace bi {

template <typename T>
__device__ __forceinline__ uint64_t limb64(const T* p, uint32_t count_T, uint32_t i) {
    if constexpr (sizeof(T) == 8) {
        return i < count_T ? p[i] : 0;
    } else {
        uint64_t x = 2 * i < count_T ? p[2 * i] : 0u;
        if (2 * i + 1 < count_T) x |= (uint64_t)p[2 * i + 1] << 32;
        return x;
    }
}

template <typename T>
__device__ __forceinline__ void put_limb64(T* p, uint32_t count_T, uint32_t i, uint64_t x) {
    if constexpr (sizeof(T) == 8) {
        if (i < count_T) p[i] = x;
    } else {
        if (2 * i < count_T) p[2 * i] = (uint32_t)x;
        if (2 * i + 1 < count_T) p[2 * i + 1] = (uint32_t)(x >> 32);
    }
}

template <typename T>
__global__ void __launch_bounds__(512)
div_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
           uint8_t* __restrict__ status, uint64_t n, DivGeom g) {
    extern __shared__ __align__(16) uint64_t smem[];
    for (uint64_t inst = blockIdx.x; inst < n; inst += gridDim.x) {
        const T* ui = u + inst * g.mu;
        const T* vi = v + inst * g.mv;
        T* qi = q + inst * g.mu;
        T* ri = r + inst * g.mv;
        div_cta(
            g, smem, [&](uint32_t i) { return limb64(ui, g.mu, i); }, [&](uint32_t i) { return limb64(vi, g.mv, i); },
            [&](uint32_t i, uint64_t x) { put_limb64(qi, g.mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, g.mv, i, x); },
            [&](uint8_t code) { if (status) status[inst] = code; });
    }
}

// ---------------------------------------------------------------------------

// One thread per instance: long division for divisors of at most MX limbs
// (divsmall.cuh).
template <typename T, int MX>
__global__ void __launch_bounds__(DIV_THREAD_CTA)
div_thread_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                  uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2, MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    for (uint64_t inst = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; inst < n;
         inst += (uint64_t)gridDim.x * blockDim.x) {
        const T* ui = u + inst * mu;
        const T* vi = v + inst * mv;
        T* qi = q + inst * mu;
        T* ri = r + inst * mv;
        const uint8_t st = div_thread<MX>(
            MU, MV, [&](uint32_t i) { return limb64(ui, mu, i); }, [&](uint32_t i) { return limb64(vi, mv, i); },
            [&](uint32_t i, uint64_t x) { put_limb64(qi, mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, mv, i, x); });
        if (status) status[inst] = st;
    }
}

// The same with the warp's 32 instances in shared memory, a row of SU (SV)
// 64-bit slots an instance, both odd so that a limb of all lanes meets every
// bank once.  Rows come and go as consecutive words; the quotient and the
// remainder take the rows of u and v: quotient limb j is stored after the limbs
// of u from j up were read, the remainder after all of v was.  Bound by the
// latency of the carry chains; registers capped for 12 or 14 CTAs an SM (8 to 10
// as it is, at 8 divisor limbs) made it 4-12 % slower.
template <typename T>
__device__ __forceinline__ void rows_in(uint64_t* rows, uint32_t slots, const T* g, uint32_t m, uint32_t count) {
    constexpr uint32_t PER = 8 / sizeof(T);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(rows);
    const uint32_t dr = 32 / m, dc = 32 - dr * m;
    uint32_t row = (threadIdx.x & 31) / m, col = (threadIdx.x & 31) - row * m;
#pragma unroll 4
    for (uint32_t i = threadIdx.x & 31; i < count * m; i += 32) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                         base + (row * slots * PER + col) * (uint32_t)sizeof(T)),
                     "l"(g + i), "n"(sizeof(T))
                     : "memory");
        row += dr, col += dc;
        if (col >= m) col -= m, row++;
    }
}

template <typename T>
__device__ __forceinline__ void rows_out(const uint64_t* rows, uint32_t slots, T* g, uint32_t m, uint32_t count) {
    constexpr uint32_t PER = 8 / sizeof(T);
    const T* words = reinterpret_cast<const T*>(rows);
    const uint32_t dr = 32 / m, dc = 32 - dr * m;
    uint32_t row = (threadIdx.x & 31) / m, col = (threadIdx.x & 31) - row * m;
#pragma unroll 4
    for (uint32_t i = threadIdx.x & 31; i < count * m; i += 32) {
        g[i] = words[row * slots * PER + col];
        row += dr, col += dc;
        if (col >= m) col -= m, row++;
    }
}

template <typename T, int MX>
__global__ void __launch_bounds__(DIV_THREAD_CTA)
div_thread_rows_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                       uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    extern __shared__ __align__(16) uint64_t smem[];
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2, MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    const uint32_t SU = MU | 1, SV = MV | 1, lane = threadIdx.x & 31;
    uint64_t* ru = smem + threadIdx.x / 32 * 32 * (SU + SV);
    uint64_t* rv = ru + 32 * SU;
    uint64_t* mu_row = ru + lane * SU;
    uint64_t* mv_row = rv + lane * SV;
    for (uint64_t first = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32; first < n;
         first += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t count = n - first < 32 ? (uint32_t)(n - first) : 32u;
        rows_in(ru, SU, u + first * mu, mu, count);
        rows_in(rv, SV, v + first * mv, mv, count);
        if (sizeof(T) == 4 && (mu & 1)) reinterpret_cast<T*>(mu_row)[mu] = 0;   // an odd count's upper word
        if (sizeof(T) == 4 && (mv & 1)) reinterpret_cast<T*>(mv_row)[mv] = 0;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (lane < count) {
            const uint8_t st = div_thread<MX>(
                MU, MV, [&](uint32_t i) { return mu_row[i]; }, [&](uint32_t i) { return mv_row[i]; },
                [&](uint32_t i, uint64_t x) { mu_row[i] = x; }, [&](uint32_t i, uint64_t x) { mv_row[i] = x; });
            if (status) status[first + lane] = st;
        }
        __syncwarp();
        rows_out(ru, SU, q + first * mu, mu, count);
        rows_out(rv, SV, r + first * mv, mv, count);
        __syncwarp();
    }
}

// Several instances a warp: long division on G-lane groups (divsmall.cuh).
template <typename T, int VPL, int G>
__global__ void __launch_bounds__(DIV_WARP_CTA)
div_group_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                 uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv);

// Rows through shared memory, or each thread its own from global memory (us,
// direct / rows, 1.0e8 bytes of operands unless n is given).  Words of u32 are
// strided worst: 125 / 72 for 16 by 8 64-bit limbs, 85 / 67 for 8 by 4, but
// 58 / 69 for 6 by 3.  u64: 72 / 63 for 16 by 8, 92 / 78 for 32 by 16, 64 / 68
// for 15 by 7, 54 / 61 for 8 by 4.  Batches that do not fill the SMs have rows
// at less latency: 50000 of 16 by 8 26.8 / 21.3, of 4 by 2 20.7 / 16.0.  Longer
// rows leave too few warps an SM: u64 64 by 16 124 / 126 and 80 by 15 138 / 150,
// u32 80 by 15 178 / 162.  Moving rows costs some 0.4 us, which few quotient limbs
// do not earn back where the operands are in the L2 already (u64 5 by 4, 5000:
// 2.9 / 3.4, 11 by 4 4.7 / 4.9, 20 by 4 7.3 / 7.3; 40000 of 11 by 4 6.6 / 7.5; 9 by 8,
// 5000: 3.4 / 3.9, 20000: 4.6 / 4.6; u32 the same of 3-limb divisors, of 4-limb ones
// by 2 3.3 / 3.7, by 6 5.1 / 4.9); with cold operands the two are equal there.
constexpr int DIV_ROWS_PER_SM = 384;
template <typename T>
static bool div_thread_rows(uint32_t MU, uint32_t MV, uint64_t n, int sms) {
    const uint32_t ql = MU - MV + 1;
    const uint64_t per_sm = n / (uint64_t)sms;
    if (MV < (sizeof(T) == 8 ? 8u : 4u)) {
        if (ql < 8 || (ql < 24 && per_sm >= 160)) return false;
    } else if (sizeof(T) == 8 ? ql < 8 && per_sm < 64 : MV < 8 && ql < 5 && per_sm < 160) {
        return false;
    }
    if (sizeof(T) == 4 && MV >= 4) return MU + MV <= 94;
    if (n <= (uint64_t)DIV_ROWS_PER_SM * (uint64_t)sms) return MU + MV <= 72;
    return sizeof(T) == 8 && MV >= 8 && MU <= 48;
}

template <typename T>
static void launch_div_thread(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv,
                              uint64_t n, cudaStream_t s) {
    const uint32_t MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    if (div_small_on_groups(MV, n, num_sms())) {   // few instances: four 8-lane groups a warp
        const uint64_t warps = (n + 3) / 4, blocks = (warps + DIV_WARP_CTA / 32 - 1) / (DIV_WARP_CTA / 32);
        div_group_kernel<T, 2, 8><<<(unsigned)blocks, DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
        return;
    }
    const uint64_t blocks = (n + DIV_THREAD_CTA - 1) / DIV_THREAD_CTA;
    const unsigned grid = (unsigned)(blocks < (1u << 20) ? blocks : (1u << 20));
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2;
    const size_t rows = DIV_THREAD_CTA * ((MU | 1) + (MV | 1)) * sizeof(uint64_t);
    // register windows of 2, 3, 4, 6, 8, 12 or 16 limbs: a divisor is
    // right-aligned in its window, whose rows below it are zeros, so the widths
    // between the powers of two ran 6-20 % faster at 3, 5, 6, 10, 12 limbs
    auto launch = [&](auto width) {
        constexpr int MX = decltype(width)::value;
        if (div_thread_rows<T>(MU, MV, n, num_sms()))   // at most 48 KB of rows
            div_thread_rows_kernel<T, MX><<<grid, DIV_THREAD_CTA, rows, s>>>(u, v, q, r, status, n, mu, mv);
        else
            div_thread_kernel<T, MX><<<grid, DIV_THREAD_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    };
    if (MV <= 2) launch(std::integral_constant<int, 2>{});
    else if (MV <= 3) launch(std::integral_constant<int, 3>{});
    else if (MV <= 4) launch(std::integral_constant<int, 4>{});
    else if (MV <= 6) launch(std::integral_constant<int, 6>{});
    else if (MV <= 8) launch(std::integral_constant<int, 8>{});
    else if (MV <= 12) launch(std::integral_constant<int, 12>{});
    else launch(std::integral_constant<int, 16>{});
}

// One warp per instance: long division for divisors of at most 32 VPL limbs
// (divsmall.cuh).
template <typename T, int VPL>
__device__ __forceinline__ void div_warp_instances(const T* __restrict__ u, const T* __restrict__ v,
                                                   T* __restrict__ q, T* __restrict__ r,
                                                   uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2, MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    const uint64_t warps = (uint64_t)gridDim.x * (DIV_WARP_CTA / 32);
    for (uint64_t inst = (uint64_t)blockIdx.x * (DIV_WARP_CTA / 32) + threadIdx.x / 32; inst < n; inst += warps) {
        const T* ui = u + inst * mu;
        const T* vi = v + inst * mv;
        T* qi = q + inst * mu;
        T* ri = r + inst * mv;
        const uint8_t st = div_warp<VPL>(
            MU, MV, [&](uint32_t i) { return limb64(ui, mu, i); }, [&](uint32_t i) { return limb64(vi, mv, i); },
            [&](uint32_t i, uint64_t x) { put_limb64(qi, mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, mv, i, x); });
        if (status && (threadIdx.x & 31) == 0) status[inst] = st;
    }
}

template <typename T, int VPL>
__global__ void __launch_bounds__(DIV_WARP_CTA)
div_warp_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    div_warp_instances<T, VPL>(u, v, q, r, status, n, mu, mv);
}

// The same, held to three CTAs (12 warps) an SM: for 24 limbs a lane, where
// ptxas otherwise takes 255 registers (8 warps an SM), 168 registers and a
// few spills ran 4-10 % faster (700- and 768-limb divisors); the 20- and
// 28-limb shapes stay on the default bound (their 3-CTA variants were slower
// or spilled 240 bytes).
template <typename T, int VPL>
__global__ void __launch_bounds__(DIV_WARP_CTA, 3)
div_warp3_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                 uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    div_warp_instances<T, VPL>(u, v, q, r, status, n, mu, mv);
}

template <typename T, int VPL, int G>
__global__ void __launch_bounds__(DIV_WARP_CTA)
div_group_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
                 uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    constexpr uint32_t ipw = 32 / G;
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2, MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    const uint64_t warps = (uint64_t)gridDim.x * (DIV_WARP_CTA / 32);
    for (uint64_t w = (uint64_t)blockIdx.x * (DIV_WARP_CTA / 32) + threadIdx.x / 32; w * ipw < n; w += warps) {
        const uint64_t inst = w * ipw + (threadIdx.x & 31) / G;
        const bool valid = inst < n;
        const uint64_t k = valid ? inst : 0;   // an invalid group reads and writes nothing
        const T* ui = u + k * mu;
        const T* vi = v + k * mv;
        T* qi = q + k * mu;
        T* ri = r + k * mv;
        const uint8_t st = div_group<VPL, G>(
            valid, MU, MV, [&](uint32_t i) { return limb64(ui, mu, i); }, [&](uint32_t i) { return limb64(vi, mv, i); },
            [&](uint32_t i, uint64_t x) { put_limb64(qi, mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, mv, i, x); });
        if (status && valid && (threadIdx.x & (G - 1)) == 0) status[inst] = st;
    }
}

// Long division for divisors of 17..1024 64-bit limbs: the group shape per
// divisor size that ran fastest on GB300 (2m/m divisions, thousands of
// instances): 8-lane groups of 3, 4, 6 and 8 limbs a lane up to 24, 32, 48
// and 64 limbs, 16-lane groups of 6 and 8 up to 96 and 128, a whole warp of 6
// and 8 up to 192 and 256, 16-lane groups of 20, 24, 28 and 32 up to 320,
// 384, 448 and 512, a warp of 20, 24, 28 and 32 up to 640, 768, 896 and 1024
// (the shapes between the powers of two run 1.07-1.4x faster there: fewer
// rows of zeros below the right-aligned divisor, fewer registers); with few instances
// (div_small_on_warps) one warp each up to 128 limbs.
template <typename T>
static void launch_div_warp(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv,
                            uint64_t n, cudaStream_t s) {
    const uint32_t MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    constexpr uint32_t WPC = DIV_WARP_CTA / 32;   // warps per CTA
    auto grid_for = [&](uint32_t ipw) {
        const uint64_t warps = (n + ipw - 1) / ipw;
        const uint64_t blocks = (warps + WPC - 1) / WPC;
        return (unsigned)(blocks < (1u << 20) ? blocks : (1u << 20));
    };
    if (div_small_on_warps(MV, n, num_sms())) {   // few instances: one warp each
        if (MV <= 32) div_warp_kernel<T, 1><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
        else if (MV <= 64) div_warp_kernel<T, 2><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
        else div_warp_kernel<T, 4><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
        return;
    }
    if (MV <= 24) div_group_kernel<T, 3, 8><<<grid_for(4), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 32) div_group_kernel<T, 4, 8><<<grid_for(4), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 48) div_group_kernel<T, 6, 8><<<grid_for(4), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 64) div_group_kernel<T, 8, 8><<<grid_for(4), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 96) div_group_kernel<T, 6, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 128) div_group_kernel<T, 8, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 192) div_warp_kernel<T, 6><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 256) div_warp_kernel<T, 8><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    // 20, 24 and 28 limbs a lane between the powers of two: a divisor is
    // right-aligned in the lanes' 32 VPL (or G VPL) limbs, whose rows below it
    // are zeros
    else if (MV <= 320) div_group_kernel<T, 20, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 384) div_group_kernel<T, 24, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 448) div_group_kernel<T, 28, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 512) div_group_kernel<T, 32, 16><<<grid_for(2), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 640) div_warp_kernel<T, 20><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 768) div_warp3_kernel<T, 24><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else if (MV <= 896) div_warp_kernel<T, 28><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
    else div_warp_kernel<T, 32><<<grid_for(1), DIV_WARP_CTA, 0, s>>>(u, v, q, r, status, n, mu, mv);
}

// One instance on NW warps: long division KB quotient limbs at a time
// (divblock.cuh) for divisors of at most 32 NW VPL limbs.  NW = 1: four
// warps a CTA, one instance each; NW > 1: one instance a CTA of NW warps.
template <typename T, int VPL, int KB, int NW>
__global__ void __launch_bounds__(NW == 1 ? DIV_WARP_CTA : 32 * NW)
div_blk_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
               uint8_t* __restrict__ status, uint64_t n, uint32_t mu, uint32_t mv) {
    __shared__ DivBlkShared<KB, NW> sh;
    const uint32_t MU = sizeof(T) == 8 ? mu : (mu + 1) / 2, MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    const uint64_t per_cta = NW == 1 ? DIV_WARP_CTA / 32 : 1;
    const uint64_t stride = (uint64_t)gridDim.x * per_cta;
    for (uint64_t inst = (uint64_t)blockIdx.x * per_cta + (NW == 1 ? threadIdx.x / 32 : 0); inst < n;
         inst += stride) {
        const T* ui = u + inst * mu;
        const T* vi = v + inst * mv;
        T* qi = q + inst * mu;
        T* ri = r + inst * mv;
        const uint8_t st = div_blk<VPL, KB, NW>(
            MU, MV, [&](uint32_t i) { return limb64(ui, mu, i); }, [&](uint32_t i) { return limb64(vi, mv, i); },
            [&](uint32_t i, uint64_t x) { put_limb64(qi, mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, mv, i, x); }, &sh);
        if (status && threadIdx.x % (32 * NW) == 0) status[inst] = st;
    }
}

template <typename T, int VPL, int KB, int NW>
static void launch_blk(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv, uint64_t n,
                       cudaStream_t s) {
    const uint64_t per_cta = NW == 1 ? DIV_WARP_CTA / 32 : 1;
    const uint64_t blocks = (n + per_cta - 1) / per_cta;
    const unsigned grid = (unsigned)(blocks < (1u << 20) ? blocks : (1u << 20));
    div_blk_kernel<T, VPL, KB, NW><<<grid, NW == 1 ? DIV_WARP_CTA : 32 * NW, 0, s>>>(u, v, q, r, status, n, mu, mv);
}

// Long division of divisors of 1025..DIV_LONG_MAX_MV limbs, KB = 8 quotient
// limbs at a time (divblock.cuh) on two or four warps.
template <typename T>
static void launch_div_blk(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv,
                           uint64_t n, cudaStream_t s) {
    const uint32_t MV = sizeof(T) == 8 ? mv : (mv + 1) / 2;
    if (MV <= 2048) launch_blk<T, 32, 8, 2>(u, v, q, r, status, mu, mv, n, s);
    else launch_blk<T, 32, 8, 4>(u, v, q, r, status, mu, mv, n, s);
}

// ---------------------------------------------------------------------------
// Long division 31 or 63 quotient limbs at a time on the tensor cores
// (divtc.cuh), one instance a CTA at a time, the CTAs persistent.  2048
// divisions of 2048 by 1024 limbs 3400 -> 565 us, 8192 of 512 by 256 1013 ->
// 409.  Bound by the latency of a block's chain -- estimate, product, fold,
// carries, each behind a barrier: issue slots 45 % busy at four CTAs an SM (what
// tensor memory holds at 1024 limbs), the tensor core 30 %.
// ---------------------------------------------------------------------------
// (P = 16 held to 12 CTAs an SM, 40 registers: 192-limb divisors 376 -> 347 us at
// 10922, 128-limb ones 418 -> 403; wider shapes ran slower so.  0 leaves the bound to
// the compiler, 64 to 96 registers; a 1 lets it take 250: 1024 limbs 565 -> 930 us.
// P = 64 at 7, 72 registers: at the compiler's 64 it spills, 2849 divisions of 1472
// by 736 limbs 521 -> 500 us, 2116 of 1982 by 991 551 -> 523; shared memory holds
// four or five CTAs there)
template <typename T, int P, int G, uint32_t HELD = 0>
__global__ void __launch_bounds__(DtShape<P, G>::NT, P == 16 ? 12 : P == 64 ? 7 : 0)
div_tc_kernel(const T* __restrict__ u, const T* __restrict__ v, T* __restrict__ q, T* __restrict__ r,
              uint8_t* __restrict__ status, uint64_t n, DtGeom g, uint32_t* gave_up) {
    extern __shared__ __align__(128) uint8_t smem_dt[];
    const DtSmem<P, G> lay(g);
    const uint32_t tmem = dt_begin<P, G, HELD>(lay, smem_dt);
    uint32_t phase = 0;
    for (uint64_t inst = blockIdx.x; inst < n; inst += gridDim.x) {
        const T* ui = u + inst * g.mu;
        const T* vi = v + inst * g.mv;
        T* qi = q + inst * g.mu;
        T* ri = r + inst * g.mv;
        const uint8_t st = dt_divide<P, G>(
            g, lay, smem_dt, tmem, phase, [&](uint32_t i) { return limb64(ui, g.mu, i); },
            [&](uint32_t i) { return limb64(vi, g.mv, i); }, [&](uint32_t i, uint64_t x) { put_limb64(qi, g.mu, i, x); },
            [&](uint32_t i, uint64_t x) { put_limb64(ri, g.mv, i, x); });
        if (status && threadIdx.x == 0) status[inst] = st;
    }
    dt_end<P, G>(lay, smem_dt, tmem, gave_up);
}

template <typename T, int P, int G>
static bi_status launch_div_tc(const T* u, const T* v, T* q, T* r, uint8_t* status, uint64_t n, const DtGeom& g,
                               cudaStream_t s) {
    const size_t smem = DtSmem<P, G>(g).total;
    auto kern = div_tc_kernel<T, P, G>;
    cudaError_t e = smem_opt_in((const void*)kern, smem);
    if (e != cudaSuccess) return set_error(BI_ECUDA, "div: %s", cudaGetErrorString(e));
    uint32_t* gave_up;
    BI_RETURN_IF(gave_up_word(&gave_up));
    const uint64_t cap = (uint64_t)num_sms() * tc_ctas_per_sm((const void*)kern, DtShape<P, G>::NT, smem, DtShape<P, G>::TMEM_COLS);
    kern<<<(unsigned)(n < cap ? n : cap), DtShape<P, G>::NT, smem, s>>>(u, v, q, r, status, n, g, gave_up);
    return check_launch("div tensor kernel");
}

bi_status div_held(const uint64_t* u, const uint64_t* v, uint64_t* q, uint64_t* r, uint8_t* status, uint32_t mu,
                   uint32_t mv, uint64_t n, uint32_t* gave_up, cudaStream_t s) {
    const DtGeom g = dt_geom(mu, mv, 8);
    const size_t smem = DtSmem<16, 1>(g).total;
    auto kern = div_tc_kernel<uint64_t, 16, 1, 1>;
    cudaError_t e = smem_opt_in((const void*)kern, smem);
    if (e != cudaSuccess) return set_error(BI_ECUDA, "held wait: %s", cudaGetErrorString(e));
    kern<<<2, DtShape<16, 1>::NT, smem, s>>>(u, v, q, r, status, n, g, gave_up);
    return check_launch("held div kernel");
}

// the narrowest accumulator whose rows hold the divisor
template <typename T>
static bi_status div_tc(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv, uint64_t n,
                        cudaStream_t s) {
    const DtGeom g = dt_geom(mu, mv, (int)sizeof(T));
    if (g.MV <= (uint32_t)DtShape<16, 1>::MAX_K) return launch_div_tc<T, 16, 1>(u, v, q, r, status, n, g, s);
    if (g.MV <= (uint32_t)DtShape<32, 1>::MAX_K) return launch_div_tc<T, 32, 1>(u, v, q, r, status, n, g, s);
    if (g.MV <= (uint32_t)DtShape<48, 1>::MAX_K) return launch_div_tc<T, 48, 1>(u, v, q, r, status, n, g, s);
    if (g.MV <= (uint32_t)DtShape<64, 1>::MAX_K) return launch_div_tc<T, 64, 1>(u, v, q, r, status, n, g, s);
    // blocks of 63 limbs: 2048 divisions of 2048 by 1024 limbs 627 -> 565 us, one
    // 87 -> 72; of 3072 by 1536 one 159 -> 119 us, 1365 of them 1013 -> 1052;
    // below 992 limbs slower (512: 435 -> 477 at 4096 of them)
    if (g.MV <= (uint32_t)DtShape<80, 2>::MAX_K) return launch_div_tc<T, 80, 2>(u, v, q, r, status, n, g, s);
    if (n <= (uint64_t)num_sms() && g.MV <= (uint32_t)DtShape<128, 2>::MAX_K)
        return launch_div_tc<T, 128, 2>(u, v, q, r, status, n, g, s);
    return launch_div_tc<T, 128, 1>(u, v, q, r, status, n, g, s);
}

// Measured against the lane groups, the warps and the shifted inverse (us, u64,
// before / on the tensor cores): an instance costs about 8K cycles before its
// first quotient block (the reciprocal, the divisor's digits), which a batch
// that fills the GPU earns back above a product of divisor and quotient limbs of
// some 6000 to 9400 (16384 divisions with 128-limb divisors: 31 quotient limbs
// 146 / 183, 62 limbs 275 / 246; 4096 with 512: 8 limbs 64 / 80, 16 limbs 93 /
// 79; 2m by m limbs: m = 80 472 / 485, 100 574 / 472, 256 1013 / 409, 1024
// 3399 / 626, 2000 6468 / 982).  With few instances the blocks' shorter chain
// wins from about 20 quotient limbs on: 1 division of 2m by m limbs with m = 40
// 20 / 13, 64 30 / 15, 256 83 / 26, 1024 360 / 89; 608 of them with m = 40 22 /
// 18; 2432 with m = 72 61 / 54, with m = 64 50 / 54.  At two to four an SM it takes
// a few more: 64 limbs by 20 quotient limbs, 304 divisions 10.2 / 10.3, 400 10.2 /
// 11.3, 608 10.2 / 12.7 (by 24 11.7 / 12.5, by 40 17.6 / 15.4); 128 limbs by 20, 608
// 12.2 / 12.8.  Four of more than 1024 limbs and few quotient limbs an SM are the
// one full wave of CTAs that 8 quotient limbs at a time beat (1215 by 8: 608
// divisions 28.7 / 35.8, 456 26.1 / 23.6, 760 57.0 / 39.4).
static bool div_use_tc(uint32_t MU, uint32_t MV, uint64_t n) {
    const uint64_t ql = MU - MV + 1, sms = (uint64_t)num_sms();
    if (MV < 40 || MV > (uint32_t)DtShape<128, 1>::MAX_K) return false;
    if (MV > 1024 && ql < 10 && n > 3 * sms && n <= 4 * sms) return false;
    if (MV >= 65 && MV * ql >= 9400 && !div_short_quotient(MV, ql, n, (int)sms)) return true;
    const bool few = n <= 2 * sms   ? ql >= 20
                     : n <= 3 * sms ? ql >= (MV < 65 ? 24u : 20u)
                                    : n <= 4 * sms && ql >= (MV < 65 ? 36u : 22u);
    return few || (MV >= 65 && ql >= 48 && n <= 16 * sms);
}

// dividend limbs (u64 view) per instance: any long division, and the shifted inverse's limit
constexpr uint32_t DIV_MAX_MU64 = 8192, DIV_SHINV_MAX_MU64 = 2048;
constexpr int DIV_AUTO = 0, DIV_SHINV = 1, DIV_LONG = 2;   // method of div_entry

template <typename T>
static bi_status div_entry(const T* u, const T* v, T* q, T* r, uint8_t* status, uint32_t mu, uint32_t mv,
                           uint64_t n, bi_stream s, int method = DIV_AUTO) {
    if (n == 0) return BI_OK;
    if (mu == 0 || mv == 0) return set_error(BI_EINVAL, "mu and mv must be >= 1");
    if (mv > mu) return set_error(BI_EINVAL, "divisor limbs mv=%u exceed dividend limbs mu=%u", mv, mu);
    if (!u || !v || !q || !r) return set_error(BI_EINVAL, "NULL buffer");
    if ((uintptr_t)u % sizeof(T) || (uintptr_t)v % sizeof(T) || (uintptr_t)q % sizeof(T) ||
        (uintptr_t)r % sizeof(T))
        return set_error(BI_EINVAL, "buffers must be aligned to the limb size");
    const DivGeom g = div_geom(mu, mv, (int)sizeof(T));
    if (g.MU > DIV_MAX_MU64) return set_error(BI_EUNSUPPORTED, "div: dividend of %u limbs above the supported size", mu);
    if (method == DIV_LONG && g.MV > (uint32_t)DIV_LONG_MAX_MV)
        return set_error(BI_EUNSUPPORTED, "div_long: divisor of %u limbs above %d 64-bit limbs", mv, DIV_LONG_MAX_MV);
    if (method == DIV_SHINV && g.MU > DIV_SHINV_MAX_MU64)
        return set_error(BI_EUNSUPPORTED, "div_shinv: dividend of %u limbs above %u 64-bit limbs", mu,
                         DIV_SHINV_MAX_MU64);
    BI_RETURN_IF(waits_ok());
    if (method != DIV_SHINV && g.MV <= (uint32_t)DIV_THREAD_MAX_MV) {
        launch_div_thread(u, v, q, r, status, mu, mv, n, (cudaStream_t)s);
        return check_launch("div thread kernel");
    }
    if (method == DIV_AUTO && div_use_tc(g.MU, g.MV, n)) return div_tc(u, v, q, r, status, mu, mv, n, (cudaStream_t)s);
    // the shifted inverse holds its operands in shared memory: dividends above
    // DIV_SHINV_MAX_MU64 limbs always take long division
    if (method != DIV_SHINV && g.MV <= (uint32_t)DIV_LONG_MAX_MV &&
        (method == DIV_LONG || g.MU > DIV_SHINV_MAX_MU64 || div_use_long(g.MV, n, num_sms()))) {
        if (g.MV <= (uint32_t)DIV_WARP_MAX_MV) {
            launch_div_warp(u, v, q, r, status, mu, mv, n, (cudaStream_t)s);
            return check_launch("div warp kernel");
        }
        launch_div_blk(u, v, q, r, status, mu, mv, n, (cudaStream_t)s);
        return check_launch("div block kernel");
    }
    const size_t smem = div_smem_bytes(g);
    if (smem > 227 * 1024) return set_error(BI_EUNSUPPORTED, "div: sizes need too much shared memory");
    const int threads = div_threads(g.MU);
    auto kern = div_kernel<T>;
    cudaError_t e = smem_opt_in((const void*)kern, smem);
    if (e != cudaSuccess) return set_error(BI_ECUDA, "div: %s", cudaGetErrorString(e));
    const uint64_t grid = n < (1ull << 30) ? n : (1ull << 30);
    kern<<<(unsigned)grid, threads, smem, (cudaStream_t)s>>>(u, v, q, r, status, n, g);
    return check_launch("div kernel");
}

}  // namespace bi

using namespace bi;

extern "C" {

uint32_t bi_max_limbs_div_u64(void) { return DIV_MAX_MU64; }
uint32_t bi_max_limbs_div_u32(void) { return 2 * DIV_MAX_MU64; }

bi_status bi_div_u64(const uint64_t* u, const uint64_t* v, uint64_t* q, uint64_t* r, uint8_t* status,
                     uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint64_t>(u, v, q, r, status, mu, mv, n, s);
}
bi_status bi_div_u32(const uint32_t* u, const uint32_t* v, uint32_t* q, uint32_t* r, uint8_t* status,
                     uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint32_t>(u, v, q, r, status, mu, mv, n, s);
}

bi_status bi_div_shinv_u64(const uint64_t* u, const uint64_t* v, uint64_t* q, uint64_t* r, uint8_t* status,
                           uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint64_t>(u, v, q, r, status, mu, mv, n, s, DIV_SHINV);
}
bi_status bi_div_shinv_u32(const uint32_t* u, const uint32_t* v, uint32_t* q, uint32_t* r, uint8_t* status,
                           uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint32_t>(u, v, q, r, status, mu, mv, n, s, DIV_SHINV);
}
bi_status bi_div_long_u64(const uint64_t* u, const uint64_t* v, uint64_t* q, uint64_t* r, uint8_t* status,
                          uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint64_t>(u, v, q, r, status, mu, mv, n, s, DIV_LONG);
}
bi_status bi_div_long_u32(const uint32_t* u, const uint32_t* v, uint32_t* q, uint32_t* r, uint8_t* status,
                          uint32_t mu, uint32_t mv, uint64_t n, bi_stream s) {
    return div_entry<uint32_t>(u, v, q, r, status, mu, mv, n, s, DIV_LONG);
}

}  // extern "C"
