// multc.cuh -- products of large operands on the 5th-generation tensor cores.
//
// The schoolbook product is a convolution of digits, C_c = sum a_x b_(c-x),
// and a convolution is a matrix product of two Toeplitz matrices: with
// columns c = P i + j (row i, 0 <= j < P) and x = P i + t,
//     C[i][j] = sum_t A[i][t] B[j][t],   A[i][t] = a[P i + t],  B[j][t] = b[j - t].
// Digits are bytes, held exactly as f16; products are below 2^16, and 128 of
// them sum to at most 128 * 255^2 < 2^23, so the tensor core's f32 sums are
// exact integers whatever their order.  A block of at most 128 terms of t
// ends in tensor memory; the threads add it to 32-bit integer sums while the
// next block runs (8192 terms of an operand sum below 2^30, the largest
// operand's 32768 below 2^31).
//
// Neither Toeplitz matrix is written out.  In the K-major layout without
// swizzle a core matrix is 8 rows of 16 bytes, contiguous:
//   A  chunk q (8 digits = one limb) of row rho lies at q * R * 16 + rho * 16,
//      rows rho of P digits: the tile of rows P i + t for t = P k + 16 s starts
//      k rows and 2 s chunks further -- one copy of a, 2 bytes a digit, serves
//      every t (a[P i + t] for t >= P is row i + 1);
//   B  core matrix (rows j = 8 j1 + j0, chunk q) depends on q - j1 alone: the
//      rows are taken in descending j1, so that core matrix x = n1 + q holds
//      the 8 x 8 Toeplitz block of two neighbouring limbs of b.  A block of t
//      needs P/8 + 15 of them (4 KB at P = 128), made from b's limbs in
//      shared memory while the tensor core works on the block before.
// A row of the accumulator is P consecutive digit columns, P/8 limbs of the
// product: its one or two threads fold them with one carry, and a carry
// lookahead over the threads joins them.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace bi {

constexpr uint32_t tc_pow2(uint32_t x) { return x <= 32 ? 32 : x <= 64 ? 64 : x <= 128 ? 128 : x <= 256 ? 256 : 512; }

template <int P>
struct TcShape {
    static constexpr int Q = P / 8;                 // limbs a row
    static constexpr int H = P >= 32 ? 2 : 1;       // draining threads a row (each has P / H accumulator columns)
    static constexpr uint32_t DRAIN = 128 * H;      // draining threads
    static constexpr int CT = P / H, QT = Q / H;    // accumulator columns and limbs a thread
    static constexpr int RB = 128 / P;              // rows of t a block
    static constexpr int KB = RB * P;               // terms of t a block, at most 128 (the f32 bound)
    static constexpr int STEPS = KB / 16;           // matrix instructions a block (K = 16 each)
    static constexpr int CM = Q + KB / 8 - 1;       // core matrices of B a block
    static constexpr int PAD = 16;                  // zero limbs below b (and 2 Q + 1 above) that blocks at its ends read
    static constexpr int NS = P > 64 ? 4 : 8;       // blocks under way: stages of B, accumulators
    static constexpr uint32_t TMEM_COLS = tc_pow2(NS * P);
    // warps: DRAIN / 32 draining, 4 making B, 2 issuing, 2 loading operands
    static constexpr uint32_t THREADS = DRAIN + 256;
};

// The layout of a kernel's operand buffers, for every instance it is given.
struct TcGeom {
    uint32_t L;            // limbs of the largest operand, in the u64 view
    uint32_t R;            // rows of the A buffer (R % 8 == 1: consecutive limbs fall into different banks)
    int32_t rho0;          // a's row at the buffer's first row (<= 0: zero rows before a)
    uint32_t NA;           // operand buffers (2: the next instance is loaded under this one's product)
};

// first and last row offset k of tile tau (t = P k ..): rows 128 tau + i + k
// that meet a's D rows, terms that meet b
__host__ __device__ inline void tc_krange(uint32_t D, uint32_t tau, int& lo, int& hi) {
    const int a = -(int)(128 * tau + 127), b = (int)D - 1 - (int)(128 * tau);
    lo = a > -(int)D ? a : -(int)D;
    hi = b < 0 ? b : 0;
}

// rows of P digits that hold L limbs, accumulator tiles of 128 rows that hold out_limbs
template <int P>
__host__ __device__ inline uint32_t tc_rows(uint32_t L) { return (L + P / 8 - 1) / (P / 8); }
template <int P>
__host__ __device__ inline uint32_t tc_tiles(uint32_t out_limbs) { return (out_limbs + 16 * P - 1) / (16 * P); }

// Widens g (zero at first) for products of L limbs to out_limbs.
template <int P>
inline void tc_geometry_add(TcGeom& g, uint32_t L, uint32_t out_limbs) {
    using S = TcShape<P>;
    int first = g.rho0, last = g.L ? g.rho0 + (int)g.R - 1 : first;
    const uint32_t D = tc_rows<P>(L);
    for (uint32_t tau = 0; tau < tc_tiles<P>(out_limbs); tau++) {
        int lo, hi;
        tc_krange(D, tau, lo, hi);
        const int nblk = (hi - lo + S::RB) / S::RB;
        const int f = (int)(128 * tau) + lo, l = (int)(128 * tau) + 127 + lo + nblk * S::RB - 1;
        first = f < first ? f : first;
        last = l > last ? l : last;
    }
    if (L > g.L) g.L = L;
    g.rho0 = first;
    g.R = (uint32_t)(last - first + 1);
    g.R += (9 - g.R % 8) % 8;
}

// Shared memory in bytes: NA times A, NA times b's limbs, the stages of B, the
// draining threads' limbs of the result, their overflows, lookahead scratch,
// the barriers and the tensor memory address.
template <int P>
struct TcSmem {
    uint32_t abytes, bbytes, braw, stage, rows, ovf, scratch, bars, total;
    __host__ __device__ explicit TcSmem(const TcGeom& g) {
        using S = TcShape<P>;
        abytes = (g.R * S::Q * 16 + 127) / 128 * 128;
        bbytes = (S::PAD + g.L + 2 * S::Q + 1 + 1) / 2 * 16;
        braw = g.NA * abytes;
        stage = (braw + g.NA * bbytes + 127) / 128 * 128;
        rows = stage + S::NS * S::CM * 128;
        ovf = rows + S::DRAIN * (S::QT + 1) * 8;
        scratch = ovf + (S::DRAIN + 2) * 8;
        bars = scratch + 16 * 4;
        total = bars + 30 * 8;
    }
};

// ---------------------------------------------------------------------------
// tensor core instructions
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tc_smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tc_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// the warp's arrival, after what its lanes did before
__device__ __forceinline__ void tc_warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(bar) : "memory");
}

// Waits for the barrier's phase; false after a second (the caller then gives the
// results up, reports it and leaves with nothing of its own in flight).
__device__ __forceinline__ bool tc_bar_wait(uint32_t bar, uint32_t parity) {
    uint64_t t0 = 0;
    for (uint32_t tries = 0;; tries++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((tries & 255u) == 255u) {
            uint64_t now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            if (now - t0 > 1000000000ull) return false;
        }
    }
}

// The same for a warp: every lane waits, every lane has the same answer.
__device__ __forceinline__ bool tc_warp_wait(uint32_t bar, uint32_t parity) {
    return __all_sync(0xffffffffu, tc_bar_wait(bar, parity));
}

// A matrix in shared memory, K-major without swizzle, as the low word of its
// descriptor: core matrices along the rows are 128 bytes apart (the high
// word's part), along K `lead` 16-byte units; `at` is the address in 16-byte
// units, so that steps along the matrix add to it.
__device__ __forceinline__ uint32_t tc_desc(uint32_t at, uint32_t lead) { return at | lead << 16; }

template <int P>
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint32_t b, bool accumulate) {
    // f16 x f16 -> f32, M = 128, N = P, both K-major
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(P / 8) << 17) | ((128u / 16) << 24);
    constexpr uint32_t high = 8u | 1u << 14;      // 128 bytes; descriptor version 1
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(d),
        "r"(a), "r"(b), "r"(idesc), "r"((uint32_t)accumulate), "r"(high)
        : "memory");
}

// One lane of a converged warp.  The instructions above take their operands
// from the warp's uniform registers: under a branch on the thread index each
// of them costs about 70 cycles to issue (200 with the address arithmetic of
// tc_product), under a warp-uniform branch and this election they run at the
// tensor core's own 65 cycles (M = 128, N = 128; 40 at N = 16).
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 8, 16 or 32 accumulator columns of the warp's 32 rows; the wait is in the
// same statement, so that no use of v can be scheduled before it
__device__ __forceinline__ void tc_ld(uint32_t addr, float (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tc_ld(uint32_t addr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tc_ld(uint32_t addr, float (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]),
          "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]),
          "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]),
          "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(addr)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// two bytes of w, picked by `sel` with 0x64 above each, as a pair of f16:
// 0x64bb is 1024 + bb
__device__ __forceinline__ uint32_t tc_digits(uint32_t w, uint32_t sel) {
    const uint32_t x = __byte_perm(w, 0x64646464u, sel);
    const __half2 y = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400)));
    return *reinterpret_cast<const uint32_t*>(&y);
}

// COLS columns of tensor memory for the CTA, its address through the word at
// shared address `at`; init() runs on one thread and its barriers are set up
// for every thread and the tensor core when this returns.
template <uint32_t COLS, typename Init>
__device__ __forceinline__ uint32_t tc_alloc(uint32_t at, Init init) {
    if (threadIdx.x == 0) {
        init();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(at) : "memory");
    return __shfl_sync(0xffffffffu, tmem, 0);
}

// Every thread, after the last use; the matrix instructions have ended.
template <uint32_t COLS>
__device__ __forceinline__ void tc_free(uint32_t tmem) {
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
}

// ---------------------------------------------------------------------------
// The kernel's body: products of the CTA's instances first, first + step, ..
// below n, its warps specialised and joined by barriers, so that the tensor
// core always has a block queued:
//   loading   the next instance's operands: a as f16 digits, b's limbs;
//   making    B's core matrices;
//   issuing   the matrix instructions, into NS accumulators in turn;
//   draining  each finished accumulator into 32-bit sums, then the product's
//             limbs, while the tensor core is on the next blocks or instance.
// HELD > 0 (a test) makes the barriers of B's stages wait for an arrival that
// never comes.
// fetch(i) gives instance i: L (at most g.L) and out_limbs, a(x) and b(x) the
// limbs of its operands (x < L), store(x, v) takes limb x < out_limbs of its
// product mod B^out_limbs.  Each role fetches an instance while it works on
// the one before.  Every wait gives up after a second; a warp whose wait ran out
// fills, issues and stores nothing more, the CTA leaves and reports to `gave_up`.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tc_carry_in(uint32_t g, uint32_t p, uint32_t nwarps, uint32_t* scratch) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t A = __ballot_sync(0xffffffffu, g | p), B = __ballot_sync(0xffffffffu, g);
    if (lane == 0) {
        const uint32_t g0 = warp_carry_resolve(A, B, 0).cout, g1 = warp_carry_resolve(A, B, 1).cout;
        scratch[warp] = g0 | (g1 & ~g0) << 1;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32) : "memory");
    const uint32_t s = lane < warp ? scratch[lane] : 0u;
    const uint32_t A2 = __ballot_sync(0xffffffffu, s != 0), B2 = __ballot_sync(0xffffffffu, s & 1);
    const uint32_t cin = (warp_carry_resolve(A2, B2, 0).carries >> warp) & 1u;
    return (warp_carry_resolve(A, B, cin).carries >> lane) & 1u;
}

template <int P, uint32_t HELD = 0, typename Fetch>
__device__ __forceinline__ void tc_products(const TcGeom& g, uint8_t* smem, uint64_t first, uint64_t step, uint64_t n,
                                            uint32_t* gave_up, Fetch fetch) {
    using S = TcShape<P>;
    constexpr int Q = S::Q, QT = S::QT, CT = S::CT;
    constexpr uint32_t ND = S::DRAIN, NS = S::NS;
    const TcSmem<P> lay(g);
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t sbase = tc_smem_addr(smem), bars = sbase + lay.bars;
    // Block c uses stage and accumulator c % NS: `made` when B's stage is
    // written, `run` when the matrix instructions are done (the stage may be
    // written again), `read` when the accumulator has been read.
    const uint32_t made = bars, run = made + 8 * NS, read = run + 8 * NS;
    const uint32_t a_full = read + 8 * NS, a_empty = a_full + 16, done = a_empty + 16;
    static_assert(3 * NS + 4 + 2 <= 30, "barriers");

    // rows around a and limbs around b are zero, and stay so
    for (uint32_t idx = tid; idx < g.NA * ((lay.abytes + lay.bbytes) / 16); idx += S::THREADS)
        *reinterpret_cast<uint4*>(smem + idx * 16) = make_uint4(0, 0, 0, 0);
    tc_fence_smem();
    const uint32_t tmem = tc_alloc<S::TMEM_COLS>(done + 8, [&] {
        for (uint32_t k = 0; k < NS; k++) {
            tc_bar_init(made + 8 * k, 1 + HELD);
            tc_bar_init(run + 8 * k, 1);
            tc_bar_init(read + 8 * k, ND / 32);
        }
        for (uint32_t k = 0; k < 2; k++) {
            tc_bar_init(a_full + 8 * k, 2);
            tc_bar_init(a_empty + 8 * k, 6);
        }
        tc_bar_init(done, 2);
    });

    bool ok = true;
    uint32_t c = 0, p = 0;      // blocks and instances so far
    if (warp >= ND / 32 + 6) {
        // ---- loading
        const uint32_t t = tid - (ND + 192);
        uint32_t before[2] = {0, 0};       // limbs each buffer holds
        auto cur = fetch(first);
        for (uint64_t i = first; i < n && ok; i += step, p++) {
            const auto next = fetch(i + step < n ? i + step : i);
            const uint32_t buf = p % g.NA;
            ok = tc_warp_wait(a_empty + 8 * buf, ((p / g.NA) & 1) ^ 1);
            if (!ok) break;
            uint8_t* as = smem + buf * lay.abytes - g.rho0 * 16;
            uint64_t* bs = reinterpret_cast<uint64_t*>(smem + lay.braw + buf * lay.bbytes) + S::PAD;
#pragma unroll 4
            for (uint32_t x = t; x < cur.L; x += 64) {
                const uint64_t v = cur.a(x);
                bs[x] = cur.b(x);
                const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
                *reinterpret_cast<uint4*>(as + (x % Q * g.R + x / Q) * 16) =
                    make_uint4(tc_digits(lo, 0x4140), tc_digits(lo, 0x4342), tc_digits(hi, 0x4140), tc_digits(hi, 0x4342));
            }
            for (uint32_t x = cur.L + t; x < (buf == 0 ? before[0] : before[1]); x += 64) {   // what the last instance had above
                bs[x] = 0;
                *reinterpret_cast<uint4*>(as + (x % Q * g.R + x / Q) * 16) = make_uint4(0, 0, 0, 0);
            }
            if (buf == 0) before[0] = cur.L;
            else before[1] = cur.L;
            tc_fence_smem();
            tc_warp_arrive(a_full + 8 * buf);
            cur = next;
        }
    } else if (warp >= ND / 32) {
        if (warp < ND / 32 + 4) {
            // ---- making B: each warp its own stages, so that several are under way
            static_assert(NS % 4 == 0, "each stage has one warp");
            const uint32_t t = tid & 31, own = warp - ND / 32, j1 = (t & 7) + 1;
            const uint32_t sel = 0x3210u + 0x1111u * (j1 & 3);
            auto cur = fetch(first);
            for (uint64_t i = first; i < n && ok; i += step, p++) {
                const auto next = fetch(i + step < n ? i + step : i);
                const uint32_t buf = p % g.NA, D = tc_rows<P>(cur.L), tiles = tc_tiles<P>(cur.out_limbs);
                ok = tc_warp_wait(a_full + 8 * buf, (p / g.NA) & 1);
                const uint32_t* bs = reinterpret_cast<const uint32_t*>(smem + lay.braw + buf * lay.bbytes) + 2 * S::PAD + (j1 >> 2);
                for (uint32_t tau = 0; tau < tiles && ok; tau++) {
                    int klo, khi;
                    tc_krange(D, tau, klo, khi);
                    for (int k0 = klo; k0 <= khi && ok; k0 += S::RB, c++) {
                        if (c % 4 != own) continue;
                        ok = tc_warp_wait(run + 8 * (c % NS), ((c / NS) & 1) ^ 1);
                        if (!ok) break;
                        // core matrix x, row j0: bytes j0 - 7 .. j0 of limb w = Q - 1 - Q k0 - x,
                        // last first; they lie in three words, `sel` bytes into the first
                        const uint32_t* src = bs + 2 * (Q - 2 - Q * k0 - (int)(t >> 3));
                        uint8_t* dst = smem + lay.stage + (c % NS) * (S::CM * 128) + t * 16;
#pragma unroll
                        for (int e = 0; e < (S::CM + 3) / 4; e++) {
                            if (4 * e + 3 >= S::CM && 4 * e + (int)(t >> 3) >= S::CM) break;
                            const uint32_t w0 = src[-8 * e], w1 = src[1 - 8 * e], w2 = src[2 - 8 * e];
                            const uint32_t zl = __byte_perm(w0, w1, sel), zh = __byte_perm(w1, w2, sel);
                            *reinterpret_cast<uint4*>(dst + e * 512) =
                                make_uint4(tc_digits(zh, 0x4243), tc_digits(zh, 0x4041), tc_digits(zl, 0x4243), tc_digits(zl, 0x4041));
                        }
                        tc_fence_smem();
                        tc_warp_arrive(made + 8 * (c % NS));
                    }
                }
                if (ok) tc_warp_arrive(a_empty + 8 * buf);     // b's limbs are read
                cur = next;
            }
        } else {
            // ---- issuing: two warps take the blocks in turn (waiting, the
            // instructions and the commit cost one warp more than the tensor
            // core takes for a block)
            const uint32_t own = warp - (ND / 32 + 4);
            auto cur = fetch(first);
            for (uint64_t i = first; i < n && ok; i += step, p++) {
                const auto next = fetch(i + step < n ? i + step : i);
                const uint32_t buf = p % g.NA, D = tc_rows<P>(cur.L), tiles = tc_tiles<P>(cur.out_limbs);
                ok = tc_warp_wait(a_full + 8 * buf, (p / g.NA) & 1);
                for (uint32_t tau = 0; tau < tiles && ok; tau++) {
                    int klo, khi;
                    tc_krange(D, tau, klo, khi);
                    const uint32_t row0 = (sbase + buf * lay.abytes) / 16 + (uint32_t)((int)(128 * tau) - g.rho0);
                    for (int k0 = klo; k0 <= khi && ok; k0 += S::RB, c++) {
                        if (c % 2 != own) continue;
                        ok = tc_warp_wait(read + 8 * (c % NS), ((c / NS) & 1) ^ 1) &&
                             tc_warp_wait(made + 8 * (c % NS), (c / NS) & 1);
                        tc_fence_after();
                        if (ok && tc_elect()) {
                            const uint32_t da = tc_desc(row0 + (uint32_t)k0, g.R);
                            const uint32_t db = tc_desc((sbase + lay.stage) / 16 + (c % NS) * (S::CM * 8), 8);
#pragma unroll
                            for (int s = 0; s < S::STEPS; s++)
                                tc_mma<P>(tmem + (c % NS) * P, da + 16 * s / P + (16 * s % P / 8) * g.R, db + 16 * s, s > 0);
                            tc_commit(run + 8 * (c % NS));
                        }
                        __syncwarp();
                    }
                }
                if (ok && tc_elect()) tc_commit(a_empty + 8 * buf);
                __syncwarp();
                cur = next;
            }
            // no matrix instruction is in flight when the tensor memory is freed
            if (tc_elect()) tc_commit(done);
            __syncwarp();
            tc_bar_wait(done, 0);
        }
    } else {
        // ---- draining
        uint64_t* rows = reinterpret_cast<uint64_t*>(smem + lay.rows);
        uint64_t* ovf = reinterpret_cast<uint64_t*>(smem + lay.ovf);
        uint32_t* scratch = reinterpret_cast<uint32_t*>(smem + lay.scratch);
        // warp w of each four may read rows 32 w .. 32 w + 31
        const uint32_t tbase = tmem + (((warp & 3) * 32) << 16) + (warp >> 2) * CT;
        const uint32_t sg = (tid & 127) * S::H + (S::H - 1 - (warp >> 2));
        // (after a wait ran out: on without waiting, in step for the barriers, storing nothing)
        auto cur = fetch(first);
        for (uint64_t i = first; i < n; i += step) {
            const auto next = fetch(i + step < n ? i + step : i);
            const uint32_t D = tc_rows<P>(cur.L), tiles = tc_tiles<P>(cur.out_limbs);
            if (tid == 0) ovf[0] = 0;
            for (uint32_t tau = 0; tau < tiles; tau++) {
                int klo, khi;
                tc_krange(D, tau, klo, khi);
                uint32_t acc[CT], bias = 0;
#pragma unroll
                for (int j = 0; j < CT; j++) acc[j] = 0;
                // v + 2^23 has the integer v in its low bits
                for (int k0 = klo; k0 <= khi; k0 += S::RB, c++) {
                    if (ok) ok = tc_warp_wait(run + 8 * (c % NS), (c / NS) & 1);
                    tc_fence_after();
                    constexpr int W = CT % 32 == 0 ? 32 : 16;
#pragma unroll
                    for (int j = 0; j < CT; j += W) {
                        float v[W];
                        tc_ld(tbase + (c % NS) * P + j, v);
                        if (j + W == CT) {
                            tc_fence_before();
                            tc_warp_arrive(read + 8 * (c % NS));
                        }
#pragma unroll
                        for (int e = 0; e < W; e++) acc[j + e] += __float_as_uint(v[e] + 8388608.0f);
                    }
                    bias += 0x4B000000u;
                }
                // the thread's limbs and their overflow (below 2^33).  Accumulator
                // columns 8 n1 .. are limb Q - 1 - n1 of the row; thread sg's
                // limbs are sg QT .. of the tile.
                uint64_t d[QT], cy = 0;
#pragma unroll
                for (int k = 0; k < QT; k++) {
                    uint64_t u[2] = {0, 0};
#pragma unroll
                    for (int s = 0; s < 8; s++) u[s / 4] += (uint64_t)(acc[8 * (QT - 1 - k) + s] - bias) << (8 * (s % 4));
                    const uint64_t t = u[0] + cy;
                    d[k] = t + (u[1] << 32);
                    cy = (u[1] >> 32) + (d[k] < t);
                    if constexpr (S::H > 1) rows[sg * (QT + 1) + k] = d[k];
                }
                ovf[sg + 1] = cy;
                asm volatile("bar.sync 1, %0;" ::"r"(ND) : "memory");
                if constexpr (S::H > 1) {     // from here on thread tid has limbs tid QT ..
#pragma unroll
                    for (int k = 0; k < QT; k++) d[k] = rows[tid * (QT + 1) + k];
                    cy = ovf[tid + 1];
                }
                const uint64_t in = ovf[tid];
                uint64_t all = ~0ull;
                uint32_t gen = 0;
#pragma unroll
                for (int k = 0; k < QT; k++) {
                    const uint64_t add = k == 0 ? in : gen;
                    d[k] += add;
                    gen = d[k] < add;
                    all &= d[k];
                }
                const uint32_t prop = all == ~0ull && !gen;
                uint32_t cin = tc_carry_in(gen, prop, ND / 32, scratch);
                if (tid == ND - 1) ovf[0] = cy + (gen | (prop & cin));
#pragma unroll
                for (int k = 0; k < QT; k++) {
                    d[k] += cin;
                    cin = d[k] < cin;
                    rows[tid * (QT + 1) + k] = d[k];
                }
                asm volatile("bar.sync 1, %0;" ::"r"(ND) : "memory");
                const uint32_t x0 = tau * 128 * Q;
                for (uint32_t idx = tid; ok && idx < 128 * Q && x0 + idx < cur.out_limbs; idx += ND)
                    cur.store(x0 + idx, rows[idx + idx / QT]);
                asm volatile("bar.sync 1, %0;" ::"r"(ND) : "memory");
            }
            cur = next;
        }
    }
    if (!ok) report_gave_up(gave_up);
    tc_free<S::TMEM_COLS>(tmem);
}

}  // namespace bi
