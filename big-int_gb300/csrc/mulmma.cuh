// mulmma.cuh -- products of medium operands on the warp's matrix instruction
// (mma.sync m16n8k16, f16 digits, f32 sums), one warp an instance.
//
// The digit convolution as in multc.cuh, with rows of 8 digits: with a tile of
// 16 rows x 8 columns covering 128 product digits,
//     C_u[i][j] (digit 128 u + 8 i + j) = sum over s + g = 8 u of F_s G_g,
//     F_s[i][k] = a[16 s + 8 i + k],   G_g[k][j] = b[16 g + j - k],
// and both fragments depend on one index only.  For a residue r of s modulo 8
// (s = r + 8 v, g = 8 w - r) the tiles are all pairs of LT + 1 F's and LT G's,
// u = v + w: each fragment is loaded once and used LT times from registers, and
// the tiles follow the product's triangle in steps of 128 digits (1.28 of its
// digit products at 64 limbs, where 16 rows of 64 columns would take 2.25).
// F comes from one f16 copy of a by ldmatrix (rows overlap), G from two copies
// of b as pairs of neighbours in falling order, one for each parity.
//
// Digits are balanced, in [-128, 127]: byte k of x + 0x8080..80 less 128, and
// one more digit, the carry.  A sum of 1024 products of at most 2^14 is an
// exact f32; above 128 limbs the sums move to integers halfway, after residues
// 0 .. 3: at 256 limbs (2048 products in the last column) both halves are 1024.
//
// Bound by the tensor core's legacy rate (8 cycles an instruction and a quarter
// SM: 338 cycles an instance of 64 limbs) and the instructions around it (229),
// which overlap little: 516 cycles an instance, 65536 full products of 64 limbs
// 237 -> 118 us.  Loading each half of F once for residues r and r + 4 (a third
// less shared memory traffic) ran 12-15 % slower, on fewer warps.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace bi {

constexpr uint64_t MM_HALF = 0x8080808080808080ull;
constexpr int MM_CTA = 128;                      // four warps, four instances

// LT: operand limbs / 16, rounded up
template <int LT, bool FULL>
struct MmShape {
    static constexpr int N = 128 * LT;                       // operand digits
    static constexpr int U = FULL ? 2 * LT : LT;             // tiles of the product
    static constexpr int E = LT % 2 == 0 ? LT / 2 : LT;      // operand limbs a lane
    static constexpr int LANES = 16 * LT / E;                // lanes that hold operand limbs
    static constexpr int O = (16 * U + 31) / 32;             // product limbs a lane
    static constexpr bool FLUSH = LT > 8;                    // sums pass 2^24
    static constexpr int AW = (N + 128 + 144) / 2;           // words: a's digits, 128 zeros below and 144 places above
    static constexpr int BW = N / 2 + 16;                    // one copy of b's pairs, 8 zero words on each side
    static constexpr int OS = 8 * O + 4;                     // words of a lane's sums (an odd number of 16 bytes)
    static constexpr int WORDS = AW + 2 * BW > 32 * OS ? AW + 2 * BW : 32 * OS;   // shared words a warp
};

// two bytes of w less 128 as a pair of f16: 0x64bb is 1024 + bb
__device__ __forceinline__ uint32_t mm_digits(uint32_t w, uint32_t sel) {
    const uint32_t x = __byte_perm(w, 0x64646464u, sel);
    const __half2 y = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t*>(&y);
}

__device__ __forceinline__ void mm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mm_ldmatrix(uint32_t (&a)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                 : "r"(addr));
}

// carry into each lane of (g, p), and out of lane LANES - 1
template <int LANES>
__device__ __forceinline__ uint32_t mm_carry(uint32_t g, uint32_t p, uint32_t& cout) {
    const WarpCarry w = warp_carry_resolve(__ballot_sync(0xffffffffu, g | p), __ballot_sync(0xffffffffu, g), 0);
    cout = LANES == 32 ? w.cout : (w.carries >> (LANES & 31)) & 1u;
    return (w.carries >> (threadIdx.x & 31)) & 1u;
}

// The lane's limbs of an instance's operands, E lane .. : it.L limbs, it.a(x)
// and it.b(x) (it.a2, it.b2 two from an even x on where it.vec says so).
template <int E>
struct MmLimbs {
    uint64_t a[E], b[E];
    template <typename Item>
    __device__ __forceinline__ void load(const Item& it) {
        const uint32_t x0 = (uint32_t)E * (threadIdx.x & 31);
        if (E % 2 == 0 && it.vec) {
#pragma unroll
            for (int e = 0; e < E; e += 2) {
                const bool in = x0 + e < it.L;     // it.L is even
                const ulonglong2 va = in ? it.a2(x0 + e) : make_ulonglong2(0, 0), vb = in ? it.b2(x0 + e) : make_ulonglong2(0, 0);
                a[e] = va.x;
                a[(e + 1) % E] = va.y;
                b[e] = vb.x;
                b[(e + 1) % E] = vb.y;
            }
            return;
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
            const bool in = x0 + e < it.L;
            a[e] = in ? it.a(x0 + e) : 0;
            b[e] = in ? it.b(x0 + e) : 0;
        }
    }
};

// One product on a warp from the lanes' limbs (it.L <= 16 LT): it.store(x, v)
// takes limb x < it.out_limbs of it (it.store2 two from an even x on, where
// it.vec says so).  sw: MmShape::WORDS words of shared memory of the warp's own.
template <int LT, bool FULL, typename Item>
__device__ __forceinline__ void mm_product(const Item& it, const MmLimbs<MmShape<LT, FULL>::E>& raw, uint32_t* sw) {
    using S = MmShape<LT, FULL>;
    constexpr int E = S::E, U = S::U, O = S::O;
    const int lane = (int)(threadIdx.x & 31);
    uint32_t* a16 = sw + 64;                       // digit 0 of a
    uint32_t* be = sw + S::AW + 8;                 // pair k of be: b[2k], b[2k - 1]
    uint32_t* bo = be + S::BW;                     // of bo: b[2k + 1], b[2k]

    // ---- balanced digits
    {
        uint64_t ta[E], tb[E];
        uint32_t ga, gb, pa, pb, ca, cb;
        auto chain = [&](const uint64_t (&x)[E], uint64_t (&t)[E], uint32_t& g, uint32_t& p) {
            g = 0;
            p = 1;
#pragma unroll
            for (int e = 0; e < E; e++) {          // x + HALF overflows iff the sum is below HALF
                t[e] = x[e] + MM_HALF;
                const uint32_t over = t[e] < MM_HALF;
                t[e] += g;
                g = over | (t[e] < g);
                p &= t[e] == ~0ull;
            }
            p &= !g;
        };
        chain(raw.a, ta, ga, pa);
        chain(raw.b, tb, gb, pb);
        if (lane >= S::LANES) ga = gb = pa = pb = 0;
        uint32_t ia = mm_carry<S::LANES>(ga, pa, ca), ib = mm_carry<S::LANES>(gb, pb, cb);
#pragma unroll
        for (int e = 0; e < E; e++) {
            ta[e] += ia;
            ia = ta[e] < ia;
            tb[e] += ib;
            ib = tb[e] < ib;
        }
        uint64_t below = __shfl_up_sync(0xffffffffu, tb[E - 1], 1);
        if (lane == 0) below = MM_HALF;
        if (lane < S::LANES) {
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int x = E * lane + e;
                const uint32_t al = (uint32_t)ta[e], ah = (uint32_t)(ta[e] >> 32);
                *reinterpret_cast<uint4*>(a16 + 4 * x) =
                    make_uint4(mm_digits(al, 0x4140), mm_digits(al, 0x4342), mm_digits(ah, 0x4140), mm_digits(ah, 0x4342));
                const uint32_t bl = (uint32_t)tb[e], bh = (uint32_t)(tb[e] >> 32);
                *reinterpret_cast<uint4*>(bo + 4 * x) =
                    make_uint4(mm_digits(bl, 0x4041), mm_digits(bl, 0x4243), mm_digits(bh, 0x4041), mm_digits(bh, 0x4243));
                const uint32_t zl = __funnelshift_l((uint32_t)(below >> 32), bl, 8), zh = __funnelshift_l(bl, bh, 8);
                *reinterpret_cast<uint4*>(be + 4 * x) =
                    make_uint4(mm_digits(zl, 0x4041), mm_digits(zl, 0x4243), mm_digits(zh, 0x4041), mm_digits(zh, 0x4243));
                below = tb[e];
            }
        }
        // zeros around them, and the carry digits (f16 1.0 is 0x3c00)
        const uint4 zero = make_uint4(0, 0, 0, 0), first = make_uint4(ca ? 0x3c00u : 0u, 0, 0, 0);
        if (lane < 16) *reinterpret_cast<uint4*>(sw + 4 * lane) = zero;
        if (lane < 18) *reinterpret_cast<uint4*>(a16 + S::N / 2 + 4 * lane) = lane == 0 ? first : zero;
        if (lane < 16) (lane < 8 ? be - 8 + lane : bo - 16 + lane)[0] = 0;
        else if (lane > 16 && lane < 24) be[S::N / 2 + lane - 16] = 0;
        else if (lane >= 24) bo[S::N / 2 + lane - 24] = lane == 24 && cb ? 0x3c000000u : 0u;
        if (lane == S::LANES - 1)
            be[S::N / 2] = (mm_digits((uint32_t)(below >> 56) | 0x8000u, 0x4041) & 0xffff0000u) | (cb ? 0x3c00u : 0u);
        __syncwarp();
    }

    // ---- the tiles
    float c[U][4];
    int32_t ci[S::FLUSH ? U : 1][4];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            c[u][k] = 0;
            if (S::FLUSH) ci[u][k] = 0;
        }
    const int gq = lane >> 2, tq = lane & 3;
    const uint32_t* bp = (gq & 1 ? bo : be) + (gq >> 1) - tq;
    // ldmatrix: rows lane & 7 of the four 8 x 8 parts (rows 0.., rows 8.., then the same 8 digits on)
    const uint32_t ap = (uint32_t)__cvta_generic_to_shared(a16) +
                        16 * ((lane & 7) + ((lane >> 3) & 1) * 8) + 16 * (lane >> 4);
    auto first_tile = [&] {   // r = 0, w = 0
        const uint32_t b0 = bp[0], b1 = bp[-4];
#pragma unroll
        for (int v = 0; v < (FULL ? LT + 1 : LT); v++) {
            uint32_t a[4];
            mm_ldmatrix(a, ap + 256 * v);
            mm_mma(c[v], a, b0, b1);
        }
    };
    // before the move below, so that both halves hold at most 1024 products a
    // column; where there is none it comes last (first it cost full products of 113
    // to 128 limbs 6 %)
    if (S::FLUSH) first_tile();
    // (all residues unrolled run 8-10 % faster up to 64 limbs, slower above)
#pragma unroll (LT <= 5 ? 8 : 1)
    for (int r = 0; r < 8; r++) {
        uint32_t b0[LT], b1[LT];
#pragma unroll
        for (int w = 1; w <= LT; w++) {
            b0[w - 1] = bp[8 * (8 * w - r)];
            b1[w - 1] = bp[8 * (8 * w - r) - 4];
        }
#pragma unroll
        for (int v = -1; v < LT; v++) {
            uint32_t a[4];
            mm_ldmatrix(a, ap + 32 * (r + 8 * v));
#pragma unroll
            for (int w = 1; w <= LT; w++)
                if (v + w < U) mm_mma(c[v + w], a, b0[w - 1], b1[w - 1]);
        }
        if (FULL && r == 0) {     // a's carry digit, in the first row of F_(8 LT)
            uint32_t a[4];
            mm_ldmatrix(a, ap + 256 * LT);
#pragma unroll
            for (int w = 1; w < LT; w++) mm_mma(c[(LT + w) % U], a, b0[w - 1], b1[w - 1]);
        }
        if (S::FLUSH && r == 3) {
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    ci[u][k] = __float2int_rn(c[u][k]);
                    c[u][k] = 0;
                }
        }
    }
    if (!S::FLUSH) first_tile();
    __syncwarp();   // the operands are read

    // ---- sums to the lanes that own their limbs: limb l's eight in lane l / O
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int l = 16 * u + gq + 8 * h;
            int2 s = make_int2(__float2int_rn(c[u][2 * h]), __float2int_rn(c[u][2 * h + 1]));
            if (S::FLUSH) {
                s.x += ci[u][2 * h];
                s.y += ci[u][2 * h + 1];
            }
            *reinterpret_cast<int2*>(sw + l / O * S::OS + l % O * 8 + 2 * tq) = s;
        }
    __syncwarp();
    uint64_t d[O];
    int64_t cy = lane == 0 ? 0 : -(1ll << 40);     // taken off here, given back with the lane below's carry
#pragma unroll
    for (int k = 0; k < O; k++) {
        const int4 s0 = *reinterpret_cast<const int4*>(sw + lane * S::OS + 8 * k);
        const int4 s1 = *reinterpret_cast<const int4*>(sw + lane * S::OS + 8 * k + 4);
        const int64_t u0 = (int64_t)s0.x + ((int64_t)s0.y << 8) + ((int64_t)s0.z << 16) + ((int64_t)s0.w << 24);
        const int64_t u1 = (int64_t)s1.x + ((int64_t)s1.y << 8) + ((int64_t)s1.z << 16) + ((int64_t)s1.w << 24);
        const __int128 t = ((__int128)u1 << 32) + u0 + cy;
        d[k] = (uint64_t)t;
        cy = (int64_t)(t >> 64);
    }
    uint64_t in = (uint64_t)__shfl_up_sync(0xffffffffu, cy + (1ll << 40), 1);
    if (lane == 0) in = 0;
    uint64_t all = ~0ull;
    uint32_t gen = 0, out;
#pragma unroll
    for (int k = 0; k < O; k++) {
        const uint64_t add = k == 0 ? in : gen;
        d[k] += add;
        gen = d[k] < add;
        all &= d[k];
    }
    uint32_t cin = mm_carry<32>(gen, all == ~0ull && !gen, out);
#pragma unroll
    for (int k = 0; k < O; k++) {
        d[k] += cin;
        cin = d[k] < cin;
    }
    const uint32_t x0 = (uint32_t)O * lane;
    if (O % 2 == 0 && it.vec) {
#pragma unroll
        for (int k = 0; k < O; k += 2)
            if (x0 + k < it.out_limbs) it.store2(x0 + k, d[k], d[(k + 1) % O]);
    } else {
#pragma unroll
        for (int k = 0; k < O; k++)
            if (x0 + k < it.out_limbs) it.store(x0 + k, d[k]);
    }
    __syncwarp();   // sw is written again by the next instance
}

}  // namespace bi
