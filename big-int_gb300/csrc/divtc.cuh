// divtc.cuh -- long division by medium and large divisors, 31 or 63 quotient
// limbs at a time, the quotient block times the divisor on the tensor cores.
//
// One CTA divides one instance; the running remainder ("window")
// lies in shared memory, the divisor as f16 digits in the Toeplitz layout of
// multc.cuh, written once per instance.  Per block of quotient limbs:
//   estimate  q^ = the top LW = 32 or 64 window limbs times the LW-limb
//             reciprocal of the divisor's top LW limbs (Barrett), the upper
//             half of an LW-by-LW limb product over the CTA's threads;
//   product   q^ V as a digit convolution: q^'s core matrices in shared
//             memory, then one chain of matrix instructions;
//   subtract  each thread folds its accumulator row with its window limbs, one
//             carry lookahead joins the rows;
//   check     a negative window or one not below the divisor (q^ is at most
//             one too large or too small; on random operands with a chance of
//             about 2^-40 at 32 limbs, 2^-16 at 64) is corrected with the whole
//             CTA.
// Digits are balanced, in [-128, 127]: byte k of x + 0x8080..80 less 128.  A
// column then sums at most 249 or 505 products (q^ has LW - 1 limbs and a carry
// digit) of magnitude 2^14 at most, below 2^22 or 2^23: one accumulator holds a
// whole block exactly.  Blocks of 63 limbs halve what a block costs whatever its
// size -- the fold and the carries over the whole window, the barriers -- and
// pay for it with a longer reciprocal and four times the estimate's products.
//
// With W < V B^(LW-1), V's top bit set and K >= LW limbs, Wt and Vh the top LW
// limbs of W (K + LW - 1 limbs) and V and I the reciprocal floor((B^2LW - 1) / Vh):
// q^ = floor((floor(Wt (I - B^LW) / B^LW) + Wt) / B).  Against W / V the limbs
// below Vh and Wt, the roundings and the columns of the product that are left out
// weigh less than LW + 8 units of the limb that the last division by B takes off,
// and the error of I (dt_recip: below 2^29 or 2^57) at most as many: together far
// below one, so that q^ differs from floor(W / V) by at most one either way.  A
// divisor of fewer than LW limbs is scaled by B^(LW-K), which scales the
// remainder.
#pragma once

#include "divsmall.cuh"
#include "multc.cuh"
#include "multhread.cuh"

namespace bi {

constexpr uint64_t DT_HALF = 0x8080808080808080ull;
constexpr int DT_MAX_CORRECTIONS = 4;    // one is needed at most

// G: limbs a lane of LW = 32 G
template <int P, int G>
struct DtShape {
    static constexpr int LW = 32 * G, KB = LW - 1;               // reciprocal limbs, quotient limbs a block
    static constexpr int Q = P / 8;                              // limbs a row
    static constexpr int H = P >= 80 ? 2 : 1;                    // threads a row of the accumulator
    static constexpr int NT = 128 * H;                           // threads
    static constexpr int QT = Q / H;                             // limbs a thread
    static constexpr int T0 = -8 * LW;                           // first term: q^'s 8 KB + 1 digits, down to a multiple of 16
    static constexpr int STEPS = (P - T0) / 16;                  // matrix instructions a block
    static constexpr int CM = Q + 2 * STEPS - 1;                 // core matrices of q^
    static constexpr int KMIN = -((-T0 + P - 1) / P);            // row offset of the first term
    static constexpr int R = ((128 - KMIN) + 6) / 8 * 8 + 1;     // rows of the divisor's image, % 8 == 1
    static constexpr int MAX_K = 128 * Q - KB - 2;               // divisor limbs: the rows hold K + KB + 2
    static constexpr uint32_t TMEM_COLS = tc_pow2(P);
    // Place of window limb x: threads 8 limbs apart would all meet in the same
    // banks, so that the eight-limb shapes pad one limb after every eight
    // (1671 -> 988 us for 1048 divisions of 4000 by 2000 limbs; the others ran
    // 3-5 % slower with it)
    __host__ __device__ static constexpr int at(int x) { return QT % 8 == 0 ? x + (x >> 3) : x; }
    static constexpr int QLO = 2 * STEPS - LW, QHI = Q + 1;      // zero limbs below and above q^ that its blocks read
};

struct DtGeom {
    uint32_t mu, mv;       // limbs per dividend / divisor in the caller's type
    uint32_t MU, MV;       // the same in 64-bit limbs
    uint32_t UL;           // window limbs (places)
};

template <int P, int G>
struct DtSmem {
    uint32_t stage, win, inv, part, qraw, qh, cs, scratch, bar, total;
    __host__ __device__ explicit DtSmem(const DtGeom& g) {
        using S = DtShape<P, G>;
        stage = S::R * S::Q * 16;
        win = stage + S::CM * 128;
        inv = win + g.UL * 8;
        part = inv + 2 * S::LW * 8;
        qraw = part + 3 * S::NT * G * 8;
        qh = qraw + (S::QLO + S::LW + S::QHI + 1) / 2 * 16;
        cs = qh + (S::LW + 2) * 8;
        scratch = cs + (S::NT + 1) * 8;
        bar = scratch + 3 * 32 * 4;
        total = bar + 16;      // the barrier, tensor memory's address, whether a wait ran out
    }
};

__host__ __device__ inline DtGeom dt_geom(uint32_t mu, uint32_t mv, int wbytes) {
    DtGeom g;
    g.mu = mu;
    g.mv = mv;
    g.MU = wbytes == 8 ? mu : (mu + 1) / 2;
    g.MV = wbytes == 8 ? mv : (mv + 1) / 2;
    g.UL = (g.MU + 130) * 9 / 8 + 2;
    g.UL = g.UL / 2 * 2;
    return g;
}

// two bytes of w less 128 as a pair of f16 (see tc_digits)
__device__ __forceinline__ uint32_t dt_digits(uint32_t w, uint32_t sel) {
    const uint32_t x = __byte_perm(w, 0x64646464u, sel);
    const __half2 y = __hsub2(*reinterpret_cast<const __half2*>(&x), __half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480)));
    return *reinterpret_cast<const uint32_t*>(&y);
}

// x = x + y (sub: x - y) mod B^len for window limbs x from x0 on and y given
// by limb(i), the whole CTA; returns the carry (borrow) out.
template <typename S, typename Limb>
__device__ uint32_t dt_addsub(uint64_t* win, int x0, Limb limb, int len, bool sub, uint32_t* scratch) {
    constexpr int NT = S::NT;
    const int per = (len + NT - 1) / NT, lo = min((int)threadIdx.x * per, len), hi = min(lo + per, len);
    uint32_t c = 0, all = 1;
    for (int i = lo; i < hi; i++) {      // carries with none in
        const uint64_t y = limb(i), a = win[S::at(x0 + i)];
        const uint64_t s = sub ? a - y : a + y;
        const uint32_t k = sub ? a < y : s < y;
        const uint64_t t = sub ? s - c : s + c;
        c = k | (sub ? s < c : t < s);
        all &= sub ? t == 0 : t == ~0ull;
    }
    const uint32_t g = c, p = hi > lo ? (all & !c) : 1u;
    const uint32_t cin = block_carry_in(g, p, threadIdx.x == 0, scratch);
    c = cin;
    for (int i = lo; i < hi; i++) {
        const uint64_t y = limb(i), a = win[S::at(x0 + i)];
        const uint64_t s = sub ? a - y : a + y;
        const uint32_t k = sub ? a < y : s < y;
        const uint64_t t = sub ? s - c : s + c;
        c = k | (sub ? s < c : t < s);
        win[S::at(x0 + i)] = t;
    }
    return __syncthreads_or(threadIdx.x == NT - 1 && (hi > lo ? c : cin));
}

// The integer v: below 2^22, 1.5 2^23 + v has it in the low bits (two ALU
// instructions, where the conversion unit takes a quarter of their rate);
// below 2^23 the conversion.
template <int G>
__device__ __forceinline__ int32_t dt_int(float v) {
    if constexpr (G == 1) return (int32_t)(__float_as_uint(v + 12582912.0f) - 0x4B400000u);
    else return __float2int_rn(v);
}

// carry out of each lane's (g, p), carry-in 0: the carry into the lane, and out of lane 31
__device__ __forceinline__ uint32_t dt_lane_carry(uint32_t g, uint32_t p, uint32_t& cout) {
    const WarpCarry w = warp_carry_resolve(__ballot_sync(0xffffffffu, g | p), __ballot_sync(0xffffffffu, g), 0);
    cout = w.cout;
    return (w.carries >> (threadIdx.x & 31)) & 1u;
}

// Limb `lane` of sum over lanes t of (lo + mid B + hi B^2) B^t + extra B^t,
// hi small: the columns of a product and a number added to it, one a lane.
__device__ __forceinline__ uint64_t dt_fold(uint64_t lo, uint64_t mid, uint64_t hi, uint64_t extra) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t m = __shfl_up_sync(0xffffffffu, mid, 1), h = __shfl_up_sync(0xffffffffu, hi, 2);
    if (lane < 1) m = 0;
    if (lane < 2) h = 0;
    uint64_t sum = lo + m;
    uint32_t e = sum < m;
    sum += h;
    e += sum < h;
    sum += extra;
    e += sum < extra;
    uint32_t ein = __shfl_up_sync(0xffffffffu, e, 1), over;
    if (lane == 0) ein = 0;
    sum += ein;
    return sum + dt_lane_carry(sum < ein, sum == ~0ull, over);
}

// One step of dt_recip: P limbs of y to 2 P.
template <int P, int LW>
__device__ __forceinline__ void dt_recip_step(const uint64_t* v, uint64_t* y, uint64_t* t) {
    const int lane = (int)(threadIdx.x & 31);
    const uint64_t* V = v + LW - 2 * P;
    const uint64_t* Y = y + LW - P;
    // column P - 1 + lane of X Y, X's limbs above its top zero, lanes 0 .. P + 1
    auto column = [&](const uint64_t* X, uint64_t& c0, uint64_t& c1, uint32_t& c2) {
        c0 = c1 = 0;
        c2 = 0;
        if (lane <= P + 1) {
#pragma unroll
            for (int i = 0; i < P; i++) mac3(c0, c1, c2, X[P - 1 + lane - i], Y[i]);
        }
    };
    uint64_t c0, c1;
    uint32_t c2, over;
    const bool mid = lane >= 1 && lane <= P + 1;
    column(V, c0, c1, c2);
    // S = V + V Y / B^P mod B^(P+1) = -E, limb j on lane j + 1; E = B^2P (1 - V x)
    uint64_t S = dt_fold(c0, c1, c2, mid ? V[lane - 1] : 0);
    const bool pos = (__shfl_sync(0xffffffffu, S, P + 1) >> 63) == 0;
    const uint32_t one = dt_lane_carry(lane == 0, lane >= 1 && S == 0, over);
    if (!pos) S = ~S + one;
    if (mid) t[lane - 1] = S;
    __syncwarp();
    // D = |E| + |E| Y / B^P, limb j on lane j + 1
    column(t, c0, c1, c2);
    const uint64_t D = dt_fold(c0, c1, c2, mid ? S : 0);
    uint64_t dl = __shfl_down_sync(0xffffffffu, D, 1);
    if (lane > P) dl = 0;
    // y B^P -+ D, kept within [0, B^2P)
    const bool in = lane < 2 * P;
    const uint64_t a = lane >= P && in ? Y[lane - P] : 0;
    uint64_t r = pos ? a - dl : a + dl;
    const uint32_t cy = dt_lane_carry(in && (pos ? a < dl : r < dl), in && (pos ? r == 0 : r == ~0ull), over);
    r = pos ? r - cy : r + cy;
    // the carry out of lane 2 P - 1 is the carry into lane 2 P (there is none above lane 31)
    if (2 * P < 32) over = __shfl_sync(0xffffffffu, cy, (2 * P) & 31);
    if (over) r = pos ? 0 : ~0ull;
    __syncwarp();
    if (in) y[LW - 2 * P + lane] = r;
    __syncwarp();
}

// Two limbs a lane, 2 lane and 2 lane + 1: x += carries of (e[k] at limb k + 1)
// for the small e, and what runs on; returns the carry out of lane 31.
__device__ __forceinline__ uint32_t dt_carry2(uint64_t (&x)[2], const uint32_t (&e)[2]) {
    uint32_t e1 = e[1], in = __shfl_up_sync(0xffffffffu, e1, 1), over;
    if ((threadIdx.x & 31) == 0) in = 0;
    x[0] += in;
    const uint32_t c0 = e[0] + (x[0] < in);
    x[1] += c0;
    // what both limbs generate above the lane's own e[1]
    const uint32_t g = x[1] < c0, cy = dt_lane_carry(g, x[1] == ~0ull && x[0] == ~0ull && !g, over);
    x[0] += cy;
    x[1] += (x[0] < cy);
    return over + __shfl_sync(0xffffffffu, e1, 31);
}

// The columns of a product, two a lane as above, folded into limbs with
// `extra` added (dt_fold for two).
__device__ __forceinline__ uint32_t dt_fold2(const uint64_t (&lo)[2], const uint64_t (&mid)[2], const uint64_t (&hi)[2],
                                             const uint64_t (&extra)[2], uint64_t (&x)[2]) {
    const uint32_t lane = threadIdx.x & 31;
    uint64_t m = __shfl_up_sync(0xffffffffu, mid[1], 1), h0 = __shfl_up_sync(0xffffffffu, hi[0], 1),
             h1 = __shfl_up_sync(0xffffffffu, hi[1], 1);
    if (lane == 0) m = h0 = h1 = 0;
    const uint64_t ms[2] = {m, mid[0]}, hs[2] = {h0, h1};
    uint32_t e[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        x[k] = lo[k] + ms[k];
        e[k] = x[k] < ms[k];
        x[k] += hs[k];
        e[k] += x[k] < hs[k];
        x[k] += extra[k];
        e[k] += x[k] < extra[k];
    }
    return dt_carry2(x, e);
}

// dt_recip's last step for 64 limbs: 32 limbs of y to 64, two columns a lane.
__device__ __forceinline__ void dt_recip_last(const uint64_t* V, uint64_t* y, uint64_t* t) {
    constexpr int P = 32;
    const int lane = (int)(threadIdx.x & 31);
    const uint64_t* Y = y + P;
    uint64_t c0[2], c1[2], c2[2], ex[2], S[2];
    auto column = [&](const uint64_t* X) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            c0[k] = c1[k] = 0;
            uint32_t h = 0;
            if (2 * lane + k <= P + 1) {
#pragma unroll 8
                for (int i = 0; i < P; i++) mac3(c0[k], c1[k], h, X[P - 1 + 2 * lane + k - i], Y[i]);
            }
            c2[k] = h;
        }
    };
    // limb j of S and D is column j + 1: index 2 lane + k = j + 1
    column(V);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * lane + k;
        ex[k] = i >= 1 && i <= P + 1 ? V[i - 1] : 0;
    }
    dt_fold2(c0, c1, c2, ex, S);
    const bool pos = (__shfl_sync(0xffffffffu, S[1], (P + 1) / 2) >> 63) == 0;
    if (!pos) {                    // ~S + 1 from index 1 on
        uint64_t n0 = lane == 0 ? 0 : ~S[0], n1 = ~S[1];
        const uint32_t one = lane == 0;
        n1 += one;
        uint32_t over;
        // a lane passes the carry when both its limbs of ~S are all ones
        const uint32_t g = lane == 0 && n1 == 0, cy = dt_lane_carry(g, lane > 0 && n0 == ~0ull && n1 == ~0ull, over);
        n0 += cy;
        n1 += lane > 0 && n0 < cy;
        S[0] = n0;
        S[1] = n1;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * lane + k;
        if (i >= 1 && i <= P + 1) t[i - 1] = S[k];
        ex[k] = i >= 1 && i <= P + 1 ? S[k] : 0;
    }
    __syncwarp();
    column(t);
    uint64_t D[2];
    dt_fold2(c0, c1, c2, ex, D);
    // y B^P -+ D: limbs 2 lane, 2 lane + 1 of D are indexes one higher
    uint64_t d[2] = {D[1], __shfl_down_sync(0xffffffffu, D[0], 1)}, r[2];
    uint32_t e[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = 2 * lane + k;
        if (i > P) d[k] = 0;
        const uint64_t a = i >= P ? Y[i - P] : 0;
        r[k] = pos ? a - d[k] : a + d[k];
        e[k] = pos ? a < d[k] : r[k] < d[k];
    }
    __syncwarp();
    uint32_t over;
    if (pos) {                     // borrows: the same on the complements
        uint64_t n[2] = {~r[0], ~r[1]};
        over = dt_carry2(n, e);
        r[0] = ~n[0];
        r[1] = ~n[1];
    } else {
        over = dt_carry2(r, e);
    }
    if (over) r[0] = r[1] = pos ? 0 : ~0ull;
    y[2 * lane] = r[0];
    y[2 * lane + 1] = r[1];
    __syncwarp();
}

// y[0..LW) = about floor((B^2LW - 1) / V) - B^LW for V = v[0..LW), top bit set,
// v[LW] = 0, by one warp: Newton's iteration x -> x + x (1 - V x) on x = 1 + y
// (V in [1/2, 1), y a fraction), from the reciprocal of the top two limbs, with
// 1, 2, .. limbs of y giving twice as many.
//
// Error: let eta = (1 - V x) B^P at P limbs.  A step leaves out less than P + 2
// units of the residual (P of columns, 2 of V's limbs below) and less than P of
// the correction, so that eta' lies above -(P + 2), or -(2 P + 2) where eta is
// negative, and below max eta^2 + P.  The two-limb start has eta in [0, 1) but
// for 2 / B, which gives (-3, 2), (-6, 11), (-10, 125), (-18, 15633), then below
// 2^28 at 32 limbs and 2^56 at 64; y is off by at most 2 eta + 1 of its last
// unit, 2^29 or 2^57.  Random divisors have some 2^24 and 2^48.  (A one-limb
// start has eta up to 2, and 2^34 and 2^66 where the top limb is just above 2^63
// and the next all ones: there nine quotient blocks of ten were one or two short
// at 64 limbs.)  `t`: 66 limbs.
template <int LW>
__device__ __forceinline__ void dt_recip(const uint64_t* v, uint64_t* y, uint64_t* t) {
    const int lane = (int)(threadIdx.x & 31);
    t[lane] = 0;
    t[32 + lane] = 0;
    if (lane < 2) t[64 + lane] = 0;
    if (lane == 0) y[LW - 1] = recip_3by2(v[LW - 1], v[LW - 2], recip_limb(v[LW - 1]));
    __syncwarp();
    dt_recip_step<1, LW>(v, y, t);
    dt_recip_step<2, LW>(v, y, t);
    dt_recip_step<4, LW>(v, y, t);
    dt_recip_step<8, LW>(v, y, t);
    dt_recip_step<16, LW>(v, y, t);
    if constexpr (LW == 64) dt_recip_last(v, y, t);
}

// One division.  load_u(i) (i < g.MU), load_v(i) (i < g.MV) give limbs,
// store_q(i, x) for i < g.MU and store_r(i, x) for i < g.MV receive the
// results.  `phase` is the barrier's.  Every thread of the CTA calls it and
// gets the status: 0, 1 for a zero divisor, 2 when the corrections or a wait
// ran out.  After a wait that ran out the CTA's barrier may be behind `phase`: its
// later divisions wait no more and are 2 as well (dt_end has the rest).
template <int P, int G, typename LoadU, typename LoadV, typename StoreQ, typename StoreR>
__device__ __forceinline__ uint8_t dt_divide(const DtGeom& g, const DtSmem<P, G>& lay, uint8_t* smem, uint32_t tmem,
                                             uint32_t& phase, LoadU load_u, LoadV load_v, StoreQ store_q,
                                             StoreR store_r) {
    using S = DtShape<P, G>;
    constexpr int Q = S::Q, H = S::H, NT = S::NT, QT = S::QT, LW = S::LW, KB = S::KB;
    const int tid = (int)threadIdx.x, lane = tid & 31;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    uint64_t* win = reinterpret_cast<uint64_t*>(smem + lay.win);
    uint64_t* inv = reinterpret_cast<uint64_t*>(smem + lay.inv);
    uint64_t* part = reinterpret_cast<uint64_t*>(smem + lay.part);
    uint64_t* qraw = reinterpret_cast<uint64_t*>(smem + lay.qraw) + S::QLO;
    uint64_t* qh = reinterpret_cast<uint64_t*>(smem + lay.qh);
    int64_t* cs = reinterpret_cast<int64_t*>(smem + lay.cs);
    uint32_t* scratch = reinterpret_cast<uint32_t*>(smem + lay.scratch);
    const uint32_t sbase = tc_smem_addr(smem), bar = sbase + lay.bar;
    const int MU = (int)g.MU, MV = (int)g.MV;

    // ---- the divisor's size and shift
    uint32_t top = 0;
    for (int i = tid; i < MV; i += NT)
        if (load_v((uint32_t)i) != 0) top = (uint32_t)i + 1;
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) scratch[warp] = top;
    __syncthreads();
    const int K = (int)__reduce_max_sync(0xffffffffu, lane < NT / 32 ? scratch[lane] : 0u);
    __syncthreads();
    if (K == 0) {
        for (int i = tid; i < MU; i += NT) store_q((uint32_t)i, 0);
        for (int i = tid; i < MV; i += NT) store_r((uint32_t)i, 0);
        __syncthreads();
        return 1;
    }
    const int s = __clzll((long long)load_v((uint32_t)K - 1));
    const int Kp = K < LW ? LW : K, z = Kp - K;
    // limb x of the divisor scaled by 2^s B^z, zero from Kp on
    auto vlimb = [&](int x) -> uint64_t {
        x -= z;
        if (x < 0 || x >= K) return 0;
        uint64_t v = load_v((uint32_t)x) << s;
        if (s && x > 0) v |= load_v((uint32_t)x - 1) >> (64 - s);
        return v;
    };
    const int nb = (MU + 1 - K + KB - 1) / KB;
    const int len = nb * KB + Kp;
    const uint64_t vtop = vlimb(Kp - 1);

    // ---- the reciprocal of the top LW limbs, on one warp
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < G; k++) {
            qh[32 * k + lane] = vlimb(Kp - LW + 32 * k + lane);
            inv[LW + 32 * k + lane] = 0;
        }
        if (lane < 2) qh[LW + lane] = 0;
        __syncwarp();
        dt_recip<LW>(qh, inv, part);
    } else {
        // the other warps: the window, the dividend scaled by 2^s B^z
        for (int i = tid - 32; i < len; i += NT - 32) {
            const int x = i - z;
            uint64_t v = x >= 0 && x < MU ? load_u((uint32_t)x) << s : 0;
            if (s && x > 0 && x <= MU) v |= load_u((uint32_t)x - 1) >> (64 - s);
            win[S::at(i)] = v;
        }
        for (int i = tid - 32; i < S::R * Q; i += NT - 32) {
            const int row = i / Q, q = i - row * Q, x = (row + S::KMIN) * Q + q;
            if (x < 0 || x > Kp) *reinterpret_cast<uint4*>(smem + (q * S::R + row) * 16) = make_uint4(0, 0, 0, 0);
        }
        for (int i = tid - 32 - S::QLO; i < LW + S::QHI; i += NT - 32)
            if (i < 0 || i >= LW) qraw[i] = DT_HALF;
    }
    // ---- the divisor's balanced digits: Kp + 1 limbs of V + 0x8080..80
    {
        const int per = (Kp + 1 + NT - 1) / NT, lo = min(tid * per, Kp + 1), hi = min(lo + per, Kp + 1);
        uint32_t c = 0, all = 1;
        for (int x = lo; x < hi; x++) {
            const uint64_t a = vlimb(x) + DT_HALF, t = a + c;
            c = (a < DT_HALF) | (t < a);
            all &= t == ~0ull;
        }
        c = block_carry_in(c, hi > lo ? (all & !c) : 1u, tid == 0, scratch);
        for (int x = lo; x < hi; x++) {
            const uint64_t a = vlimb(x) + DT_HALF, t = a + c;
            c = (a < DT_HALF) | (t < a);
            const uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
            const int row = x / Q - S::KMIN, q = x % Q;
            *reinterpret_cast<uint4*>(smem + (q * S::R + row) * 16) =
                make_uint4(dt_digits(tl, 0x4140), dt_digits(tl, 0x4342), dt_digits(th, 0x4140), dt_digits(th, 0x4342));
        }
    }
    __syncthreads();

    volatile uint32_t* lost = reinterpret_cast<volatile uint32_t*>(smem + lay.bar + 12);
    bool ok = *lost == 0;
    int fixes = 0;
    for (int blk = nb - 1; blk >= 0; blk--) {
        const int w0 = blk * KB;          // the window: limbs w0 .. w0 + Kp + 30
        // ---- estimate: columns LW - 1 .. 2 LW - 2 of Wt inv, each warp its share of every column
#pragma unroll
        for (int k = 0; k < G; k++) {
            uint64_t c0 = 0, c1 = 0;
            uint32_t c2 = 0;
            const uint64_t* iv = inv + LW - 1 + 32 * k + lane - (int)warp;
#pragma unroll
            for (int e = 0; e < 32 * LW / NT; e++)
                mac3(c0, c1, c2, win[S::at(w0 + Kp - 1 + (int)warp + NT / 32 * e)], iv[-(NT / 32) * e]);
            const int at = (int)warp * LW + 32 * k + lane;
            part[at] = c0;
            part[G * NT + at] = c1;
            part[2 * G * NT + at] = c2;
        }
        __syncthreads();
        if (warp == 0) {
            uint64_t lo[G], mid[G], hi[G];
#pragma unroll
            for (int k = 0; k < G; k++) {
                lo[k] = mid[k] = hi[k] = 0;
#pragma unroll
                for (int e = 0; e < NT / 32; e++) {
                    const int at = LW * e + G * lane + k;
                    const uint64_t a = part[at], b = part[G * NT + at];
                    lo[k] += a;
                    const uint64_t cb = b + (lo[k] < a);
                    mid[k] += cb;
                    hi[k] += part[2 * G * NT + at] + (mid[k] < cb) + (cb < b);
                }
            }
            // limb i: the low part of column LW + i, the middle of the one below, the high of the next, and Wt
            uint64_t below_hi = __shfl_up_sync(0xffffffffu, hi[G - 1], 1), above_lo = __shfl_down_sync(0xffffffffu, lo[0], 1);
            if (lane == 0) below_hi = 0;
            if (lane == 31) above_lo = 0;
            uint64_t sum[G];
            uint32_t e[G], over;
#pragma unroll
            for (int k = 0; k < G; k++) {
                const uint64_t x = k + 1 < G ? lo[(k + 1) % G] : above_lo, y = k > 0 ? hi[(k + G - 1) % G] : below_hi;
                sum[k] = x + mid[k];
                e[k] = sum[k] < x;
                sum[k] += y;
                e[k] += sum[k] < y;
                const uint64_t wl = win[S::at(w0 + Kp - 1 + G * lane + k)];
                sum[k] += wl;
                e[k] += sum[k] < wl;
            }
            if constexpr (G == 1) {
                uint32_t ein = __shfl_up_sync(0xffffffffu, e[0], 1);
                if (lane == 0) ein = 0;
                sum[0] += ein;
                sum[0] += dt_lane_carry(sum[0] < ein, sum[0] == ~0ull, over);
                over += __shfl_sync(0xffffffffu, e[0], 31);
            } else {
                over = dt_carry2(sum, e);
            }
            // the quotient block is limbs 1 .. : balanced digits of it, and itself
            uint64_t qt[G], bt[G];
            qt[G - 1] = __shfl_down_sync(0xffffffffu, sum[0], 1);
            if constexpr (G == 2) qt[0] = sum[G - 1];
            uint32_t be[G];
#pragma unroll
            for (int k = 0; k < G; k++) {
                if (over) qt[k] = ~0ull;
                if (k == G - 1 && lane == 31) qt[k] = 0;
                qh[G * lane + k] = qt[k];
                bt[k] = qt[k] + DT_HALF;
                be[k] = bt[k] < DT_HALF;
            }
            if constexpr (G == 1) bt[0] += dt_lane_carry(be[0], bt[0] == ~0ull, over);
            else dt_carry2(bt, be);
#pragma unroll
            for (int k = 0; k < G; k++) qraw[G * lane + k] = bt[k];
        }
        __syncthreads();
        // ---- q^'s core matrices (multc.cuh's, of the balanced digits)
        {
            const uint32_t j1 = (tid & 7) + 1, sel = 0x3210u + 0x1111u * (j1 & 3);
            const uint32_t* src = reinterpret_cast<const uint32_t*>(qraw) + 2 * (Q - 2 - S::T0 / 8 - (tid >> 3)) + (j1 >> 2);
#pragma unroll
            for (int e = 0; e < (S::CM + NT / 8 - 1) / (NT / 8); e++) {
                if (NT / 8 * e + NT / 8 - 1 >= S::CM && NT / 8 * e + (tid >> 3) >= S::CM) break;
                const uint32_t w0 = src[-NT / 4 * e], w1 = src[1 - NT / 4 * e], w2 = src[2 - NT / 4 * e];
                const uint32_t zl = __byte_perm(w0, w1, sel), zh = __byte_perm(w1, w2, sel);
                *reinterpret_cast<uint4*>(smem + lay.stage + tid * 16 + e * (NT * 16)) =
                    make_uint4(dt_digits(zh, 0x4243), dt_digits(zh, 0x4041), dt_digits(zl, 0x4243), dt_digits(zl, 0x4041));
            }
        }
        tc_fence_smem();
        tc_fence_before();
        __syncthreads();
        if (warp == 0) {
            tc_fence_after();
            if (tc_elect()) {
                const uint32_t da = tc_desc(sbase / 16, S::R), db = tc_desc((sbase + lay.stage) / 16, 8);
#pragma unroll
                for (int st = 0; st < S::STEPS; st++) {
                    const int t = S::T0 + 16 * st, k = t >= 0 ? 0 : -((-t + P - 1) / P);
                    tc_mma<P>(tmem, da + (uint32_t)((k - S::KMIN) + (t - k * P) / 8 * S::R), db + 16 * st, st > 0);
                }
                tc_commit(bar);
            }
            __syncwarp();
        }
        if (ok) ok = tc_warp_wait(bar, phase);
        phase ^= 1;
        tc_fence_after();
        // ---- window -= q^ V.  Accumulator columns 8 n1 .. are limb Q - 1 - n1 of
        // the row; with two threads a row the second four warps have its low
        // half.  Segment sg is limbs QT sg ..; its carry out is signed, and made
        // nonnegative for the next segment by 2^30, which that one has taken off.
        const int half = H == 1 ? 0 : (int)(warp >> 2), sg = (tid & 127) * H + (H - 1 - half);
        const int x0 = QT * sg, lim = Kp + KB;
        uint64_t d[QT];
        int64_t c = sg == 0 ? 0 : -(1ll << 30);
        const uint32_t tb = tmem + (((warp & 3) * 32) << 16) + half * (P / H);
        auto limb_of = [&](int k, const float* v) {
            int64_t u0 = 0, u1 = 0;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                u0 += (int64_t)dt_int<G>(v[e]) << (8 * e);
                u1 += (int64_t)dt_int<G>(v[4 + e]) << (8 * e);
            }
            const __int128 t = (__int128)(unsigned __int128)(x0 + k < lim ? win[S::at(w0 + x0 + k)] : 0) + c - u0 - ((__int128)u1 << 32);
            d[k] = (uint64_t)t;
            c = (int64_t)(t >> 64);
        };
#pragma unroll
        for (int k = 0; k + 1 < QT; k += 2) {
            float v[16];
            tc_ld(tb + 8 * (QT - 2 - k), v);
            limb_of(k, v + 8);
            limb_of(k + 1, v);
        }
        if constexpr (QT % 2 == 1) {
            float v[8];
            tc_ld(tb, v);
            limb_of(QT - 1, v);
        }
        cs[sg + 1] = c + (1ll << 30);
        tc_fence_before();
        __syncthreads();
        const uint64_t in = sg == 0 ? 0 : (uint64_t)cs[sg];
        uint64_t all = ~0ull;
        uint32_t gen = 0;
#pragma unroll
        for (int k = 0; k < QT; k++) {
            const uint64_t add = k == 0 ? in : gen;
            d[k] += add;
            gen = d[k] < add;
            all &= d[k];
        }
        // carries between the segments, from every warp's masks
        const bool prop = all == ~0ull && !gen;
        {
            const uint32_t G = __ballot_sync(0xffffffffu, gen != 0), Pm = __ballot_sync(0xffffffffu, prop);
            if (lane == 0) {
                scratch[2 * warp] = G;
                scratch[2 * warp + 1] = Pm;
            }
        }
        __syncthreads();
        uint32_t cin = 0, crow = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint32_t gu = scratch[2 * r], pu = scratch[2 * r + 1];
            const uint32_t gl = H == 1 ? 0 : scratch[8 + 2 * r], pl = H == 1 ? ~0u : scratch[9 + 2 * r];
            const uint32_t G = gu | (pu & gl);
            const WarpCarry rc = warp_carry_resolve(G | (pu & pl), G, crow);
            if (r == (int)(warp & 3)) {
                const uint32_t low = rc.carries >> lane & 1u;
                cin = H == 1 || half ? low : (gl >> lane & 1u) | ((pl >> lane & 1u) & low);
            }
            crow = rc.cout;
        }
        bool neg = sg == NT - 1 && c + (int64_t)(gen | (prop & cin)) < 0;
#pragma unroll
        for (int k = 0; k < QT; k++) {
            const int x = x0 + k;
            d[k] += cin;
            cin = d[k] < cin;
            if (x < lim) win[S::at(w0 + x)] = d[k];
            // not below the divisor, perhaps
            if ((x == Kp && d[k] != 0) || (x == Kp - 1 && d[k] >= vtop)) neg = true;
        }
        if (__syncthreads_or(neg)) {
            // ---- correct: rare.  The limb above the window's Kp tells the sign.
            const bool low = (win[S::at(w0 + Kp)] >> 63) != 0;
            int step = 0;
            __syncthreads();
            for (int it = 0; it < DT_MAX_CORRECTIONS; it++) {
                if (low) {
                    step--;
                    if (dt_addsub<S>(win, w0, [&](int i) { return vlimb(i); }, lim, false, scratch)) break;
                } else {
                    if (dt_addsub<S>(win, w0, [&](int i) { return vlimb(i); }, lim, true, scratch)) {
                        dt_addsub<S>(win, w0, [&](int i) { return vlimb(i); }, lim, false, scratch);
                        break;
                    }
                    step++;
                }
                if (it == DT_MAX_CORRECTIONS - 1) fixes = 1;
            }
            if (tid == 0 && step != 0) {          // the quotient block by as much
                uint64_t k = (uint64_t)(step < 0 ? -step : step);
                for (int i = 0; i < KB && k; i++) {
                    const uint64_t x = qh[i];
                    qh[i] = step < 0 ? x - k : x + k;
                    k = step < 0 ? x < k : qh[i] < k;
                }
            }
            __syncthreads();
        }
        if (tid < KB && blk * KB + tid < MU) store_q((uint32_t)(blk * KB + tid), qh[tid]);
    }
    // ---- the quotient's zero limbs, the remainder scaled back
    for (int i = nb * KB + tid; i < MU; i += NT) store_q((uint32_t)i, 0);
    for (int i = tid; i < MV; i += NT) {
        uint64_t x = 0;
        if (i < K) {
            x = win[S::at(z + i)] >> s;
            if (s && i + 1 < K) x |= win[S::at(z + i + 1)] << (64 - s);
        }
        store_r((uint32_t)i, x);
    }
    if (!ok) *lost = 1;
    return __syncthreads_or(!ok || fixes) ? 2 : 0;
}

// The barrier and tensor memory of a CTA that divides, before and after all its
// divisions.  HELD > 0 (a test): the barrier waits for an arrival that never comes.
template <int P, int G, uint32_t HELD = 0>
__device__ __forceinline__ uint32_t dt_begin(const DtSmem<P, G>& lay, uint8_t* smem) {
    const uint32_t bar = tc_smem_addr(smem) + lay.bar;
    return tc_alloc<DtShape<P, G>::TMEM_COLS>(bar + 8, [&] {
        tc_bar_init(bar, 1 + HELD);
        *reinterpret_cast<volatile uint32_t*>(smem + lay.bar + 12) = 0;
    });
}

// A wait ran out: waits, with the same limit, until all that the CTA issued has
// ended, and tells the host.  `at` is a free word of shared memory.
__device__ __forceinline__ void dt_settle(uint32_t at, uint32_t* gave_up) {
    if (threadIdx.x == 0) {
        report_gave_up(gave_up);
        tc_bar_init(at, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (__shfl_sync(0xffffffffu, threadIdx.x >> 5, 0) == 0) {
        if (tc_elect()) tc_commit(at);         // by the thread that issues: all it issued
        __syncwarp();
    }
    tc_bar_wait(at, 0);
}

// (never run, but it moves the registers of the kernel's loop: 63-limb blocks keep
// theirs with the call, 2048 by 1024 limbs 565 / 573 us, the others without it, 512
// by 256 410 / 423)
static __device__ __noinline__ void dt_settle_call(uint32_t at, uint32_t* gave_up) { dt_settle(at, gave_up); }

template <int P, int G>
__device__ __forceinline__ void dt_end(const DtSmem<P, G>& lay, uint8_t* smem, uint32_t tmem, uint32_t* gave_up) {
    __syncthreads();
    if (*reinterpret_cast<volatile uint32_t*>(smem + lay.bar + 12) != 0) {
        if constexpr (G == 1) dt_settle(tc_smem_addr(smem) + lay.cs, gave_up);
        else dt_settle_call(tc_smem_addr(smem) + lay.cs, gave_up);
    }
    tc_free<DtShape<P, G>::TMEM_COLS>(tmem);
}

}  // namespace bi
