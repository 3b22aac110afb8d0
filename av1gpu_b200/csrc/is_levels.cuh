// is_levels.cuh - levels of coefficients: quantisation without a division, levels packed 4 bits each, and the exact rate of a
// packed row.  Device code of the closed loop (is_small.cuh, grp_eval_x) and of the analysis (is_tiny.cuh); the CPU tests
// compile it for the host (tests/arith_host.cpp).
#pragma once
#include "is_hd.cuh"

namespace is {

typedef long long i64;
constexpr int FB = 3;                                            // fractional bits of the forward-transform coefficients
constexpr int TXC_2D = 0, TXC_HORIZ = 1;                         // av1core's tx classes (is_small.cuh checks these)
constexpr int EOB_STRIDE = 4, BASE_STRIDE = 5, BR_STRIDE = 5;    // entries a CDF of coeff_base_eob, coeff_base, coeff_br

// a quantiser step's divisions by 64 step as multiplications: (n M) >> 32 is n / (64 step) or one less (n < 2^32)
IS_HD uint32_t quant_recip(int step) { return 0xFFFFFFFFu / (64u * (unsigned)step); }

// level of a coefficient, its distance from the dequantised value and its packed forms (tx sizes of dequantisation
// denominator 1); no branch: the coefficients of a row are independent chains.  M: quant_recip(step)
template <int BD>
IS_DEV int quant_level(int v, int step, uint32_t M, i64 &dist) {
    const int a = abs(v), St = step << FB;
    const uint32_t n = (uint32_t)(8 * a + 3 * St), d = (uint32_t)(8 * St);
    uint32_t u = __umulhi(n, M);   // n / d or one less
    u += n - u * d >= d;
    const int l = a * 32 >= 21 * St ? min((int)u, 16383) : 0;
    // |dequantised|: 24 bits, clamped to 2^(7 + BD) below and one less above zero
    const int dq = min((l * step) & 0xFFFFFF, (1 << (7 + BD)) - (v >= 0 ? 1 : 0));
    const int df = a - dq * (1 << FB);
    dist += (i64)df * df;
    return v < 0 ? -l : l;
}

template <int LW> using PackedRow = typename std::conditional<LW == 4, unsigned long long, uint32_t>::type;   // 4 bits a column

// The neighbours of the contexts of a whole row (spec 8.3.2, Sig_Ref_Diff_Offset and Mag_Ref_Offset_With_Tx_Class; the library
// checks both against av1core's tables at upload): at(dr, dc) is the packed row dr rows below, moved dc columns left.
// base_sum: the sum of the base contexts' five (of at most 3 each: 4 bits a sum); br_third: the third neighbour of the ranges'
// contexts, beside (0, 1) and (1, 0).
template <typename Row, typename At>
IS_HD Row base_sum(bool c2, bool ch, const At &at) {
    return at(0, 1) + at(1, 0) + (c2 ? at(1, 1) + at(0, 2) + at(2, 0) : ch ? at(0, 2) + at(0, 3) + at(0, 4) : at(2, 0) + at(3, 0) + at(4, 0));
}
template <typename Row, typename At>
IS_HD Row br_third(bool c2, bool ch, const At &at) {
    return c2 ? at(1, 1) : ch ? at(0, 2) : at(2, 0);
}

// bits of the coefficients of row rr of a tx block of 1 << LW columns whose levels are packed 4 bits each: a0 .. a4 the rows
// rr .. rr + 4 capped at 3, b0 .. b2 the rows rr .. rr + 2 capped at 15 (a3, a4 and b2 are used by the vertical class only).
// Every sign counts one bit (the caller corrects the DC's).  tab: scan position | context offset << 8 of the row's
// positions; level(j): the signed level of column j.
template <int LW, int LH, typename Level>
IS_DEV int row_bits(int rr, PackedRow<LW> a0, PackedRow<LW> a1, PackedRow<LW> a2, PackedRow<LW> a3, PackedRow<LW> a4, PackedRow<LW> b0,
                    PackedRow<LW> b1, PackedRow<LW> b2, int cls, int eob, const uint16_t *tab, const uint16_t *cBase, const uint16_t *cEob,
                    const uint16_t *cBr, const Level &level) {
    typedef PackedRow<LW> Row;
    constexpr int W = 1 << LW, N = 1 << (LW + LH);
    int b = 0;
    const bool c2 = cls == TXC_2D, ch = cls == TXC_HORIZ;
    const Row m = base_sum<Row>(c2, ch, [&](int dr, int dc) -> Row { return (dr == 0 ? a0 : dr == 1 ? a1 : dr == 2 ? a2 : dr == 3 ? a3 : a4) >> (4 * dc); });
    const Row x2 = br_third<Row>(c2, ch, [&](int dr, int dc) -> Row { return (dr == 0 ? b0 : dr == 1 ? b1 : b2) >> (4 * dc); });
    // base symbols of the row, without branches: a coefficient past the end of block costs nothing, the last one takes
    // the end-of-block table
    Row big = 0;
#pragma unroll
    for (int j = 0; j < W; j++) {
        const int t = tab[j], c = t & 0xFF, l3 = (int)(a0 >> (4 * j)) & 3;
        int ctx = min(((int)(m >> (4 * j) & 15) + 1) >> 1, 4) + (t >> 8);
        if (j == 0) ctx = rr == 0 && cls == TXC_2D ? 0 : ctx;
        const int ectx = c == 0 ? 0 : c <= N / 8 ? 1 : c <= N / 4 ? 2 : 3;
        // (a valid entry for every coefficient: the last one's level is at least 1)
        const int bits = *(c == eob - 1 ? cEob + ectx * EOB_STRIDE + l3 - 1 : cBase + ctx * BASE_STRIDE + l3);
        b += (c < eob ? bits : 0) + (l3 ? 256 : 0);
        big |= (Row)(l3 > 2 ? 1 : 0) << (4 * j);
    }
    // the ranges and remainders of the levels above 2, one after the other
#pragma unroll 1
    for (; big; big &= big - 1) {
        const int sh = LW == 4 ? __ffsll((long long)big) - 1 : __ffs((int)big) - 1, j = sh >> 2;
        const int l = (int)(b0 >> sh) & 15, right = (int)((b0 >> sh) >> 4) & 15;
        int mg = right + ((int)(b1 >> sh) & 15) + ((int)(x2 >> sh) & 15);
        mg = min((mg + 1) >> 1, 6);
        const int near = cls == TXC_2D ? (rr < 2 && j < 2) : cls == TXC_HORIZ ? j == 0 : rr == 0;
        const uint16_t *cr = cBr + ((rr | j) == 0 ? mg : near ? mg + 7 : mg + 14) * BR_STRIDE;
        const int rem = l - 3, full = (rem * 11) >> 5;   // rem / 3: at most 4 symbols
        b += full * cr[3];
        if (full < 4) b += cr[rem - 3 * full];
        if (l == 15) {
            const int v = abs(level(j));
            if (v > 14) b += (2 * (31 - __clz(v - 14)) + 1) * 256;
        }
    }
    return b;
}

}  // namespace is
