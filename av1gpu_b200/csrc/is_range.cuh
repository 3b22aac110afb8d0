// is_range.cuh - the arithmetic of the entropy coder's parallel form: CDF adaptation by entries, the range coder's steps from an
// unknown start, the code value as digits with carries.  Used by is_k_ent.cu; the CPU tests compile it for the host
// (tests/arith_host.cpp) against a serial coder.
#pragma once
#include "is_hd.cuh"

namespace is {

// A coder step of symbol s of an alphabet of nm1 + 1 symbols with bounds fl / fh (32768 x the probability of the
// symbols after s - 1 / after s): the upper half holds fl's bits from 6 on (the coder reads no lower ones; bit 15 set: fl
// is the whole range, symbol 0) and nm1 - s below them, the lower half fh
IS_DEV uint32_t step_hi(uint32_t fl, int below) { return (fl & 0xFFC0u) | (uint32_t)below; }
IS_DEV uint32_t pack_step(uint32_t fl, uint32_t fh, int s, int nm1) { return (step_hi(fl, nm1 - s) << 16) | fh; }
constexpr uint32_t STEP_FIRST = 1u << 31;
IS_DEV uint32_t step_ev(uint32_t e) { return (e >> 14) & 0xFCu; }   // 4 (nm1 - s)

// The CDFs in the inverse form of the bounds, a = 32768 - c: symbol s has fl = a[s - 1] (32768 for s = 0) and fh = a[s] (0
// for the last); spec 8.2.6's adaptation moves entries before s up by (32768 - a) >> rate and the others down by
// a >> rate, which is a += (T - a) >> rate with T = 32768 or 2^rate - 1 (the arithmetic shift rounds down).
// A lane holds one entry a: 4 lanes walk a CDF of up to 4 symbols, 16 a larger one.  The lane of entry s leaves the
// step's lower half, that of entry s - 1 the upper one (the last lane for s = 0), so a symbol costs no exchange between
// lanes.  One lane with the three entries of a small CDF, the bounds selected and packed, took 100 cycles a symbol.
IS_DEV void adapt_entry(int &a, int j, int s, int nm1, int last, int rate, uint16_t *at) {
    const int up = s > j;
    if (j == s) at[0] = (uint16_t)a;
    if (s ? j == s - 1 : j == last) at[1] = (uint16_t)step_hi(s ? (uint32_t)a : 32768u, nm1 - s);
    a += ((up ? 32768 : (1 << rate) - 1) - a) >> rate;
}
constexpr int RG_STATES = 128;
// one range step in a form with a short dependent chain.  The range is held as the float bits of the unnormalised
// range: its mantissa is the normalised one, so the renormalisation is an addition (the magic-number conversion of the
// 16-bit sum), and (r >> 8) in bits 16-23 gives ((r >> 8) p) >> 1 as the upper word of one product with p << 15.
struct RangeStep {
    uint32_t mu, mv, keep, k;          // p of fl and fh << 15 (0 for fl of a STEP_FIRST); 0xFFFF for a STEP_FIRST; the rest
};
IS_DEV RangeStep range_step(uint32_t e) {
    const bool first = e & STEP_FIRST;
    RangeStep s;
    s.mu = first ? 0u : (e & 0xFFC00000u) >> 7;
    s.mv = (e & 0xFFC0u) << 9;
    s.keep = first ? 0xFFFFu : 0u;
    s.k = 0x4B000000u + (first ? 0u - step_ev(e) : 4u);
    return s;
}
IS_DEV uint32_t range_bits(uint32_t r) { return __float_as_uint((float)r); }
IS_DEV uint32_t range_of(uint32_t b) { return ((b >> 8) & 0x7FFFu) | 0x8000u; }   // the normalised range
IS_DEV uint32_t range_next(uint32_t b, const RangeStep &s) {   // float bits of u - v
    const uint32_t r8 = (b & 0x7F0000u) | 0x800000u;
    const uint32_t rn = (__umulhi(r8, s.mu) + s.k) - __umulhi(r8, s.mv) + (range_of(b) & s.keep);
    return __float_as_uint(__uint_as_float(rn) - 8388608.0f);
}

// a step from range b (float bits): its term of the code value and the bits it shifts out (term | bits << 16), and the next range
IS_DEV uint32_t range_term(uint32_t e, uint32_t &b, uint32_t &bits) {
    const uint32_t r = range_of(b);
    const uint32_t u = (e & STEP_FIRST) ? r : (((r >> 8) * (e >> 22)) >> 1) + step_ev(e) + 4u;
    b = range_next(b, range_step(e));
    bits = 15u + 127u - (b >> 23);
    return (r - u) | (bits << 16);
}

// bytes of a tile whose steps shifted c bits out: the whole bytes sent while coding (the first after 9 bits), then the
// flush, which sends what is left of c + 1 bits
IS_DEV uint32_t rg_bytes(uint64_t c) {
    const uint64_t n0 = c >= 9 ? (c - 9) / 8 + 1 : 0;
    const int s = (int)((long long)c - 9 - 8 * (long long)n0) + 10;
    return (uint32_t)(n0 + (s + 7) / 8);
}
// a tile's digits: bit i of the payload (0 the first byte's top bit) is bit i + 16 from the top of the digits; a term of
// 16 bits after c shifted bits starts at bit c + 15
IS_DEV uint64_t rg_digits(uint32_t bytes) { return (bytes + 1) / 2 + 4; }
constexpr uint32_t RG_ROUND = 0x3FFF;   // the flush rounds up by this after the last step
// the parts of a term that starts a bits into a digit, in that digit and in the next
IS_DEV uint32_t digit_hi(uint32_t x, uint32_t a) { return x >> a; }
IS_DEV uint32_t digit_lo(uint32_t x, uint32_t a) { return (x << (16 - a)) & 0xFFFFu; }
// a digit with the two digits after it carried into it once: at most 65536
IS_DEV uint32_t digit_sum(uint32_t d0, uint32_t d1, uint32_t d2) {
    const uint32_t n0 = (d0 & 0xFFFFu) + (d1 >> 16), n1 = (d1 & 0xFFFFu) + (d2 >> 16);
    return (n0 & 0xFFFFu) + (n1 >> 16);
}
// 32 digits by their bits: those that generate a carry, and those that generate or propagate one.  The carries into them and
// out of the last are those of the addition of the two words (bit 0 the lowest digit)
IS_DEV uint32_t carries_in(uint32_t gen, uint32_t any, uint32_t cin) { return (any + gen + cin) ^ any ^ gen; }
IS_DEV uint32_t carry_out(uint32_t gen, uint32_t any, uint32_t cin) { return (uint32_t)(((uint64_t)any + gen + cin) >> 32); }
// byte at of a payload after c shifted bits: the flush sets bit c and clears those after it
IS_DEV uint8_t payload_byte(uint32_t x, uint64_t c, uint64_t at) {
    const long long last = (long long)c - 8 * (long long)at;
    if (last < 0) x = 0;
    else if (last < 8) x = (x & (0xFF00u >> last)) | (0x80u >> last);
    return (uint8_t)x;
}

}  // namespace is
