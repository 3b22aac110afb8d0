// Host build of the kernels' arithmetic that needs no table of av1core (is_levels.cuh, is_range.cuh), with plain restatements
// beside it: the exact rate and quantisation of a coefficient by its definition, a serial multi-symbol range coder with CDF
// adaptation, and the decoder of spec 8.2.  Test infrastructure only.
#include "is_levels.cuh"
#include "is_range.cuh"

#include <random>
#include <vector>

using namespace is;

namespace {

typedef std::mt19937_64 Rng;
int pick(Rng &g, int lo, int hi) { return lo + (int)(g() % (uint64_t)(hi - lo + 1)); }

// neighbours of the base and the range contexts (spec 8.3.2), (row, column): 2D, HORIZ, VERT
const int kSig[3][5][2] = {{{0, 1}, {1, 0}, {1, 1}, {0, 2}, {2, 0}}, {{0, 1}, {1, 0}, {0, 2}, {0, 3}, {0, 4}}, {{1, 0}, {0, 1}, {2, 0}, {3, 0}, {4, 0}}};
const int kMag[3][3][2] = {{{0, 1}, {1, 0}, {1, 1}}, {{0, 1}, {1, 0}, {0, 2}}, {{0, 1}, {1, 0}, {2, 0}}};

template <int LW, int LH> int levels_size(Rng &g, int rounds) {
    constexpr int W = 1 << LW, H = 1 << LH, N = W * H;
    for (int it = 0; it < rounds; it++) {
        uint16_t base[42 * 5], eobc[4 * 4], br[21 * 5], tab[N];
        for (auto &v : base) v = (uint16_t)pick(g, 0, 4000);
        for (auto &v : eobc) v = (uint16_t)pick(g, 0, 4000);
        for (auto &v : br) v = (uint16_t)pick(g, 0, 4000);
        const int cls = pick(g, 0, 2);
        int order[N];
        for (int i = 0; i < N; i++) order[i] = i;
        std::shuffle(order, order + N, g);            // (any scan)
        for (int c = 0; c < N; c++) tab[order[c]] = (uint16_t)(c | pick(g, 0, 37) << 8);
        int q[N], eob = 0;
        const int kind = pick(g, 0, 4), fill = pick(g, 1, 100);
        for (int i = 0; i < N; i++) {
            int v = 0;
            if (pick(g, 1, 100) <= fill)
                v = kind == 0 ? pick(g, 0, 3) : kind == 1 ? pick(g, 0, 20) : kind == 2 ? 16383 : kind == 3 ? (pick(g, 0, 1) ? 15 : 14) : pick(g, 0, 16383);
            q[i] = pick(g, 0, 1) ? -v : v;
            if (v) eob = std::max(eob, (tab[i] & 0xFF) + 1);
        }
        if (!eob) continue;
        // by definition
        long want = 0;
        for (int i = 0; i < N; i++) {
            const int c = tab[i] & 0xFF, off = tab[i] >> 8, row = i / W, col = i % W, a = std::abs(q[i]);
            if (c >= eob) continue;
            auto lev = [&](int dr, int dc, int cap) { return row + dr < H && col + dc < W ? std::min(std::abs(q[(row + dr) * W + col + dc]), cap) : 0; };
            if (c == eob - 1) {
                want += eobc[(c == 0 ? 0 : c <= N / 8 ? 1 : c <= N / 4 ? 2 : 3) * 4 + std::min(a, 3) - 1];
            } else {
                int mag = 0;
                for (auto &k : kSig[cls]) mag += lev(k[0], k[1], 3);
                const int ctx = cls == 0 && i == 0 ? 0 : std::min((mag + 1) >> 1, 4) + off;
                want += base[ctx * 5 + std::min(a, 3)];
            }
            if (a) want += 256;
            if (a > 2) {
                int mag = 0;
                for (auto &k : kMag[cls]) mag += lev(k[0], k[1], 15);
                mag = std::min((mag + 1) >> 1, 6);
                const bool near = cls == 0 ? row < 2 && col < 2 : cls == 1 ? col == 0 : row == 0;
                const uint16_t *cb = br + (i == 0 ? mag : near ? mag + 7 : mag + 14) * 5;
                int rem = std::min(a, 15) - 3;
                for (int k = 0; k < 4; k++) {
                    const int s = std::min(rem, 3);
                    want += cb[s];
                    rem -= s;
                    if (s < 3) break;
                }
            }
            if (a > 14) {
                int bits = 0;
                while ((a - 14) >> (bits + 1)) bits++;
                want += (2 * bits + 1) * 256;
            }
        }
        // packed
        PackedRow<LW> p3[H + 4] = {}, p15[H + 4] = {};
        for (int i = 0; i < N; i++) {
            p3[i / W] |= (PackedRow<LW>)std::min(std::abs(q[i]), 3) << (4 * (i % W));
            p15[i / W] |= (PackedRow<LW>)std::min(std::abs(q[i]), 15) << (4 * (i % W));
        }
        long got = 0;
        for (int r = 0; r < H; r++)
            got += row_bits<LW, LH>(r, p3[r], p3[r + 1], p3[r + 2], p3[r + 3], p3[r + 4], p15[r], p15[r + 1], p15[r + 2], cls, eob, tab + r * W, base,
                                    eobc, br, [&](int j) -> int { return q[r * W + j]; });
        if (got != want) return it + 1;
    }
    return 0;
}

template <int BD> int quant_one(int v, int step) {
    const int a = std::abs(v), S = step << FB;
    long l = 0;
    if ((long)a * 32 >= 21l * S) l = std::min((8l * a + 3l * S) / (8l * S), 16383l);
    long dq = (l * step) & 0xFFFFFF;
    dq = v < 0 ? -std::min(dq, 1l << (7 + BD)) : std::min(dq, (1l << (7 + BD)) - 1);
    const long df = (long)v - dq * (1 << FB);
    i64 dist = 5;
    const int got = quant_level<BD>(v, step, quant_recip(step), dist);
    return got == (v < 0 ? -l : l) && dist == 5 + df * df ? 0 : 1;
}

// ---- the serial coder: spec-format CDFs (cumulative, then the counter), adapted symbol by symbol ----
enum { ADAPT = 0, BIT = 1, SPLIT_H = 2, SPLIT_V = 3 };   // a symbol word's kind; alphabet - 1 << 2, symbol << 6, CDF << 16

void adapt(uint16_t *cdf, int s, int n) {
    const int rate = 3 + (cdf[n] > 15) + (cdf[n] > 31) + (n > 3 ? 2 : 1);
    for (int i = 0; i < n - 1; i++) cdf[i] = (uint16_t)(i < s ? cdf[i] - (cdf[i] >> rate) : cdf[i] + ((32768 - cdf[i]) >> rate));
    cdf[n] = (uint16_t)(cdf[n] + (cdf[n] < 32));
}
// probability of the partitions that split the bottom (H) or right (V) half at the frame edge, of 32768
int split_mass(const uint16_t *cdf, int n, bool vert) {
    static const int h[6] = {2, 3, 4, 6, 7, 9}, v[6] = {1, 3, 4, 5, 6, 8};   // partitions (spec 9.3.1's two lists)
    int m = 0;
    for (int k = 0; k < 6; k++) {
        const int p = vert ? v[k] : h[k];
        if (p < n) m += cdf[p] - cdf[p - 1];
    }
    return m;
}
// a word's interval: 32768 x the probability of the symbols after s - 1 and after s
void bounds(uint32_t w, uint16_t *cdfs, uint32_t &fl, uint32_t &fh, int &below) {
    const int kind = w & 3, nm1 = (w >> 2) & 15, s = (w >> 6) & 15;
    uint16_t *c = cdfs + (w >> 16);
    below = nm1 - s;
    if (kind == ADAPT) {
        fl = s ? 32768u - c[s - 1] : 32768u;
        fh = 32768u - c[s];
        adapt(c, s, nm1 + 1);
    } else {
        const uint32_t m = kind == BIT ? 16384u : (uint32_t)split_mass(c, 10, kind == SPLIT_V);
        fl = s ? m : 32768u;
        fh = s ? 0u : m;
        below = 1 - s;
    }
}

}  // namespace

extern "C" {

int levels_check(unsigned seed, int rounds) {
    Rng g(seed);
    int r;
    if ((r = levels_size<2, 2>(g, rounds))) return 1000000 + r;
    if ((r = levels_size<3, 3>(g, rounds))) return 2000000 + r;
    if ((r = levels_size<2, 3>(g, rounds))) return 3000000 + r;
    if ((r = levels_size<3, 2>(g, rounds))) return 4000000 + r;
    if ((r = levels_size<2, 4>(g, rounds))) return 5000000 + r;
    if ((r = levels_size<4, 2>(g, rounds))) return 6000000 + r;
    return 0;
}

// every value around a level's thresholds for the steps given, and random ones
int quant_check(const int *steps, int n, unsigned seed, int rounds) {
    Rng g(seed);
    for (int k = 0; k < n; k++) {
        for (int l = 0; l < 400; l++)
            for (int d = -2; d <= 2; d++)
                for (int f : {21 * 8 * steps[k] / 32, 5 * steps[k]}) {
                    const int v = 8 * steps[k] * l + f + d;
                    if (v > (1 << 21)) continue;
                    if (quant_one<8>(v, steps[k]) || quant_one<8>(-v, steps[k]) || quant_one<10>(v, steps[k]) || quant_one<10>(-v, steps[k])) return k + 1;
                }
        for (int i = 0; i < rounds; i++) {
            const int v = pick(g, -(1 << 21), 1 << 21) >> pick(g, 0, 20);
            if (quant_one<8>(v, steps[k]) || quant_one<10>(v, steps[k])) return -(k + 1);
        }
    }
    return 0;
}

// The serial coder: the code value is the sum of the steps' (r - u) after the bits shifted out before them, added bit by bit;
// then rounded up to the shortest end that stays in the last interval.  Returns the payload's bytes.
long serial_code(const uint32_t *words, long n, const uint16_t *cdf, long ncdf, uint8_t *out, long cap) {
    std::vector<uint16_t> c(cdf, cdf + ncdf);
    std::vector<uint8_t> bit(n * 15 + 64, 0);   // bit[0] is above the payload (never set at the end)
    auto add = [&](uint32_t x, long at) {       // 16 bits, the first at bit[at]
        int carry = 0;
        for (long k = at + 15; k >= 0 && (x || carry || k >= at); k--) {
            const int t = bit[k] + (int)(x & 1) + carry;
            bit[k] = t & 1;
            carry = t >> 1;
            x >>= 1;
            if (k <= at && !carry) break;
        }
    };
    uint32_t r = 32768;
    long shifted = 0;
    for (long i = 0; i < n; i++) {
        uint32_t fl, fh;
        int below;
        bounds(words[i], c.data(), fl, fh, below);
        const uint32_t v = (((r >> 8) * (fh >> 6)) >> 1) + 4 * below;
        const uint32_t u = fl >= 32768 ? r : (((r >> 8) * (fl >> 6)) >> 1) + 4 * (below + 1);
        add(r - u, shifted);
        for (r = u - v; r < 32768; r <<= 1) shifted++;
    }
    add(0x3FFF, shifted);
    bit[shifted + 1] = 1;                       // payload bit `shifted`: the last one
    for (size_t k = shifted + 2; k < bit.size(); k++) bit[k] = 0;
    const long bytes = (shifted + 1 + 7) / 8;
    if (bytes > cap || bit[0]) return -1;
    for (long k = 0; k < bytes; k++) {
        out[k] = 0;
        for (int b = 0; b < 8; b++) out[k] = (uint8_t)(out[k] << 1 | bit[1 + 8 * k + b]);
    }
    return bytes;
}

// The decoder of spec 8.2 on a payload: the index of the first symbol it reads otherwise, or n.
long spec_decode(const uint8_t *data, long sz, const uint32_t *words, long n, const uint16_t *cdf, long ncdf) {
    std::vector<uint16_t> c(cdf, cdf + ncdf);
    long at = 0;
    auto f = [&](int k) {
        uint32_t x = 0;
        for (; k > 0; k--, at++) x = x << 1 | (at < 8 * sz ? (data[at >> 3] >> (7 - (at & 7))) & 1u : 0u);
        return x;
    };
    int numBits = (int)std::min<long>(sz * 8, 15);
    uint32_t value = ((1u << 15) - 1) ^ (f(numBits) << (15 - numBits)), range = 1u << 15;
    long maxBits = 8 * sz - 15;
    for (long i = 0; i < n; i++) {
        const int kind = words[i] & 3, nm1 = (words[i] >> 2) & 15, want = (words[i] >> 6) & 15;
        uint16_t *p = c.data() + (words[i] >> 16), two[3];
        const int N = kind == ADAPT ? nm1 + 1 : 2;
        if (kind != ADAPT) {
            two[0] = (uint16_t)(32768 - (kind == BIT ? 16384 : split_mass(p, 10, kind == SPLIT_V)));
            two[1] = 32768;
            two[2] = 0;
        }
        const uint16_t *q = kind == ADAPT ? p : two;
        uint32_t cur = range, prev;
        int s = -1;
        do {
            s++;
            prev = cur;
            const uint32_t ff = (1u << 15) - q[s];
            cur = (((range >> 8) * (ff >> 6)) >> 1) + 4 * (N - s - 1);
        } while (value < cur);
        range = prev - cur;
        value -= cur;
        int bits = 0;
        while ((range << bits) < 32768) bits++;
        range <<= bits;
        numBits = (int)std::min<long>(bits, std::max<long>(0, maxBits));
        const uint32_t pad = f(numBits) << (bits - numBits);
        value = pad ^ (((value + 1) << bits) - 1);
        maxBits -= bits;
        if (s != want) return i;
        if (kind == ADAPT) {
            const int rate = 3 + (p[N] > 15) + (p[N] > 31) + std::min(N >= 4 ? (N >= 8 ? (N >= 16 ? 4 : 3) : 2) : 1, 2);
            int tmp = 0;
            for (int k = 0; k < N - 1; k++) {
                if (k == s) tmp = 32768;
                if (tmp < p[k]) p[k] = (uint16_t)(p[k] - ((p[k] - tmp) >> rate));
                else p[k] = (uint16_t)(p[k] + ((tmp - p[k]) >> rate));
            }
            p[N] = (uint16_t)(p[N] + (p[N] < 32));
        }
    }
    return n;
}

// The kernels' way on the host, with their arithmetic: lists by CDF, an entry a lane; chunks from every start, strung together;
// terms into digits; carries 32 x 32 digits at a time.  chunk: nominal steps of a chunk.
long parallel_code(const uint32_t *words, long n, const uint16_t *cdf, long ncdf, long chunk, uint8_t *out, long cap) {
    std::vector<uint32_t> step(n);
    std::vector<std::vector<uint32_t>> list(ncdf);
    for (long i = 0; i < n; i++) {
        const uint32_t w = words[i], s = (w >> 6) & 15;
        if ((w & 3) == BIT) step[i] = pack_step(s ? 16384u : 32768u, s ? 0u : 16384u, (int)s, 1);
        else list[w >> 16].push_back((uint32_t)i);
    }
    for (long o = 0; o < ncdf; o++) {
        if (list[o].empty()) continue;
        int nm1 = 9;                           // (split words alone: a partition CDF of 10)
        for (uint32_t i : list[o]) if ((words[i] & 3) == ADAPT) nm1 = (words[i] >> 2) & 15;
        const int lanes = nm1 > 3 ? 16 : 4, e = nm1 > 2 ? 5 : 4;
        int a[16];
        for (int j = 0; j < lanes; j++) a[j] = j < nm1 ? 32768 - cdf[o + j] : 0;
        int count = cdf[o + nm1 + 1];
        for (uint32_t i : list[o]) {
            const int kind = words[i] & 3, s = (words[i] >> 6) & 15;
            if (kind != ADAPT) {
                uint16_t c[12];
                for (int j = 0; j <= nm1; j++) c[j] = (uint16_t)(32768 - a[j]);
                const uint32_t m = (uint32_t)split_mass(c, nm1 + 1, kind == SPLIT_V);
                step[i] = pack_step(s ? m : 32768u, s ? 0u : m, s, 1);
                continue;
            }
            uint16_t at[2] = {0, 0};
            for (int j = 0; j < lanes; j++) adapt_entry(a[j], j, s, nm1, lanes - 1, e + (count > 15) + (count > 31), at);
            step[i] = (uint32_t)at[1] << 16 | at[0];
            count++;
        }
    }
    // chunks
    const long nc = (n + chunk - 1) / chunk;
    std::vector<long> start(nc, -1);
    for (long k = 0; k < nc; k++) {
        if (k == 0) start[k] = 0;
        else
            for (long j = k * chunk; j < std::min(n, (k + 1) * chunk); j++)
                if (!(step[j] & STEP_FIRST)) { start[k] = j; break; }
    }
    auto end = [&](long k) {
        for (long q = k + 1; q < nc; q++) if (start[q] >= 0) return start[q];
        return n;
    };
    std::vector<uint32_t> first(nc, 0), last(nc, 0);
    uint32_t cur = 0;
    for (long k = 0; k < nc; k++) {
        first[k] = cur;
        if (start[k] < 0) continue;
        uint32_t map[RG_STATES];
        for (int t = 0; t < RG_STATES; t++) {
            uint32_t b = range_bits(k == 0 ? 0x8000u : (uint32_t)(128 + t) << 8);
            for (long j = start[k]; j < end(k); j++) b = range_next(b, range_step(step[j]));
            map[t] = (b >> 16) & 0x7F;
        }
        cur = map[cur];
    }
    std::vector<uint32_t> term(n);
    uint64_t c = 0;
    std::vector<uint64_t> place(n);
    for (long k = 0; k < nc; k++) {
        if (start[k] < 0) continue;
        uint32_t b = range_bits(k == 0 ? 0x8000u : (128 + first[k]) << 8);
        for (long j = start[k]; j < end(k); j++) {
            uint32_t d;
            place[j] = c;
            term[j] = range_term(step[j], b, d) & 0xFFFFu;
            c += d;
        }
        last[k] = range_of(b) & 0xFF;
        long q = k - 1;
        while (q >= 0 && start[q] < 0) q--;
        if (k) term[start[k]] += last[q];
        if (term[start[k]] > 0xFFFF) return -2;
    }
    const uint32_t bytes = rg_bytes(c);
    const uint64_t nd = rg_digits(bytes);
    if ((long)bytes > cap) return -1;
    std::vector<uint64_t> dig(nd + 2, 0);
    auto put = [&](uint32_t x, uint64_t at) {
        const uint64_t q = at + 15;
        dig[q >> 4] += digit_hi(x, (uint32_t)q & 15);
        dig[(q >> 4) + 1] += digit_lo(x, (uint32_t)q & 15);
    };
    for (long j = 0; j < n; j++) put(term[j], place[j]);
    put(RG_ROUND, c);
    for (uint64_t d : dig) if (d >> 32) return -3;
    uint32_t cin = 0;
    for (uint64_t b0 = 0; b0 < nd; b0 += 1024) {
        uint32_t v[1024], gen[32] = {}, any[32] = {}, G = 0, P = 0;
        for (int k = 0; k < 1024; k++) {
            const uint64_t i = b0 + k, m = nd - 1 - i;
            v[k] = i < nd ? digit_sum((uint32_t)dig[m], m + 1 < nd ? (uint32_t)dig[m + 1] : 0, m + 2 < nd ? (uint32_t)dig[m + 2] : 0) : 0;
            gen[k >> 5] |= (uint32_t)(v[k] > 0xFFFFu) << (k & 31);
            any[k >> 5] |= (uint32_t)(v[k] >= 0xFFFFu) << (k & 31);
        }
        for (int w = 0; w < 32; w++) {
            G |= carry_out(gen[w], any[w], 0) << w;
            P |= carry_out(gen[w], any[w], 1) << w;
        }
        const uint32_t cw = carries_in(G, P, cin);
        cin = carry_out(G, P, cin);
        for (int k = 0; k < 1024; k++) {
            const uint64_t i = b0 + k;
            if (i >= nd) break;
            const uint64_t m = nd - 1 - i;
            const uint32_t x = (v[k] + (carries_in(gen[k >> 5], any[k >> 5], (cw >> (k >> 5)) & 1) >> (k & 31) & 1)) & 0xFFFFu;
            if (m > 0)
                for (int z = 0; z < 2; z++)
                    if (2 * (m - 1) + z < bytes) out[2 * (m - 1) + z] = payload_byte((z ? x : x >> 8) & 0xFFu, c, 2 * (m - 1) + z);
        }
    }
    return bytes;
}

// carries_in / carry_out over 32 digits, against a carry taken from digit to digit
int carry_check(unsigned seed, int rounds) {
    Rng g(seed);
    for (int it = 0; it < rounds; it++) {
        uint32_t gen = 0, any = 0, in = 0;
        const uint32_t cin = (uint32_t)g() & 1;
        uint32_t cy = cin;
        const int pg = pick(g, 0, 30), pp = pick(g, 0, 100);
        for (int k = 0; k < 32; k++) {
            const uint32_t ge = pick(g, 1, 100) <= pg, pr = !ge && pick(g, 1, 100) <= pp;
            gen |= ge << k;
            any |= (ge | pr) << k;
            in |= cy << k;
            cy = ge | (pr & cy);
        }
        if (carries_in(gen, any, cin) != in || carry_out(gen, any, cin) != cy) return it + 1;
    }
    return 0;
}

}  // extern "C"
