// Host build of the kernels' arithmetic that needs no table of av1core (is_levels.cuh), with plain restatements
// beside it: the exact rate and quantisation of a coefficient by its definition.  Test infrastructure only.
#include "is_levels.cuh"

#include <random>

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

}  // extern "C"
