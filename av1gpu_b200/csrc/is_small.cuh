// is_small.cuh - the closed loop's evaluation of small tx blocks (4x4, 8x8, 4x8, 8x4, 4x16, 16x4: nine leaves in ten).
//
// The same integers as grp_eval_x (forward transform, quantisation, distortion, exact rate), with the size known at
// compile time and two lanes a task, so that a warp evaluates up to 16 (candidate, tx type) tasks at once.  What bounds it
// is the latency of one warp per SM sub-partition, part of it instruction fetch: a leaf runs through its code about once
// (a 1920x1080 search, 36,774 leaves: 1,100 instruction lookups in the L1.5 cache a leaf, of which 300 miss, with the polls of
// idle warps).  So:
//   - a lane transforms its half of the columns one after the other, then its half of the rows with the quantisation of a
//     row right after it: one copy of each network in the code (13 .. 33 KB a size).  Everything unrolled in registers, 70 KB
//     for 8x8, made the closed loop of a 4000x3000 picture 108 ms, this form 99 ms, grp_eval_x (run-time sizes, the networks
//     called out of line) 124 ms;
//   - quantisation divides by a multiplication with the step's reciprocal and one correction, and has no branches: the
//     coefficients of a row are independent chains;
//   - the levels of a row lie in one word, 4 bits each (capped at 15, and at 3 for the base contexts), so the context
//     sums of a whole row are a few shifts and additions of words instead of five bounds-checked loads a coefficient;
//   - the scan position and the position's context offset come from one table load a coefficient.
// quant_level, row_bits (is_levels.cuh) and pos_entry are also the analysis' (k_analysis_tiny, one thread a block).
#pragma once
#include "is_dev.cuh"
#include "is_levels.cuh"

namespace is {

static_assert(TXC_2D == AV1G_TX_CLASS_2D && TXC_HORIZ == AV1G_TX_CLASS_HORIZ && EOB_STRIDE == IS_CD(coeff_base_eob, 3) &&
              BASE_STRIDE == IS_CD(coeff_base, 3) && BR_STRIDE == IS_CD(coeff_br, 3), "is_levels.cuh");

constexpr int SMALL_SIZES = 6;
// Transform_Row_Shift of these sizes (the library checks it against av1core's table at upload)
__host__ __device__ constexpr int small_row_shift(int lw, int lh) { return lw + lh >= 6 ? 1 : 0; }
// sizes in the order 4x4, 8x8, 4x8, 8x4, 4x16, 16x4
__device__ __forceinline__ int small_size(int i) {
    return i == 0 ? AV1G_TX_4X4 : i == 1 ? AV1G_TX_8X8 : i == 2 ? AV1G_TX_4X8 : i == 3 ? AV1G_TX_8X4 : i == 4 ? AV1G_TX_4X16 : AV1G_TX_16X4;
}
struct __align__(16) SmallTabs {
    uint16_t pos[SMALL_SIZES][3][64];   // per (size, class, natural position): scan position | context offset << 8
    uint8_t typeIdx[16];                // index of a tx type in TX_SET_INTRA_1
};
// entry of scan position c of (size, class): its natural position's scan position | context offset << 8
__device__ __forceinline__ void pos_entry(uint16_t *tab, const RateTabs &T, int txSz, int cls, int c) {
    const int p = T.scan[c_scanOff[txSz][cls] + c], row = p >> ST(Tx_Width_Log2)[txSz], col = p & (txw(txSz) - 1);
    const int off = cls == AV1G_TX_CLASS_2D ? T.baseCtx[txSz * 25 + min(row, 4) * 5 + min(col, 4)]
                                            : ST(Coeff_Base_Pos_Ctx_Offset)[min(cls == AV1G_TX_CLASS_VERT ? row : col, 2)];
    tab[p] = (uint16_t)(c | off << 8);
}
// all threads of the CTA, after the scans are staged (and a barrier); followed by a barrier
__device__ __forceinline__ void small_tabs_stage(SmallTabs &S, const RateTabs &T, int tid, int nt) {
    for (int k = tid; k < SMALL_SIZES * 3 * 64; k += nt) {
        const int si = k / 192, cls = (k / 64) % 3, c = k % 64, txSz = small_size(si);
        if (c >= txw(txSz) * txh(txSz)) continue;
        pos_entry(S.pos[si][cls], T, txSz, cls, c);
    }
    for (int t = tid; t < 16; t += nt) S.typeIdx[t] = (uint8_t)tx_index_in_set(AV1G_TX_SET_INTRA_1, t);
}

// words of the packed rows of one task: H rows and 4 rows of zeros below, capped at 3, then capped at 15; an odd stride
// keeps the tasks of a warp on different banks
template <int LW, int LH> constexpr int small_words() { return 2 * ((1 << LH) + 4) * (LW == 4 ? 2 : 1) + 1; }

// One evaluation by lanes g = 0, 1 of a pair (all lanes of the warp call it together): src and pred are W x H in shared
// memory, rows are small_words() words of scratch and q the W x H levels of the task.  dcM / acM: floor(2^32 / (64 step)).
template <int BD, int LW, int LH, typename Px>
__device__ __forceinline__ EvalOut small_eval(int si, const Px *src, const Px *pred, int txType, int plane, int skipCtx, int dcCtx, int intraDir,
                                              int dcQ, int acQ, uint32_t dcM, uint32_t acM, const uint16_t *C, const SmallTabs &S,
                                              int32_t *buf, uint32_t *rows, int16_t *q, int g) {
    constexpr int W = 1 << LW, H = 1 << LH, CW = W / 2, RH = H / 2;
    typedef PackedRow<LW> Row;
    const int txSz = LW == LH ? (LW == 2 ? AV1G_TX_4X4 : AV1G_TX_8X8) : LW == 2 ? (LH == 3 ? AV1G_TX_4X8 : AV1G_TX_4X16)
                   : LW == 3 ? AV1G_TX_8X4 : AV1G_TX_16X4;
    constexpr int rowShift = small_row_shift(LW, LH);
    constexpr int rect = (LW - LH == 1 || LH - LW == 1) ? 1 : 0;
    constexpr int E = rowShift + 4 + FB - (LW + LH - 2);
    constexpr int s0 = 17 - BD - LH > 0 ? 17 - BD - LH : 0;
    constexpr int s2 = s0 - LW - E;
    constexpr int dsh = 16 - 2 * FB - (2 * (rowShift + 4) - (LW + LH - 2) + rect);
    const int ck = col_kind(txType), rk = row_kind(txType);
    const int cls = txType == AV1G_IDTX ? AV1G_TX_CLASS_2D : tx_class(txType);
    // ---- columns g CW .. g CW + CW - 1, one after the other (one copy of the networks) ----
#pragma unroll 1
    for (int j = g * CW; j < (g + 1) * CW; j++) {
        int t[H];
#pragma unroll
        for (int i = 0; i < H; i++) t[i] = ((int)src[i * W + j] - (int)pred[i * W + j]) * (1 << s0);
        fwd1d<H>(ck, t);
#pragma unroll
        for (int i = 0; i < H; i++) buf[i * W + j] = (t[i] + (1 << (LW - 1))) >> LW;
    }
    __syncwarp();
    // ---- quantisation (the tx sizes' dequantisation denominator is 1), levels, packed rows ----
    const uint16_t *tab = S.pos[si][cls];
    Row *r3 = reinterpret_cast<Row *>(rows), *r15 = r3 + (H + 4);
    i64 dist = 0;
    int eob = 0;
#pragma unroll 1
    for (int rr = g * RH; rr < (g + 1) * RH; rr++) {
        Row p3 = 0, p15 = 0;
        uint32_t lv[CW];
        int row[W];
#pragma unroll
        for (int j = 0; j < W; j++) row[j] = buf[rr * W + j];
        fwd1d<W>(rk, row);
#pragma unroll
        for (int j = 0; j < W; j++) {
            int v = row[j];
            if (rect) v = (v * 5793 + 2048) >> 12;
            if constexpr (s2 > 0) v = (v + (1 << (s2 - 1))) >> s2;
            else v = v * (1 << -s2);
            const bool dc = j == 0 && rr == 0;
            const int qv = quant_level<BD>(v, dc ? dcQ : acQ, dc ? dcM : acM, dist), l = abs(qv);
            eob = max(eob, l ? (int)(tab[rr * W + j] & 0xFF) + 1 : 0);
            p3 |= (Row)min(l, 3) << (4 * j);
            p15 |= (Row)min(l, 15) << (4 * j);
            if (j & 1) lv[j >> 1] |= (uint32_t)qv << 16; else lv[j >> 1] = (uint32_t)qv & 0xFFFFu;
        }
#pragma unroll
        for (int j = 0; j < CW; j++) reinterpret_cast<uint32_t *>(q)[rr * CW + j] = lv[j];
        if constexpr (LW == 4) {   // (the scratch is 4-byte aligned)
            uint32_t *a = rows + 2 * rr, *b = rows + 2 * (H + 4 + rr);
            a[0] = (uint32_t)p3; a[1] = (uint32_t)(p3 >> 32);
            b[0] = (uint32_t)p15; b[1] = (uint32_t)(p15 >> 32);
        } else {
            r3[rr] = p3;
            r15[rr] = p15;
        }
    }
    constexpr int RW = LW == 4 ? 2 : 1;
#pragma unroll
    for (int k = 0; k < 4 * RW; k++) rows[(g * (H + 4) + H) * RW + k] = 0;   // the rows below: lane 0's of one kind, lane 1's of the other
    eob = max(eob, __shfl_xor_sync(0xffffffffu, eob, 1));
    __syncwarp();
    // ---- rate ----
    const int ptype = plane > 0;
    const int txSzCtx = (ST(Tx_Size_Sqr)[txSz] + ST(Tx_Size_Sqr_Up)[txSz] + 1) >> 1;
    const uint16_t *cBase = C + ci_base(txSzCtx, ptype, 0), *cBr = C + ci_br(txSzCtx, ptype, 0), *cEob = C + ci_base_eob(txSzCtx, ptype, 0);
    auto get = [&](int k) -> Row {
        if constexpr (LW == 4) return (Row)rows[2 * k] | (Row)rows[2 * k + 1] << 32;
        else return rows[k];
    };
    int b = 0;
    if (eob) {
#pragma unroll 1
        for (int i = 0; i < RH; i++) {
            const int rr = g * RH + i;
            const Row a0 = get(rr), a1 = get(rr + 1), a2 = get(rr + 2), b0 = get(H + 4 + rr), b1 = get(H + 4 + rr + 1);
            b += row_bits<LW, LH>(rr, a0, a1, a2, cls == AV1G_TX_CLASS_VERT ? get(rr + 3) : 0, cls == AV1G_TX_CLASS_VERT ? get(rr + 4) : 0, b0, b1,
                                  cls == AV1G_TX_CLASS_VERT ? get(H + 4 + rr + 2) : 0, cls, eob, tab + rr * W, cBase, cEob, cBr,
                                  [&](int j) -> int { return q[rr * W + j]; });
        }
        if (g == 0 && q[0]) b += C[ci_dc_sign(ptype, dcCtx) + (q[0] < 0)] - 256;   // the DC sign has its own contexts
    }
    __syncwarp();
    // txb_skip, tx type (TX_SET_INTRA_1 for every one of these sizes), eob position
    int bb;
    if (eob == 0) {
        bb = C[ci_txb_skip(txSzCtx, skipCtx) + 1];
    } else {
        bb = C[ci_txb_skip(txSzCtx, skipCtx)];
        if (plane == 0) bb += C[ci_set1(ST(Tx_Size_Sqr)[txSz], intraDir) + S.typeIdx[txType]];
        const int pt = eob <= 2 ? eob : 2 + (31 - __clz(eob - 1));
        bb += C[ci_eob_pt(LW + LH - 4, ptype, tx_class(txType) == AV1G_TX_CLASS_2D ? 0 : 1) + pt - 1];
        if (pt >= 3) {
            const int rem = eob - ((1 << (pt - 2)) + 1);
            bb += C[ci_eob_extra(txSzCtx, ptype, pt - 3) + ((rem >> (pt - 3)) & 1)] + (pt - 3) * 256;
        }
    }
    EvalOut o;
    o.R = b + __shfl_xor_sync(0xffffffffu, b, 1) + bb;
    o.D = (dist + __shfl_xor_sync(0xffffffffu, dist, 1)) << dsh;
    o.eob = eob;
    return o;
}

// one copy per size, called with scalars
template <int BD, int LW, int LH, typename Px>
__device__ __noinline__ EvalOut small_eval_x(int si, const Px *src, const Px *pred, int txType, int plane, int skipCtx, int dcCtx, int intraDir,
                                             int dcQ, int acQ, uint32_t dcM, uint32_t acM, const uint16_t *C, const SmallTabs *S,
                                             int32_t *buf, uint32_t *rows, int16_t *q, int g) {
    IS_SHARED_PTR(buf);
    IS_SHARED_PTR(src); IS_SHARED_PTR(pred); IS_SHARED_PTR(C); IS_SHARED_PTR(S); IS_SHARED_PTR(rows); IS_SHARED_PTR(q);
    return small_eval<BD, LW, LH, Px>(si, src, pred, txType, plane, skipCtx, dcCtx, intraDir, dcQ, acQ, dcM, acM, C, *S, buf, rows, q, g);
}
// task slices of a round: the block at buf (an odd stride: the tasks of a warp on different banks), packed rows, levels
template <int BD, typename Px>
__device__ __forceinline__ EvalOut small_eval_size(int txSz, const Px *src, const Px *pred, int txType, int plane, int skipCtx, int dcCtx,
                                                   int intraDir, int dcQ, int acQ, uint32_t dcM, uint32_t acM, const uint16_t *C,
                                                   const SmallTabs *S, int32_t *buf, uint32_t *rows, int16_t *q, int task, int g) {
#define IS_SMALL(si, LW, LH) small_eval_x<BD, LW, LH, Px>(si, src, pred, txType, plane, skipCtx, dcCtx, intraDir, dcQ, acQ, dcM, acM, C, S, \
                                                          buf + task * ((1 << (LW + LH)) + 3), rows + task * small_words<LW, LH>(), q + (task << (LW + LH)), g)
    switch (txSz) {
    case AV1G_TX_4X4: return IS_SMALL(0, 2, 2);
    case AV1G_TX_8X8: return IS_SMALL(1, 3, 3);
    case AV1G_TX_4X8: return IS_SMALL(2, 2, 3);
    case AV1G_TX_8X4: return IS_SMALL(3, 3, 2);
    case AV1G_TX_4X16: return IS_SMALL(4, 2, 4);
    default: return IS_SMALL(5, 4, 2);
    }
#undef IS_SMALL
}

}  // namespace is
