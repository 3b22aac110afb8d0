// is_k_test.cu - the kernels of is_test_eval_mixed, in a unit of their own: a program that does not call it never loads them.
#include "is_units.cuh"
#include "is_small.cuh"
#include "is_tiny.cuh"

namespace is {

// the evaluations of the small tx sizes as the search runs them, every block with a tx type of its own.  FORM 0: the closed
// loop's, two lanes a block, 16 blocks a warp (small_eval); FORM 1: the analysis', one thread a block (thr_eval for the 4- and
// 8-point sizes, mid_eval for the others).  One warp a CTA; blocks past the last repeat it.
template <typename Px> struct MixedScr {
    RateStage T;
    SmallTabs tabs;
    uint16_t pos[3 * 64];   // the analysis' table of the size: rows of 64 (mid_eval) or 32 entries (thr_eval)
    Px src[16 * 64], pred[16 * 64];
    int32_t buf[16 * 67];
    uint32_t rows[16 * small_words<2, 4>()];
    int16_t q[32][66];
};
template <int BD, int FORM>
__global__ void __launch_bounds__(32) k_test_eval_mixed(int n, const uint16_t *src, const uint16_t *pred, int txSz, const uint8_t *types, int plane,
                                                        int dcQ, int acQ, int qctx, int skipCtx, int dcCtx, int intraDir, int16_t *lv, long long *D,
                                                        long long *R, int32_t *eob) {
    typedef typename std::conditional<BD == 8, uint8_t, uint16_t>::type Px;
    extern __shared__ __align__(16) unsigned char tsm[];
    MixedScr<Px> &S = *reinterpret_cast<MixedScr<Px> *>(tsm);
    const int lane = threadIdx.x, nc = txw(txSz) * txh(txSz);
    const RateTabs T = rate_tabs_stage(S.T, qctx, lane, 32);
    __syncthreads();
    small_tabs_stage(S.tabs, T, lane, 32);
    for (int k = lane; k < 3 * nc; k += 32) pos_entry(S.pos + k / nc * (nc == 64 ? 64 : 32), T, txSz, k / nc, k % nc);
    __syncthreads();
    if constexpr (FORM == 0) {
        const int b0 = blockIdx.x * 16, k = lane >> 1, b = min(b0 + k, n - 1);
        for (int i = lane; i < 16 * nc; i += 32) {
            const size_t at = (size_t)min(b0 + i / nc, n - 1) * nc + i % nc;
            S.src[i] = (Px)src[at];
            S.pred[i] = (Px)pred[at];
        }
        __syncwarp();
        int16_t *q = &S.q[0][0];
        const EvalOut o = small_eval_size<BD, Px>(txSz, S.src + k * nc, S.pred + k * nc, types[b], plane, skipCtx, dcCtx, intraDir, dcQ, acQ,
                                                  quant_recip(dcQ), quant_recip(acQ), S.T.cost, &S.tabs, S.buf, S.rows, q, k, lane & 1);
        __syncwarp();
        if (b0 + k < n) {
            for (int i = lane & 1; i < nc; i += 2) lv[(size_t)b * nc + i] = q[k * nc + i];
            if (!(lane & 1)) { D[b] = o.D; R[b] = o.R; eob[b] = o.eob; }
        }
    } else {
        const int at = blockIdx.x * 32 + lane, b = min(at, n - 1);
        const EvalIn e{types[b], plane, skipCtx, dcCtx, intraDir, dcQ, acQ, quant_recip(dcQ), quant_recip(acQ), T};
        const uint16_t *s = src + (size_t)b * nc, *p = pred + (size_t)b * nc;
        int res[64];
        EvalOut o;
#pragma unroll
        for (int i = 0; i < 64; i++) res[i] = i < nc ? (int)s[i] - (int)p[i] : 0;
        int16_t *qs = S.q[lane];
        const uint16_t *tab = S.pos;
        if (txSz == AV1G_TX_8X8) o = mid_eval<BD, 3, 3>(txSz, res, e, tab, qs);
        else if (txSz == AV1G_TX_4X16) o = mid_eval<BD, 2, 4>(txSz, res, e, tab, qs);
        else if (txSz == AV1G_TX_16X4) o = mid_eval<BD, 4, 2>(txSz, res, e, tab, qs);
        else if (txSz == AV1G_TX_4X4) o = thr_eval<BD, 2, 2>(txSz, res, e, tab);
        else if (txSz == AV1G_TX_4X8) o = thr_eval<BD, 2, 3>(txSz, res, e, tab);
        else o = thr_eval<BD, 3, 2>(txSz, res, e, tab);
        if (at < n) {
            if (txSz == AV1G_TX_8X8 || txSz == AV1G_TX_4X16 || txSz == AV1G_TX_16X4)   // (the others keep their levels in registers)
                for (int i = 0; i < nc; i++) lv[(size_t)b * nc + i] = qs[i];
            D[b] = o.D; R[b] = o.R; eob[b] = o.eob;
        }
    }
}

cudaError_t test_upload(const TableBlob &B) { return upload_common(B); }

cudaError_t test_eval_mixed(int form, int bitDepth, int n, const uint16_t *src, const uint16_t *pred, int txSz, const uint8_t *types, int plane,
                            int dcQ, int acQ, int qctx, int skipCtx, int dcCtx, int intraDir, int16_t *lv, long long *D, long long *R,
                            int32_t *eob) {
    const bool g10 = bitDepth == 10;
    const int per = form ? 32 : 16, smem = g10 ? (int)sizeof(MixedScr<uint16_t>) : (int)sizeof(MixedScr<uint8_t>);
    auto *k = g10 ? (form ? k_test_eval_mixed<10, 1> : k_test_eval_mixed<10, 0>) : (form ? k_test_eval_mixed<8, 1> : k_test_eval_mixed<8, 0>);
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    k<<<(n + per - 1) / per, 32, smem>>>(n, src, pred, txSz, types, plane, dcQ, acQ, qctx, skipCtx, dcCtx, intraDir, lv, D, R, eob);
    return cudaGetLastError();
}

}  // namespace is
