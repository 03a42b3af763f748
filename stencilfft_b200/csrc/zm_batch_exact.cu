// zm_batch_exact.cu -- the complex64 Poisson call on tiles that keep the rounding of the
// VEC x M split.
//
// The residual Lap(phi) / h^2 - rhs amplifies phi's rounding, so these calls, with a residual
// or without, keep the operations of the split's stages (zm_tile.cuh) one for one: rows of VEC points, the
// inter-step twiddle w_N^{n1 k2}, columns in the stages of radix_schedule(M, 16) with the
// twiddle w_{Ns R}^{k r} before each later stage, and plain codelet constants.  What changes
// is where they run: the in-place digits, padded slots, one barrier per stage, coalesced
// sweeps and contiguous twiddle rows of zm_axis.cuh, with the split's digits in place of
// those sized by N.  Per element and stage the split multiplies before a stage by a value of
// (previous outputs of the sub-transform, this stage's input digit); here the same value is
// applied to the same element after the previous stage.  N = 64 .. 4096, VEC = 2 .. 16.
// 96 fields of N = 256 .. 2048, P = 2, B = N / 8: 2.31 -> 1.60 ms per call, 1.76 -> 1.30 ms
// without the residual (1.13 ms on the axis tiles, which round differently).
#include "zm_batch.cuh"
#include "zm_batch_axis.cuh"

namespace zm {

// digits of n = (n2 | n1) high to low: VEC, then M in the order of its stages (forward); the
// inverse's column stages take k1 from its top, which makes the last digit the remainder one
template <int LV, int LM, bool INV> struct SplitDigits {
    static constexpr int LN = LV + LM, Q = (LM + 3) / 4, REM = LM % 4 ? LM % 4 : 4, NST = 1 + Q;
    static constexpr int lr(int s) { return s == 0 ? LV : s == (INV ? Q : 1) ? REM : 4; }
    static constexpr int sh(int s) {
        int b = 0;
        for (int q = s + 1; q < NST; q++) b += lr(q);
        return b;
    }
    // bits of the column digits between the row digit and s (forward)
    static constexpr int up(int s) {
        int b = 0;
        for (int q = 1; q < s; q++) b += lr(q);
        return b;
    }
    static constexpr int r0(int s) { return !INV && up(s) > 0 ? 0 : 1; }
    static constexpr int row(int s) { return INV || s == 0 ? sh(s) : up(s) + (s + 1 < NST ? lr(s + 1) : 0); }
    static constexpr int tw(int s) {
        int o = 0;
        for (int q = 0; q < s; q++) o += 1 << (lr(q) + row(q));
        return o;
    }
    template <int s> static __host__ __device__ constexpr int col(int iv) {
        if constexpr (INV || s == 0) {
            return iv & ((1 << sh(s)) - 1);
        } else {   // (previous column digits, the next digit)
            constexpr int nl = lr(s + 1);
            return (((iv >> sh(s)) & ((1 << up(s)) - 1)) << nl) | ((iv & ((1 << sh(s)) - 1)) >> (sh(s) - nl));
        }
    }
};

struct AxisExactMap : AxisGlobalMap {
    static constexpr int COMP64 = 0;   // plain codelet constants, as the split's stages
};

// frequency bits k of an element -> its index before the inverse's first stage
template <typename DI> __host__ __device__ constexpr int inverse_index(int k) {
    int i = 0, o = 0;
    for (int s = 0; s < DI::NST; s++) {
        i |= ((k >> o) & ((1 << DI::lr(s)) - 1)) << DI::sh(s);
        o += DI::lr(s);
    }
    return i;
}

// One tile of N = 2^(LV + LM) points per line.  The y step's last forward stage multiplies by
// the Poisson factor; where the inverse starts on other digits (REM < 4, two column stages or
// more) the tile is handed over through shared memory, else in registers.
template <int LV, int LM>
__device__ __noinline__ void exact_tile(int op, cpx<float> *S, const cpx<float> *in, cpx<float> *out,
                                        const BatchField &f, int64_t l0, float scale, double a) {
    constexpr int LN = LV + LM, LTL = kBatchTileLog - LN, LP = kBatchPtsLog;
    using DF = SplitDigits<LV, LM, false>;
    using DI = SplitDigits<LV, LM, true>;
    using AF = AxisPass<float, LN, LTL, LP, 4, false, AxisExactMap, DF>;
    using AI = AxisPass<float, LN, LTL, LP, 4, true, AxisExactMap, DI>;
    using C = cpx<float>;
    const Geom &g = f.g;
    const int tid = threadIdx.x;
    const tw<float> *twf = reinterpret_cast<const tw<float> *>(f.exf), *twi = reinterpret_cast<const tw<float> *>(f.exi);
    const int which = op == BOP_X_FWD ? 0 : op == BOP_X_INV ? 2 : 1;
    AxisExactMap m;
    m.m = f.ex + which;
    const LineAddr la = line_addr(g, op == BOP_Y_POISSON ? PASS_Y2 : PASS_X2, l0, __ldg(&m.m->lg));
    if (op == BOP_X_FWD) {
        AF::run(S, in + la.a_base, out + la.f_base, m, twf, tid, false, 1.f, 0.f);
        return;
    }
    if (op == BOP_X_INV) {
        AI::run(S, in + la.f_base, out + la.a_base, m, twi, tid, true, scale, 0.f);
        return;
    }
    AF::load_vec(S, in + la.a_base, m, tid);
    AF::template inner_stages<0>(S, twf, tid);
    __syncthreads();
    constexpr int lr = DF::lr(DF::NST - 1), R = 1 << lr, HI = 1 << (LP - lr), N = 1 << LN;
    constexpr bool SAME = DF::Q == 1 || DF::REM == 4;
    const float a2 = (float)(a * a);
    C x[HI][R];
#pragma unroll
    for (int h = 0; h < HI; h++) {
        const int U = tid + h * AF::NT, t = U & ((1 << LTL) - 1), iu = U >> LTL;
        const C *s = S + axis_slot((iu << (lr + LTL)) | t);
#pragma unroll
        for (int r = 0; r < R; r++) x[h][r] = s[axis_slot(r << LTL)];
        dft<R, -1, float>(x[h]);
        const int64_t l = l0 + t, cid = l >> g.logL, p = l & (g.L - 1);
        const int kx = (int)d_ct(cid * g.L + d_lp(p, g), g), sx = kx >= N / 2 ? kx - N : kx, sx2 = sx * sx;
        int k0 = 0, o = 0;
#pragma unroll
        for (int q = 0; q + 1 < DF::NST; q++) {
            k0 |= ((iu >> (DF::sh(q) - lr)) & ((1 << DF::lr(q)) - 1)) << o;
            o += DF::lr(q);
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = k0 + (r << (LN - lr)), sy = r >= R / 2 ? k - N : k, ksq = sx2 + sy * sy;
            const float fac = ksq == 0 ? 0.f : -__frcp_rn(a2 * (float)ksq);
            x[h][r] = {x[h][r].x * fac, x[h][r].y * fac};
        }
        if constexpr (SAME) dft<R, 1, float>(x[h]);
    }
    if constexpr (!SAME) __syncthreads();
#pragma unroll
    for (int h = 0; h < HI; h++) {
        const int U = tid + h * AF::NT, t = U & ((1 << LTL) - 1), iu = U >> LTL;
        if constexpr (SAME) {
            C *s = S + axis_slot((iu << (lr + LTL)) | t);
#pragma unroll
            for (int r = 0; r < R; r++) s[axis_slot(r << LTL)] = x[h][r];
        } else {
            int k0 = 0, o = 0;
#pragma unroll
            for (int q = 0; q + 1 < DF::NST; q++) {
                k0 |= ((iu >> (DF::sh(q) - lr)) & ((1 << DF::lr(q)) - 1)) << o;
                o += DF::lr(q);
            }
            C *s = S + axis_slot((inverse_index<DI>(k0) << LTL) | t);
#pragma unroll
            for (int r = 0; r < R; r++) s[axis_slot(inverse_index<DI>(r << (LN - lr)) << LTL)] = x[h][r];
        }
    }
    __syncthreads();
    if constexpr (!SAME) {   // the inverse's first stage, on the remainder digit
        constexpr int li = DI::lr(DI::NST - 1), RI = 1 << li;
#pragma unroll
        for (int h = 0; h < 1 << (LP - li); h++) {
            const int U = tid + h * AI::NT, t = U & ((1 << LTL) - 1), iu = U >> LTL;
            C *s = S + axis_slot((iu << (li + LTL)) | t);
            C y[RI];
#pragma unroll
            for (int r = 0; r < RI; r++) y[r] = s[axis_slot(r << LTL)];
            dft<RI, 1, float>(y);
#pragma unroll
            for (int r = 0; r < RI; r++) s[axis_slot(r << LTL)] = y[r];
        }
        __syncthreads();
    }
    AI::template inner_stages<AI::NST - 2>(S, twi, tid);
    AI::store_vec(S, out + la.a_base, m, tid, false, 1.f, 0.f);
}

__global__ void __launch_bounds__(kBatchThreads, 4) batch_exact_kernel(const BatchParams bp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<float> *s = reinterpret_cast<cpx<float> *>(smem_raw);
    __shared__ int s_ok;
    constexpr int TP = 1 << kBatchTileLog;
    for (int st = 0; st < bp.nsteps; st++) {
        if (st > 0 && !grid_barrier(bp.bar, gridDim.x + bp.missing, bp.abort, bp.err, &s_ok)) return;
        const int op = bp.step[st].op;
        if (op == BOP_NOP) continue;
        const BatchStep &S = bp.step[st];
        const int ntiles = (int)bp.tiles, hop = walks_back(bp, st) ? -(int)gridDim.x : (int)gridDim.x;
        int tile = hop < 0 ? ntiles - 1 - (int)blockIdx.x : (int)blockIdx.x;
        int fi = tile < ntiles ? __ldg(bp.tile_field + tile) : 0;
        for (; (unsigned)tile < (unsigned)ntiles; tile += hop) {
            const BatchField &f = bp.fields[fi];
            if ((unsigned)(tile + hop) < (unsigned)ntiles) fi = __ldg(bp.tile_field + tile + hop);
            const Geom &g = f.g;
            const int64_t sub = tile - f.tile0;   // of the field
            const cpx<float> *in = reinterpret_cast<const cpx<float> *>(S.in) + f.off;
            cpx<float> *out = reinterpret_cast<cpx<float> *>(S.out) + f.off;
            if (op == BOP_RESIDUAL) {
                residual_tile<float, TP>(g, S.a, in, reinterpret_cast<const cpx<float> *>(S.aux) + f.off, out,
                                         sub * TP, s, threadIdx.x);
                continue;
            }
            const float sc = (float)(1.0 / ((double)g.n * (double)g.n));
            __syncthreads();   // the previous tile is done with the shared memory
#define ZM_EX(LN, LV)                                                                                        \
    case LN << 4 | LV:                                                                                       \
        exact_tile<LV, LN - LV>(op, s, in, out, f, sub << (kBatchTileLog - LN), sc, S.a);                    \
        break;
#define ZM_EXN(LN) ZM_EX(LN, 1) ZM_EX(LN, 2) ZM_EX(LN, 3) ZM_EX(LN, 4)
            switch (g.logN << 4 | g.logVEC) {
                ZM_EXN(6) ZM_EXN(7) ZM_EXN(8) ZM_EXN(9) ZM_EXN(10) ZM_EXN(11) ZM_EXN(12)
            default: break;
            }
#undef ZM_EXN
#undef ZM_EX
        }
    }
}

BatchFn batch_exact_fn() { return batch_exact_kernel; }

bool batch_exact_fits(const Geom &g) { return g.logVEC >= 1 && g.logVEC <= 4 && g.logN >= 6 && g.logN <= 12; }

std::vector<int> batch_exact_digits(const Geom &g, bool inverse) {
    const int q = (g.logM + 3) / 4, rem = g.logM % 4 ? g.logM % 4 : 4;
    std::vector<int> lrs{g.logVEC};
    for (int s = 1; s <= q; s++) lrs.push_back(s == (inverse ? q : 1) ? rem : 4);
    return lrs;
}

void batch_exact_twiddles(const Geom &g, bool inverse, std::vector<int64_t> *exps) {
    const std::vector<int> lrs = batch_exact_digits(g, inverse);
    if (inverse) {   // before stage s: w^{k_s v}, v the outputs so far
        axis_twiddles(g, lrs, exps);
        return;
    }
    const int ln = g.logN;
    for (int64_t k = 0; k < g.vec; k++)
        for (int64_t v = 0; v < g.m; v++) exps->push_back(k * v);
    int up = 0;   // bits of the column digits before s
    for (size_t s = 1; s + 1 < lrs.size(); up += lrs[s], s++)
        for (int64_t r = 0; r < 1 << lrs[s]; r++)
            for (int64_t c = 0; c < 1 << (up + lrs[s + 1]); c++) {
                const int64_t nn = c & ((1 << lrs[s + 1]) - 1);
                int64_t upper = c >> lrs[s + 1], kk = r << up;   // outputs so far: low digits first
                int o = up;
                for (size_t q = s; q-- > 1;) {                   // the last digit lies lowest in `upper`
                    o -= lrs[q];
                    kk |= (upper & ((1 << lrs[q]) - 1)) << o;
                    upper >>= lrs[q];
                }
                exps->push_back((kk * nn) << (ln - (up + lrs[s] + lrs[s + 1])));
            }
}

}  // namespace zm
