// zm_batch_axis.cuh -- tiles of a batch on the axis pass sized by N alone (zm_axis.cuh).
//
// A tile is 4096 points: TL = 4096 / N lines of one field, 256 threads of 16 points, so one
// CTA shape serves every N from 64 to 4096 and every (P, B); the field's layout is its two
// weight tables in global memory.  The fused Poisson y step (complex128; complex64 calls run
// the tiles of zm_batch_exact.cu) keeps the spectrum of a tile in registers: the last
// digit's forward DFT, the division and the same digit's inverse DFT are one stage, so it
// costs five barriers and four shared-memory round trips instead of the two transforms'
// eight and seven.
#pragma once

#include "zm_axis.cuh"

namespace zm {

constexpr int kBatchTileLog = 12;   // log2 points per tile
constexpr int kBatchPtsLog = 4;     // log2 points per thread

// digits of index i above the last one -> the low bits of the frequency they stand for
template <int LN, int LE> ZM_DEV int axis_low_freq(int iu) {
    constexpr int NST = axis_stages(LN, LE), lrl = axis_lr(LN, LE, NST - 1);
    int k = 0, o = 0;
#pragma unroll
    for (int s = 0; s + 1 < NST; s++) {
        const int lr = axis_lr(LN, LE, s);
        k |= ((iu >> (axis_sh(LN, LE, s) - lrl)) & ((1 << lr) - 1)) << o;
        o += lr;
    }
    return k;
}

// The last digit of a y tile: forward DFT, times -1 / (a^2 |k|^2) (k = 0 -> 0), inverse DFT.
// Line l0 + t holds the x frequency ct(cid L + lp(p)) of its row p of rank column cid
// (reciprocal_to_global, utils.h:265-268).
template <int LN, int LTL, int LP, int LE>
ZM_DEV void poisson_stage(cpx<double> *S, const Geom &g, int64_t l0, double a, int tid) {
    using T = double;
    using A = AxisPass<T, LN, LTL, LP, LE, false>;
    constexpr int NST = A::NST, lr = axis_lr(LN, LE, NST - 1), R = 1 << lr, N = 1 << LN;
    const T a2 = (T)(a * a);
#pragma unroll
    for (int h = 0; h < 1 << (LP - lr); h++) {
        const int U = tid + h * A::NT, t = U & ((1 << LTL) - 1), iu = U >> LTL;
        const int64_t l = l0 + t, cid = l >> g.logL, p = l & (g.L - 1);
        const int kx = (int)d_ct(cid * g.L + d_lp(p, g), g), sx = kx >= N / 2 ? kx - N : kx;
        const int k0 = axis_low_freq<LN, LE>(iu), sx2 = sx * sx;
        cpx<T> *s = S + axis_slot((iu << (lr + LTL)) | t);
        cpx<T> x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = s[axis_slot(r << LTL)];
        dft<R, -1, T, A::COMP>(x);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = k0 + (r << (LN - lr)), sy = r >= R / 2 ? k - N : k;
            const int ksq = sx2 + sy * sy;
            const T f = ksq == 0 ? 0.0 : -1.0 / (a2 * (double)ksq);
            x[r] = {x[r].x * f, x[r].y * f};
        }
        dft<R, 1, T, A::COMP>(x);
#pragma unroll
        for (int r = 0; r < R; r++) s[axis_slot(r << LTL)] = x[r];
    }
}

enum AxisTileOp : int { ATILE_FWD = 0, ATILE_INV = 1, ATILE_POISSON = 2 };

// One tile of N = 2^LN points per line, lines l0 .. of a field; a function of its own per N
// (the persistent kernel would otherwise hold the registers of all of them).
template <typename T, int LN>
__device__ __noinline__ void batch_axis_tile(int op, cpx<T> *S, const cpx<T> *in, cpx<T> *out, const Geom &g,
                                             const AxisMap *map, const void *tw_, bool xpass, int64_t l0, T scale,
                                             double a) {
    constexpr int LTL = kBatchTileLog - LN, LP = kBatchPtsLog, LE = 4;
    using AF = AxisPass<T, LN, LTL, LP, LE, false, AxisGlobalMap>;
    using AI = AxisPass<T, LN, LTL, LP, LE, true, AxisGlobalMap>;
    const AxisGlobalMap m{map};
    const zm::tw<T> *tb = reinterpret_cast<const zm::tw<T> *>(tw_);
    const int tid = threadIdx.x;
    const LineAddr la = line_addr(g, xpass ? PASS_X2 : PASS_Y2, l0, __ldg(&map->lg));
    if (op == ATILE_FWD) {
        AF::run(S, in + la.a_base, out + la.f_base, m, tb, tid, false, T(1), T(0));
    } else if (op == ATILE_INV) {
        AI::run(S, in + la.f_base, out + la.a_base, m, tb, tid, scale != T(1), scale, T(0));
    } else if constexpr (sizeof(T) == 8) {
        AF::load_vec(S, in + la.a_base, m, tid);
        AF::template inner_stages<0>(S, tb, tid);
        __syncthreads();
        poisson_stage<LN, LTL, LP, LE>(S, g, l0, a, tid);
        __syncthreads();
        AI::template inner_stages<AI::NST - 2>(S, tb, tid);
        AI::store_vec(S, out + la.a_base, m, tid, false, T(1), T(0));
    }
}

}  // namespace zm
