// zm_axis.cuh -- the axis pass of any layout, sized by N alone.
//
// Same computation as line_fft_kernel (zm_fft.cu): one pass transforms the N-point lines of
// one axis and moves them from the layout of one stage of the reference's pipeline to the
// next.  A DFT does not depend on how the layout splits N = VEC * M, only its addresses do,
// and every address here is a sum of one weight per bit: vector side element n of line l
// sits at A(l) + sum of A_b over the set bits b of n, frequency k at F(l) + sum of F_b over
// those of k (block-cyclic deal, vector packing, row interleave and rank chunks are all bit
// permutations, N, B and P being powers of two).  So the transform is compiled per N and the
// layout arrives as two short tables of weights (AxisMap, built once per plan): every
// (P, B), every axis of 2D and 3D fields and both directions run the same code.
//
// A tile of TL = 2^LTL lines x N points lives in shared memory at index I = i TL + t.  The
// N-point transform is digits of at most 2^LE points, high to low, in place (forward:
// decimation in frequency): stage s transforms digit s of i, multiplies by w^{k_s v} (v the
// lower digits; table rows contiguous in v) and writes the same slots back, so one barrier
// separates two stages.  Afterwards i holds the digits of k in reversed order.  The
// inverse runs the transposed algorithm (stages in reverse, conjugate twiddles before the
// DFT) on the same slots.
//   * the lines are the lowest bits of I: neighbouring lanes share v, so a twiddle row is
//     read as a broadcast;
//   * slot(I) = I + I/16 + I/256 + I/4096: bit b of I weighs 2^(b mod 4) modulo the 16
//     eight-byte banks, so lanes on any four index bits that differ modulo 4 are free of
//     conflicts, and a register's slot is the unit's plus a constant;
//   * the frequency side moves between registers and global memory, the threads of the
//     stage next to it numbered in the order of the frequency-side addresses;
//   * the vector side goes through the tile in the order of its own addresses (16-byte
//     accesses), because the registers of the stage next to it hold its contiguous axis.
#pragma once

#include "zm_common.cuh"
#include "zm_internal.h"
#include "zm_lines.cuh"

namespace zm {

constexpr int axis_stages(int ln, int le) { return (ln + le - 1) / le; }
// log2 radix of stage s, and the bits of i below its digit
constexpr int axis_lr(int ln, int le, int s) { return s == 0 ? ln - le * (axis_stages(ln, le) - 1) : le; }
constexpr int axis_sh(int ln, int le, int s) { return le * (axis_stages(ln, le) - 1 - s); }
// first entry of stage s in the twiddle table (row k of stage s: 2^sh entries)
constexpr int axis_tw(int ln, int le, int s) {
    int o = 0;
    for (int q = 0; q < s; q++) o += 1 << (axis_lr(ln, le, q) + axis_sh(ln, le, q));
    return o;
}
__host__ __device__ constexpr int axis_slot(int i) { return i + (i >> 4) + (i >> 8) + (i >> 12); }

// LP: log2 points per thread; LE: log2 of the largest digit (LE <= LP)
template <typename T, int LN, int LTL, int LP, int LE> struct AxisCfg {
    static constexpr int NT = 1 << (LN + LTL - LP), LNT = LN + LTL - LP;
    static constexpr int NST = axis_stages(LN, LE);
    static constexpr size_t SMEM = sizeof(cpx<T>) * (size_t)(axis_slot((1 << (LN + LTL)) - 1) + 1);
    // 64 registers for 32 words of points per thread, 128 for 64
    static constexpr int WORDS = (int)sizeof(cpx<T>) / 4 << LP;
    static constexpr int BY_REG = (WORDS <= 32 ? 1024 : 512) / NT;
    static constexpr int BY_SMEM = (int)((size_t)227 * 1024 / (SMEM + 1024));
    static constexpr int MINB0 = BY_REG < BY_SMEM ? BY_REG : BY_SMEM;
    static constexpr int MINB = MINB0 < 1 ? 1 : (MINB0 > 16 ? 16 : MINB0);
};

// sums over the set bits of tid of two weight lists
template <int NB> ZM_DEV void axis_bits(int tid, const int *wa, const int *ws, int &a, int &s) {
    a = 0;
    s = 0;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const int m = (tid >> b) & 1;
        a += m * wa[b];
        s += m * ws[b];
    }
}
// offset of register r: the sum of the weights w[0 ..] over its set bits
template <int NB> ZM_DEV int axis_reg(int r, const int *w) {
    int o = 0;
#pragma unroll
    for (int b = 0; b < NB; b++)
        if (r >> b & 1) o += w[b];
    return o;
}

template <typename T, int LN, int LTL, int LP, int LE, bool INV> struct AxisPass {
    using C = cpx<T>;
    using CF = AxisCfg<T, LN, LTL, LP, LE>;
    static constexpr int NT = CF::NT, LNT = CF::LNT, NST = CF::NST, EPT = 1 << LP;
    static constexpr int DIR = INV ? 1 : -1;
    // codelet constants as hi + lo pairs: the 45 degree ones, and complex64's 32-point level.
    // Round trip against FP64, without and with: 3D N = 256 c64 2.8e-7 / 2.4e-7 (at every
    // constant 2.2e-7), N = 1024 (32-point digits) 2.8e-7 / 2.2e-7, 3D N = 512 3.3e-7 /
    // 2.6e-7; 3D N = 256 c128 5.4e-16 / 4.2e-16; times within 1 % of each other.
    static constexpr int COMP = sizeof(T) == 4 ? 2 : 1;

    // global vector side <-> tile, in address order: thread bits first; complex64 keeps the
    // lowest address bit in the registers (16-byte accesses)
    static ZM_DEV void load_vec(C *S, const C *in, const AxisMap &m, int tid) {
        int a0, s0;
        axis_bits<LNT>(tid, m.va, m.vs, a0, s0);
        C v[EPT];
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int r = 0; r < EPT; r += 2) {
                const float4 q = __ldg(reinterpret_cast<const float4 *>(in + a0 + axis_reg<LP>(r, m.va + LNT)));
                v[r] = {q.x, q.y};
                v[r + 1] = {q.z, q.w};
            }
        } else {
#pragma unroll
            for (int r = 0; r < EPT; r++) v[r] = ldg(in + a0 + axis_reg<LP>(r, m.va + LNT));
        }
#pragma unroll
        for (int r = 0; r < EPT; r++) S[s0 + axis_reg<LP>(r, m.vs + LNT)] = v[r];
    }
    static ZM_DEV void store_vec(const C *S, C *out, const AxisMap &m, int tid, bool scl, T sr, T si) {
        int a0, s0;
        axis_bits<LNT>(tid, m.va, m.vs, a0, s0);
        constexpr int ST = sizeof(T) == 4 ? 2 : 1;
#pragma unroll
        for (int r = 0; r < EPT; r += ST) {
            C v[ST];
#pragma unroll
            for (int q = 0; q < ST; q++) {
                v[q] = S[s0 + axis_reg<LP>(r + q, m.vs + LNT)];
                if (scl) v[q] = {sr * v[q].x - si * v[q].y, sr * v[q].y + si * v[q].x};
            }
            C *o = out + a0 + axis_reg<LP>(r, m.va + LNT);
            if constexpr (ST == 2) *reinterpret_cast<float4 *>(o) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
            else *o = v[0];
        }
    }

    // stage s on the units of this thread; the stage next to the frequency side (the last
    // forward, the first inverse) takes its units in frequency-side order and reads or
    // writes global memory at `gm`
    template <int s> static ZM_DEV void stage(C *S, C *gm, const AxisParams &p, int tid, bool scl, T sr, T si) {
        constexpr int lr = axis_lr(LN, LE, s), sh = axis_sh(LN, LE, s), shp = sh + LTL;
        constexpr int R = 1 << lr, LU = LP - lr;
        constexpr bool EDGE = s == NST - 1;
        if constexpr (EDGE) {
            int fa0, fs0;
            axis_bits<LNT>(tid, p.m.fa, p.m.fs, fa0, fs0);
#pragma unroll
            for (int u = 0; u < 1 << LU; u++) {
                C x[R];
                const int slot = fs0 + axis_reg<LU>(u, p.m.fs + LNT);
                C *g = gm + fa0 + axis_reg<LU>(u, p.m.fa + LNT);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if constexpr (INV) x[r] = ldg(g + axis_reg<lr>(r, p.m.fr));
                    else x[r] = S[slot + axis_slot(r << shp)];
                }
                dft<R, DIR, T, COMP>(x);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if constexpr (INV) {
                        S[slot + axis_slot(r << shp)] = x[r];
                    } else {
                        if (scl) x[r] = {x[r].x * sr - x[r].y * si, x[r].x * si + x[r].y * sr};
                        g[axis_reg<lr>(r, p.m.fr)] = x[r];
                    }
                }
            }
        } else {
            // thread -> (low line bits, v, index bits above the digit); the units of one `h`
            // differ in the highest line bits only
            constexpr int LUT = LTL < LU ? LTL : LU, LT0 = LTL - LUT, HI = 1 << (LU - LUT), LO = 1 << LUT;
            const tw<T> *tb = reinterpret_cast<const tw<T> *>(p.tw) + axis_tw(LN, LE, s);
#pragma unroll
            for (int h = 0; h < HI; h++) {
                const int U = tid + h * NT;
                const int iv = U >> LT0;                       // (bits above the digit, v)
                const int v = iv & ((1 << sh) - 1);
                const int i = ((iv >> sh) << (sh + lr)) | v;
                const int slot = axis_slot((i << LTL) | (U & ((1 << LT0) - 1)));
                C x[LO][R];
#pragma unroll
                for (int q = 0; q < LO; q++) {
#pragma unroll
                    for (int r = 0; r < R; r++) x[q][r] = S[slot + axis_slot(q << LT0 | r << shp)];
                }
                if constexpr (INV) {
#pragma unroll
                    for (int r = 1; r < R; r++) {
                        const tw<T> w = ldtw(tb, (r << sh) + v);
#pragma unroll
                        for (int q = 0; q < LO; q++) x[q][r] = twmul<true>(x[q][r], w);
                    }
                }
#pragma unroll
                for (int q = 0; q < LO; q++) dft<R, DIR, T, COMP>(x[q]);
                if constexpr (!INV) {
#pragma unroll
                    for (int r = 1; r < R; r++) {
                        const tw<T> w = ldtw(tb, (r << sh) + v);
#pragma unroll
                        for (int q = 0; q < LO; q++) x[q][r] = twmul<false>(x[q][r], w);
                    }
                }
#pragma unroll
                for (int q = 0; q < LO; q++) {
#pragma unroll
                    for (int r = 0; r < R; r++) S[slot + axis_slot(q << LT0 | r << shp)] = x[q][r];
                }
            }
        }
    }
    template <int s> static ZM_DEV void forward_from(C *S, C *gm, const AxisParams &p, int tid, bool scl, T sr, T si) {
        __syncthreads();
        stage<s>(S, gm, p, tid, scl, sr, si);
        if constexpr (s + 1 < NST) forward_from<s + 1>(S, gm, p, tid, scl, sr, si);
    }
    template <int s> static ZM_DEV void inverse_from(C *S, C *gm, const AxisParams &p, int tid) {
        stage<s>(S, gm, p, tid, false, T(1), T(0));
        __syncthreads();
        if constexpr (s > 0) inverse_from<s - 1>(S, gm, p, tid);
    }
};

template <typename T, int LN, int LTL, int LP, int LE, bool INV>
__global__ void __launch_bounds__((AxisCfg<T, LN, LTL, LP, LE>::NT), (AxisCfg<T, LN, LTL, LP, LE>::MINB))
    axis_pass_kernel(const __grid_constant__ AxisParams p) {
    using A = AxisPass<T, LN, LTL, LP, LE, INV>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *S = reinterpret_cast<cpx<T> *>(smem_raw);
    const int tid = threadIdx.x;
    const LineAddr la = line_addr(p.g, p.kind, (int64_t)blockIdx.x << LTL, p.m.lg);
    const cpx<T> *in = reinterpret_cast<const cpx<T> *>(p.in);
    cpx<T> *out = reinterpret_cast<cpx<T> *>(p.out);
    const bool scl = p.apply_scale;
    const T sr = (T)p.scale_re, si = (T)p.scale_im;
    if constexpr (!INV) {
        A::load_vec(S, in + la.a_base, p.m, tid);
        A::template forward_from<0>(S, out + la.f_base, p, tid, scl, sr, si);
    } else {
        A::template inverse_from<A::NST - 1>(S, const_cast<cpx<T> *>(in) + la.f_base, p, tid);
        A::store_vec(S, out + la.a_base, p.m, tid, scl, sr, si);
    }
}

template <typename T, int LN, int LTL, int LP, int LE, bool INV>
cudaError_t launch_axis(const AxisParams &p, int64_t nlines, cudaStream_t st) {
    using CF = AxisCfg<T, LN, LTL, LP, LE>;
    auto kern = axis_pass_kernel<T, LN, LTL, LP, LE, INV>;
    if constexpr (CF::SMEM > 48 * 1024) {
        static bool done[64] = {false};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 64 || !done[dev]) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CF::SMEM);
            if (e != cudaSuccess) return e;
            if (dev < 64) done[dev] = true;
        }
    }
    kern<<<(unsigned)(nlines >> LTL), CF::NT, CF::SMEM, st>>>(p);
    count_launch();
    return cudaGetLastError();
}

}  // namespace zm
