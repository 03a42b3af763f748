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
// The same as a trait of AxisPass, which other digit lists replace (zm_batch_exact.cu):
// row(s): log2 entries per row of stage s's table; col<s>(iv): the entry of a thread whose
// index bits outside the digit are iv (those above it, then the lower digits v)
template <int LN, int LE> struct AxisDigits {
    static constexpr int NST = axis_stages(LN, LE);
    static constexpr int lr(int s) { return axis_lr(LN, LE, s); }
    static constexpr int sh(int s) { return axis_sh(LN, LE, s); }
    static constexpr int row(int s) { return sh(s); }
    static constexpr int tw(int s) { return axis_tw(LN, LE, s); }
    template <int s> static __host__ __device__ constexpr int col(int iv) { return iv & ((1 << sh(s)) - 1); }
    static constexpr int r0(int) { return 1; }   // first row whose entries are not all 1
};
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

    // Twiddles kept in tensor memory by the persistent form: a thread's entries of stage s are
    // the rows k = 1 .. R - 1 of its HI index values, four words each, in its own lane.
    static constexpr int units(int s) {
        const int lu = LP - axis_lr(LN, LE, s);
        return 1 << (lu - (LTL < lu ? LTL : lu));
    }
    static constexpr int words(int s) { return 4 * ((1 << axis_lr(LN, LE, s)) - 1) * units(s); }
    // 512 columns hold NT / 128 threads per lane and MINB CTAs per SM
    static constexpr int BUDGET = NT >= 128 ? 512 / MINB / (NT / 128) : 0;
    // stages in tensor memory: from the last one back, as many as fit
    static constexpr int first_tm() {
        int w = 0, s = NST - 1;
        while (s > 0 && w + (words(s - 1) + 15) / 16 * 16 <= BUDGET) w += (words(--s) + 15) / 16 * 16;
        return s;
    }
    static constexpr int TM0 = first_tm();
    static constexpr int tm_at(int s) {   // first column of stage s in a thread's share
        int w = 0;
        for (int q = TM0; q < s; q++) w += (words(q) + 15) / 16 * 16;
        return w;
    }
    static constexpr int SHARE = tm_at(NST - 1);
    static constexpr int cols() {
        int c = 32;
        while (c < SHARE * (NT / 128)) c *= 2;
        return c;
    }
    // The persistent form is for tiles that leave room for one CTA per SM, where nothing else
    // covers a tile's loads: N = 8192 c64 701 / 728 -> 646 / 682 us forward / inverse, c128
    // 1402 / 1535 -> 1182 / 1491 (twiddles in tensor memory alone 695 / 730 and 1354 / 1479).
    // With two CTAs or more it is no faster (N = 4096 c64 136 / 160 against 142 / 159, 3D
    // N = 256 c64 156 / 159 against 175 / 177), nor on one-line complex64 tiles of 2^14
    // points, whose strided side moves single elements (4266 / 3520 against 4472 / 4342).
    static constexpr bool TM_OK = MINB == 1 && LN == 13 && TM0 < NST - 1 && cols() <= 512;
};

// The weight tables as the kernel sees them: launch parameters, or a table in global memory
// (batches, one per field layout).
template <bool CONST> struct AxisParamMapOf {
    static constexpr bool CONST_IN = CONST;   // ld_field: a plain launch that does not write its input
    static constexpr int COMP64 = 2;          // compensated codelet constants in complex64 (dft)
    const AxisMap &m;
    ZM_DEV int va(int i) const { return m.va[i]; }
    ZM_DEV int vs(int i) const { return m.vs[i]; }
    ZM_DEV int fa(int i) const { return m.fa[i]; }
    ZM_DEV int fs(int i) const { return m.fs[i]; }
    ZM_DEV int fr(int i) const { return m.fr[i]; }
};
using AxisParamMap = AxisParamMapOf<false>;
struct AxisGlobalMap {
    static constexpr bool CONST_IN = false;   // an earlier step of the launch wrote it
    // (forward, division, inverse of 256 fields of 256^2: 1.86e-7 of FP64 with 2, 1.76e-7 with 3,
    // which is 0.5 % slower)
    static constexpr int COMP64 = 3;
    const AxisMap *m;
    ZM_DEV int va(int i) const { return __ldg(m->va + i); }
    ZM_DEV int vs(int i) const { return __ldg(m->vs + i); }
    ZM_DEV int fa(int i) const { return __ldg(m->fa + i); }
    ZM_DEV int fs(int i) const { return __ldg(m->fs + i); }
    ZM_DEV int fr(int i) const { return __ldg(m->fr + i); }
};

// sum of the weights w(0 .. NB - 1) over the set bits of x (a constant, once unrolled, for
// the registers of a thread)
template <int NB, typename W> ZM_DEV int axis_bits(int x, W &&w) {
    int o = 0;
#pragma unroll
    for (int b = 0; b < NB; b++) o += (x >> b & 1) * w(b);
    return o;
}

template <typename T, int LN, int LTL, int LP, int LE, bool INV, typename MAP = AxisParamMap,
          typename D = AxisDigits<LN, LE>>
struct AxisPass {
    using C = cpx<T>;
    using CF = AxisCfg<T, LN, LTL, LP, LE>;
    static constexpr int NT = CF::NT, LNT = CF::LNT, NST = D::NST, EPT = 1 << LP;
    static constexpr int DIR = INV ? 1 : -1;
    // codelet constants as hi + lo pairs: the 45 degree ones, and complex64's 32-point level.
    // Round trip against FP64, without and with: 3D N = 256 c64 2.8e-7 / 2.4e-7 (at every
    // constant 2.2e-7), N = 1024 (32-point digits) 2.8e-7 / 2.2e-7, 3D N = 512 3.3e-7 /
    // 2.6e-7; 3D N = 256 c128 5.4e-16 / 4.2e-16; times within 1 % of each other.
    static constexpr int COMP = sizeof(T) == 4 ? MAP::COMP64 : 1;

    // global vector side <-> tile, in address order: thread bits first; complex64 keeps the
    // lowest address bit in the registers (16-byte accesses)
    // BAR: a barrier between the loads and the tile's first write (the tile is still being read)
    template <bool BAR = false> static ZM_DEV void load_vec(C *S, const C *in, const MAP &m, int tid) {
        in += axis_bits<LNT>(tid, [&](int b) { return m.va(b); });
        S += axis_bits<LNT>(tid, [&](int b) { return m.vs(b); });
        auto ra = [&](int r) { return axis_bits<LP>(r, [&](int b) { return m.va(LNT + b); }); };
        auto rs = [&](int r) { return axis_bits<LP>(r, [&](int b) { return m.vs(LNT + b); }); };
        C v[EPT];
        if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int r = 0; r < EPT; r += 2) {
                const float4 *g = reinterpret_cast<const float4 *>(in + ra(r));
                const float4 q = ld_field<MAP::CONST_IN>(g);
                v[r] = {q.x, q.y};
                v[r + 1] = {q.z, q.w};
            }
        } else {
#pragma unroll
            for (int r = 0; r < EPT; r++) v[r] = ld_field<MAP::CONST_IN>(in + ra(r));
        }
        if constexpr (BAR) __syncthreads();
#pragma unroll
        for (int r = 0; r < EPT; r++) S[rs(r)] = v[r];
    }
    // this thread's share of the next tile into L2
    static ZM_DEV void prefetch(const void *p) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"((unsigned long long)__cvta_generic_to_global(p)));
    }
    static ZM_DEV void prefetch_vec(const C *in, const MAP &m, int tid) {
        in += axis_bits<LNT>(tid, [&](int b) { return m.va(b); });
#pragma unroll
        for (int r = 0; r < EPT; r += sizeof(T) == 4 ? 2 : 1)
            prefetch(in + axis_bits<LP>(r, [&](int b) { return m.va(LNT + b); }));
    }
    static ZM_DEV void prefetch_edge(const C *gm, const MAP &m, int tid) {
        constexpr int lr = D::lr(NST - 1), R = 1 << lr, LU = LP - lr;
        gm += axis_bits<LNT>(tid, [&](int b) { return m.fa(b); });
#pragma unroll
        for (int u = 0; u < 1 << LU; u++)
#pragma unroll
            for (int r = 0; r < R; r++)
                prefetch(gm + axis_bits<LU>(u, [&](int b) { return m.fa(LNT + b); }) + axis_bits<lr>(r, [&](int b) { return m.fr(b); }));
    }
    static ZM_DEV void store_vec(const C *S, C *out, const MAP &m, int tid, bool scl, T sr, T si) {
        out += axis_bits<LNT>(tid, [&](int b) { return m.va(b); });
        S += axis_bits<LNT>(tid, [&](int b) { return m.vs(b); });
        auto ra = [&](int r) { return axis_bits<LP>(r, [&](int b) { return m.va(LNT + b); }); };
        auto rs = [&](int r) { return axis_bits<LP>(r, [&](int b) { return m.vs(LNT + b); }); };
        constexpr int ST = sizeof(T) == 4 ? 2 : 1;
#pragma unroll
        for (int r = 0; r < EPT; r += ST) {
            C v[ST];
#pragma unroll
            for (int q = 0; q < ST; q++) {
                v[q] = S[rs(r + q)];
                if (scl) v[q] = {sr * v[q].x - si * v[q].y, sr * v[q].y + si * v[q].x};
            }
            if constexpr (ST == 2)
                *reinterpret_cast<float4 *>(out + ra(r)) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
            else out[ra(r)] = v[0];
        }
    }

    // The stage next to the frequency side (the last one forward, the first inverse): units
    // in frequency-side order, global memory at `gm` on that side.
    template <bool BAR = false> static ZM_DEV void edge_stage(C *S, C *gm, const MAP &m, int tid, bool scl, T sr, T si) {
        constexpr int lr = D::lr(NST - 1), R = 1 << lr, LU = LP - lr;
        gm += axis_bits<LNT>(tid, [&](int b) { return m.fa(b); });
        S += axis_bits<LNT>(tid, [&](int b) { return m.fs(b); });
        auto ga = [&](int r) { return axis_bits<lr>(r, [&](int b) { return m.fr(b); }); };
#pragma unroll
        for (int u = 0; u < 1 << LU; u++) {
            C x[R];
            C *s = S + axis_bits<LU>(u, [&](int b) { return m.fs(LNT + b); });
            C *g = gm + axis_bits<LU>(u, [&](int b) { return m.fa(LNT + b); });
#pragma unroll
            for (int r = 0; r < R; r++) {
                if constexpr (INV) x[r] = ld_field<MAP::CONST_IN>(g + ga(r));
                else x[r] = s[axis_slot(r << LTL)];
            }
            dft<R, DIR, T, COMP>(x);
            if constexpr (BAR && INV)
                if (u == 0) __syncthreads();
#pragma unroll
            for (int r = 0; r < R; r++) {
                if constexpr (INV) {
                    s[axis_slot(r << LTL)] = x[r];
                } else {
                    if (scl) x[r] = {x[r].x * sr - x[r].y * si, x[r].x * si + x[r].y * sr};
                    g[ga(r)] = x[r];
                }
            }
        }
    }
    // An inner stage: thread -> (low line bits, v, index bits above the digit); the units of
    // one `h` differ in the highest line bits only and share their twiddles.  TM: the
    // twiddles come from the thread's share of tensor memory at `tm`, else from the table.
    template <int s> struct Inner {
        static constexpr int lr = D::lr(s), sh = D::sh(s), shp = sh + LTL, R = 1 << lr, LU = LP - lr;
        static constexpr int LUT = LTL < LU ? LTL : LU, LT0 = LTL - LUT, HI = 1 << (LU - LUT), LO = 1 << LUT;
        static ZM_DEV int iv(int tid, int h) { return (tid + h * NT) >> LT0; }   // (bits above the digit, v)
        static ZM_DEV int col(int tid, int h) { return D::template col<s>(iv(tid, h)); }   // of the twiddle table
    };
    template <int s, bool TM> static ZM_DEV void inner_stage(C *S, const tw<T> *tb, uint32_t tm, int tid) {
        using G = Inner<s>;
        constexpr int R = G::R, HI = G::HI, LO = G::LO, LT0 = G::LT0, sh = G::sh, shp = G::shp, lr = G::lr;
        constexpr bool MEM = TM && s >= CF::TM0;
        tb += D::tw(s);
#pragma unroll
        for (int h = 0; h < HI; h++) {
            const int iv = G::iv(tid, h);
            const int i = ((iv >> sh) << (sh + lr)) | (iv & ((1 << sh) - 1));
            const int slot = axis_slot((i << LTL) | ((tid + h * NT) & ((1 << LT0) - 1)));
            C x[LO][R];
#pragma unroll
            for (int q = 0; q < LO; q++) {
#pragma unroll
                for (int r = 0; r < R; r++) x[q][r] = S[slot + axis_slot(q << LT0 | r << shp)];
            }
            auto twiddle = [&]() {
                if constexpr (MEM) {
                    // entry h (R - 1) + r - 1 of the stage, four entries per 16 columns
#pragma unroll
                    for (int c = h * (R - 1) / 4; c <= ((h + 1) * (R - 1) - 1) / 4; c++) {
                        uint32_t w16[16];
                        tmem_ld16(tm + CF::tm_at(s) + 16 * c, w16);
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int r = 4 * c + e - h * (R - 1) + 1;
                            if (r < 1 || r >= R) continue;
                            tw<T> w;
                            memcpy(&w, w16 + 4 * e, 16);
#pragma unroll
                            for (int q = 0; q < LO; q++) x[q][r] = twmul<INV>(x[q][r], w);
                        }
                    }
                } else {
#pragma unroll
                    for (int r = D::r0(s); r < R; r++) {
                        const tw<T> w = ldtw(tb, (r << D::row(s)) + G::col(tid, h));
#pragma unroll
                        for (int q = 0; q < LO; q++) x[q][r] = twmul<INV>(x[q][r], w);
                    }
                }
            };
            if constexpr (INV) twiddle();
#pragma unroll
            for (int q = 0; q < LO; q++) dft<R, DIR, T, COMP>(x[q]);
            if constexpr (!INV) twiddle();
#pragma unroll
            for (int q = 0; q < LO; q++) {
#pragma unroll
                for (int r = 0; r < R; r++) S[slot + axis_slot(q << LT0 | r << shp)] = x[q][r];
            }
        }
    }
    // this thread's entries of stages s .. into its share of tensor memory
    template <int s> static ZM_DEV void park_twiddles(const tw<T> *tb, uint32_t tm, int tid) {
        if constexpr (s < NST - 1) {
            using G = Inner<s>;
            constexpr int NE = (G::R - 1) * G::HI;
            const tw<T> *t = tb + D::tw(s);
#pragma unroll 1
            for (int c = 0; c < (NE + 3) / 4; c++) {
                uint32_t w16[16];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int n = 4 * c + e < NE ? 4 * c + e : NE - 1;
                    const int h = n / (G::R - 1), r = n % (G::R - 1) + 1;
                    const tw<T> w = ldtw(t, (r << D::row(s)) + G::col(tid, h));
                    memcpy(w16 + 4 * e, &w, 16);
                }
                tmem_st16(tm + CF::tm_at(s) + 16 * c, w16);
            }
            park_twiddles<s + 1>(tb, tm, tid);
        }
    }
    // stages s .. NST - 2 forward, s .. 0 inverse, a barrier before / after each
    template <int s, bool TM = false> static ZM_DEV void inner_stages(C *S, const tw<T> *tb, int tid, uint32_t tm = 0) {
        if constexpr (s >= 0 && s < NST - 1) {
            if constexpr (!INV) __syncthreads();
            inner_stage<s, TM>(S, tb, tm, tid);
            if constexpr (INV) __syncthreads();
            inner_stages<(INV ? s - 1 : s + 1), TM>(S, tb, tid, tm);
        }
    }
    // one tile, vector side -> frequency side (forward) or back; TM: persistent form, the
    // previous tile may still be read when this one starts
    template <bool TM = false>
    static ZM_DEV void run(C *S, const C *in, C *out, const MAP &m, const tw<T> *tb, int tid, bool scl, T sr, T si,
                           uint32_t tm = 0, const C *next = nullptr) {
        if constexpr (!INV) {
            load_vec<TM>(S, in, m, tid);
            if constexpr (TM)
                if (next) prefetch_vec(next, m, tid);
            inner_stages<0, TM>(S, tb, tid, tm);
            __syncthreads();
            edge_stage(S, out, m, tid, scl, sr, si);
        } else {
            edge_stage<TM>(S, const_cast<C *>(in), m, tid, false, T(1), T(0));
            if constexpr (TM)
                if (next) prefetch_edge(next, m, tid);
            __syncthreads();
            inner_stages<NST - 2, TM>(S, tb, tid, tm);
            store_vec(S, out, m, tid, scl, sr, si);
        }
    }
};

template <typename T, int LN, int LTL, int LP, int LE, bool INV>
__global__ void __launch_bounds__((AxisCfg<T, LN, LTL, LP, LE>::NT), (AxisCfg<T, LN, LTL, LP, LE>::MINB))
    axis_pass_kernel(const __grid_constant__ AxisParams p) {
    using A = AxisPass<T, LN, LTL, LP, LE, INV>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *S = reinterpret_cast<cpx<T> *>(smem_raw);
    overlap_next();
    const LineAddr la = line_addr(p.g, p.kind, (int64_t)blockIdx.x << LTL, p.m.lg);
    const cpx<T> *in = reinterpret_cast<const cpx<T> *>(p.in);
    cpx<T> *out = reinterpret_cast<cpx<T> *>(p.out);
    const tw<T> *tb = reinterpret_cast<const tw<T> *>(p.tw);
    const AxisParamMap m{p.m};
    overlap_wait();
    A::run(S, in + (INV ? la.f_base : la.a_base), out + (INV ? la.a_base : la.f_base), m, tb, threadIdx.x,
           p.apply_scale, (T)p.scale_re, (T)p.scale_im);
}

// The persistent form, one CTA per SM: CTA c walks tiles c, c + CTAs, ..., each thread's stage
// twiddles (the same for every tile) in tensor memory, and asks for its next tile in L2 as
// soon as it holds the current one.  CONST: non-coherent loads, for inverse passes that do
// not run in place, launched plainly (launch_axis).
template <typename T, int LN, int LTL, int LP, int LE, bool INV, bool CONST>
__global__ void __launch_bounds__((AxisCfg<T, LN, LTL, LP, LE>::NT), (AxisCfg<T, LN, LTL, LP, LE>::MINB))
    axis_tm_kernel(const __grid_constant__ AxisParams p, unsigned tiles) {
    using A = AxisPass<T, LN, LTL, LP, LE, INV, AxisParamMapOf<CONST>>;
    using CF = typename A::CF;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_tm;
    cpx<T> *S = reinterpret_cast<cpx<T> *>(smem_raw);
    const int tid = threadIdx.x;
    const tw<T> *tb = reinterpret_cast<const tw<T> *>(p.tw);
    if (tid < 32) tmem_alloc(&s_tm, CF::cols());
    __syncthreads();
    tmem_fence_after();
    const uint32_t tm0 = s_tm;
    // warp w reaches lanes 32 (w mod 4) ..; its column share is number w / 4
    const uint32_t tm = tm0 + ((uint32_t)(tid >> 5 & 3) << 21) + (uint32_t)(tid >> 7) * CF::SHARE;
    A::template park_twiddles<CF::TM0>(tb, tm, tid);
    overlap_next();
    overlap_wait();
    const cpx<T> *in = reinterpret_cast<const cpx<T> *>(p.in);
    cpx<T> *out = reinterpret_cast<cpx<T> *>(p.out);
    const AxisParamMapOf<CONST> m{p.m};
#pragma unroll 1
    for (unsigned c = blockIdx.x; c < tiles; c += gridDim.x) {
        const LineAddr la = line_addr(p.g, p.kind, (int64_t)c << LTL, p.m.lg);
        const cpx<T> *nx = nullptr;
        if (c + gridDim.x < tiles) {
            const LineAddr ln = line_addr(p.g, p.kind, (int64_t)(c + gridDim.x) << LTL, p.m.lg);
            nx = in + (INV ? ln.f_base : ln.a_base);
        }
        A::template run<true>(S, in + (INV ? la.f_base : la.a_base), out + (INV ? la.a_base : la.f_base), m, tb, tid,
                              p.apply_scale, (T)p.scale_re, (T)p.scale_im, tm, nx);
    }
    tmem_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tm0, CF::cols());
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
    const unsigned tiles = (unsigned)(nlines >> LTL);
    if constexpr (CF::TM_OK) {
        static int resident[64] = {0};
        int dev = 0;
        cudaGetDevice(&dev);
        // The inverse's strided loads are faster non-coherent (N = 8192, us per transform, coherent /
        // non-coherent: c64 704 / 682, c128 1545 / 1491; the forward's are not, c64 645 / 673), which
        // is right only for an input that nothing writes while the kernel runs: not in place, and
        // launched plainly, after all that came before it.
        auto ktm = axis_tm_kernel<T, LN, LTL, LP, LE, INV, false>;
        auto kconst = axis_tm_kernel<T, LN, LTL, LP, LE, INV, INV>;
        int ctas = dev < 64 ? resident[dev] : 0;
        if (!ctas) {
            int sms = 0;
            cudaError_t e = cudaFuncSetAttribute(ktm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CF::SMEM);
            if (e == cudaSuccess && INV)
                e = cudaFuncSetAttribute(kconst, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CF::SMEM);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            ctas = sms;   // one per SM
            if (dev < 64) resident[dev] = ctas;
        }
        if (tiles >= 3 * (unsigned)ctas) {
            count_launch();
            if (INV && p.in != p.out) {
                kconst<<<(unsigned)ctas, CF::NT, CF::SMEM, st>>>(p, tiles);
                return cudaGetLastError();
            }
            return launch_overlapped(ktm, (unsigned)ctas, CF::NT, CF::SMEM, st, p, tiles);
        }
    }
    count_launch();
    return launch_overlapped(kern, tiles, CF::NT, CF::SMEM, st, p);
}

}  // namespace zm
