// zm_layout.cu -- layout converters, reciprocal-space pointwise operators and
// seeded field generators on the interleaved layouts.
//
// The converters are bit permutations; the others are element-wise maps driven by the index
// maps of zmodel/utils.h: real_to_global (166-170, 193-198) for the real-space layout and
// reciprocal_to_global (265-268, 298-302) for the transform output.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "zm_common.cuh"
#include "zm_index.cuh"
#include "zm_internal.h"

namespace zm {

// ------------------------------------------------------------------ converters
// N, B and P are powers of two, so natural order <-> real or reciprocal layout permutes the
// bits of the element index.  A CTA moves a tile whose index bits are the lowest bits of
// both sides' addresses (PermMap, built once per plan): it reads it in the order of the
// input's addresses and writes it in the order of the output's, through shared memory, so
// both sides move as runs of 256 bytes or more whatever the layout.  Slots are padded as in
// the axis pass (bit b weighs 2^(b mod 4) modulo the banks), and the tile bits are numbered
// so that the lanes of either side fall on distinct banks.
// Bound by DRAM (N = 8192 c64: 0.165 ms for 2F at the copy bandwidth).  P = 4, B = 8: natural
// -> real 0.288 -> 0.163 ms, real -> natural 0.800 -> 0.162; B = 256 (VP = 2): natural ->
// reciprocal 0.508 -> 0.168, reciprocal -> natural 1.647 -> 0.166 ms, against kernels that
// gathered or scattered element by element, or in transposes of up to VP frequencies.
// Tiles of twice the size leave six CTAs per SM: 0.185 ms (c128 0.370 -> 0.320 ms).
__host__ __device__ constexpr int perm_slot(int i) { return i + (i >> 4) + (i >> 8); }

// E = 2^LE elements per tile, 2^(LE - 8) per thread
template <typename T, int LE>
__global__ void __launch_bounds__(256) permute_kernel(const cpx<T> *in, cpx<T> *out,
                                                      const __grid_constant__ PermMap m) {
    constexpr int LP = LE > 8 ? LE - 8 : 0, LNT = LE - LP, EPT = 1 << LP;
    constexpr bool PAIR = sizeof(T) == 4 && LP >= 1;   // 16-byte accesses: address bit 0 in the registers
    constexpr int R0 = PAIR ? 1 : 0;                   // list position of the first thread bit
    __shared__ cpx<T> S[perm_slot((1 << LE) - 1) + 1];
    const int tid = threadIdx.x;
    // register bit q of a side: list entry 0 (PAIR) or the ones behind the thread bits
    auto reg = [](int q) { return PAIR && q == 0 ? 0 : LNT + q; };
    int64_t bi = 0, bo = 0;
    for (int f = 0; f < m.nf; f++) {
        bi += (int64_t)(blockIdx.x & m.fmask[f]) << m.fin[f];
        bo += (int64_t)((blockIdx.x & m.fmask[f]) >> m.flow[f]) << m.fout[f];
    }
    int si = 0, so = 0;
#pragma unroll
    for (int b = 0; b < LNT; b++) {
        const int bit = tid >> b & 1;
        bi += (int64_t)bit << m.ia[R0 + b];
        si += bit * m.is[R0 + b];
        bo += (int64_t)bit << m.oa[R0 + b];
        so += bit * m.os[R0 + b];
    }
    auto off = [&](int r, const unsigned char *a) {
        int64_t o = 0;
#pragma unroll
        for (int q = 0; q < LP; q++)
            if (r >> q & 1) o += int64_t{1} << a[reg(q)];
        return o;
    };
    auto slot = [&](int r, const short *s) {
        int o = 0;
#pragma unroll
        for (int q = 0; q < LP; q++)
            if (r >> q & 1) o += s[reg(q)];
        return o;
    };
    cpx<T> v[EPT];
    overlap_wait();
#pragma unroll
    for (int r = 0; r < EPT; r += 1 + R0) {
        if constexpr (PAIR) {
            const float4 q = ld_field(reinterpret_cast<const float4 *>(in + bi + off(r, m.ia)));
            v[r] = {q.x, q.y};
            v[r + 1] = {q.z, q.w};
        } else {
            v[r] = ld_field(in + bi + off(r, m.ia));
        }
    }
#pragma unroll
    for (int r = 0; r < EPT; r++) S[si + slot(r, m.is)] = v[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < EPT; r += 1 + R0) {
        cpx<T> *o = out + bo + off(r, m.oa);
        if constexpr (PAIR) {
            const cpx<T> x = S[so + slot(r, m.os)], y = S[so + slot(r + 1, m.os)];
            *reinterpret_cast<float4 *>(o) = make_float4(x.x, x.y, y.x, y.y);
        } else {
            *o = S[so + slot(r, m.os)];
        }
    }
}

// nat[b]: natural address bit of interleaved address bit b
PermMap perm_map(const Geom &g, int dtype, bool reciprocal, bool to_natural) {
    PermMap m;
    memset(&m, 0, sizeof m);
    const int tb = g.dim * g.logN;
    m.le = std::min(tb, dtype == 0 ? 10 : 11);   // 17 KB of shared memory, eight CTAs per SM
    std::vector<int> out_of(tb), in_of(tb);   // output bit of an input bit and back
    for (int b = 0; b < tb; b++) {
        const int64_t w = reciprocal ? recip_gidx(int64_t{1} << b, g) : real_gidx(int64_t{1} << b, g);
        int nat = 0;
        while ((int64_t{1} << nat) < w) nat++;
        if (to_natural) out_of[b] = nat;
        else out_of[nat] = b;
    }
    for (int b = 0; b < tb; b++) in_of[out_of[b]] = b;
    // tile bits (named by their input bit): the lowest of both sides in turn
    std::vector<char> in_tile(tb, 0);
    int count = 0;
    auto take = [&](int ib) {
        if (count < m.le && !in_tile[ib]) {
            in_tile[ib] = 1;
            count++;
        }
    };
    for (int q = 0; q < tb; q++) take(q), take(in_of[q]);
    std::vector<int> li, lo, rest;   // by input address, by output address
    for (int b = 0; b < tb; b++) (in_tile[b] ? li : rest).push_back(b);
    lo = li;
    std::sort(lo.begin(), lo.end(), [&](int x, int y) { return out_of[x] < out_of[y]; });
    // index bits: `ph` lane bits of the input side at 0 .. ph - 1, those of the output side
    // on different bits modulo 4, the others behind
    const int ph = std::min(dtype == 0 ? 3 : 4, m.le - (m.le > 8 && dtype != 0 ? 1 : 0)), r0 = m.le > 8 && dtype != 0 ? 1 : 0;
    std::vector<int> idx(tb, -1);
    std::vector<char> used(m.le, 0);
    auto put = [&](int bit, int at) {
        idx[bit] = at;
        used[at] = 1;
    };
    for (int q = 0; q < ph; q++) put(li[r0 + q], q);
    unsigned taken = 0;
    for (int q = 0; q < ph; q++)
        if (idx[lo[r0 + q]] >= 0) taken |= 1u << (idx[lo[r0 + q]] & 3);
    for (int q = 0; q < ph; q++) {
        const int bit = lo[r0 + q];
        if (idx[bit] >= 0) continue;
        for (int pass = 0; pass < 2 && idx[bit] < 0; pass++)
            for (int at = 0; at < m.le && idx[bit] < 0; at++)
                if (!used[at] && (pass == 1 || (!(taken >> (at & 3) & 1) && (at & 3) < (dtype == 0 ? 3 : 4)))) {
                    put(bit, at);
                    taken |= 1u << (at & 3);
                }
    }
    for (int b : li)
        if (idx[b] < 0)
            put(b, (int)(std::find(used.begin(), used.end(), 0) - used.begin()));
    for (int q = 0; q < m.le; q++) {
        m.ia[q] = (unsigned char)li[q];
        m.is[q] = (short)perm_slot(1 << idx[li[q]]);
        m.oa[q] = (unsigned char)out_of[lo[q]];
        m.os[q] = (short)perm_slot(1 << idx[lo[q]]);
    }
    // block index bits in input order, in fields of consecutive bits on both sides
    for (size_t j = 0; j < rest.size(); j++) {
        if (j > 0 && rest[j] == rest[j - 1] + 1 && out_of[rest[j]] == out_of[rest[j - 1]] + 1) {
            m.fmask[m.nf - 1] |= 1u << j;
            continue;
        }
        m.fmask[m.nf] = 1u << j;
        m.flow[m.nf] = (unsigned char)j;
        m.fin[m.nf] = (unsigned char)(rest[j] - (int)j);
        m.fout[m.nf] = (unsigned char)out_of[rest[j]];
        m.nf++;
    }
    return m;
}

template <typename T, int LE>
static cudaError_t launch_permute(const PermMap &m, int64_t tiles, const void *in, void *out, cudaStream_t st) {
    count_launch();
    return launch_overlapped(permute_kernel<T, LE>, (unsigned)tiles, LE < 8 ? 1 << LE : 256, 0, st,
                             reinterpret_cast<const cpx<T> *>(in), reinterpret_cast<cpx<T> *>(out), m);
}

cudaError_t launch_convert(const zm_plan_s *p, bool reciprocal, bool to_natural, const void *in,
                           void *out, cudaStream_t st) {
    const PermMap &m = p->perm[reciprocal][to_natural];
    const int64_t tiles = p->total >> m.le;
#define ZM_PERM(T, LE) \
    case LE: return launch_permute<T, LE>(m, tiles, in, out, st);
    if (p->dtype == 0) {
        switch (m.le) {
            ZM_PERM(double, 2) ZM_PERM(double, 4) ZM_PERM(double, 6) ZM_PERM(double, 8) ZM_PERM(double, 9)
            ZM_PERM(double, 10) ZM_PERM(double, 3)
        default: return cudaErrorInvalidValue;
        }
    } else {
        switch (m.le) {
            ZM_PERM(float, 2) ZM_PERM(float, 4) ZM_PERM(float, 6) ZM_PERM(float, 8) ZM_PERM(float, 9)
            ZM_PERM(float, 10) ZM_PERM(float, 3) ZM_PERM(float, 11)
        default: return cudaErrorInvalidValue;
        }
    }
#undef ZM_PERM
}

// --------------------------------------------------------- spectral operators
// CEPT consecutive elements at a CEPT-aligned index, as 16-byte vectors (N^dim, N >= 2, is a
// multiple of CEPT)
constexpr int CEPT = 4;
template <typename T> ZM_DEV void ld_run(const cpx<T> *p, cpx<T> *v) {
    constexpr int NV = CEPT * (int)sizeof(cpx<T>) / 16;
#pragma unroll
    for (int q = 0; q < NV; q++)
        reinterpret_cast<uint4 *>(v)[q] = ld_field(reinterpret_cast<const uint4 *>(p) + q);
}
template <typename T> ZM_DEV void st_run(cpx<T> *p, const cpx<T> *v) {
    constexpr int NV = CEPT * (int)sizeof(cpx<T>) / 16;
#pragma unroll
    for (int q = 0; q < NV; q++) reinterpret_cast<uint4 *>(p)[q] = reinterpret_cast<const uint4 *>(v)[q];
}
// Each thread scales CEPT consecutive elements.  The multiplier is computed in the
// working precision: FP64 for complex128; FP32 for complex64, where its relative error
// (a few ulp of FP32) stays far inside the complex64 bar, and the FP64 exp / division
// made the kernel issue bound.
// I: the integer type of the frequencies and of |k|^2, int32_t where 3 (N / 2)^2 fits
// (N <= 2^14), exact either way.  The CEPT positions share the other axes'
// frequencies; along the position axis bit b of the position is worth 2^b inside a run of
// VP, and VEC 2^(b - log VP) beyond it (reciprocal_to_global, utils.h:265-268), one constant
// per bit, so layouts with VP < 4 take no full map per element either (N = 4096 c64,
// VP = 1: 92 -> 43 us, VP >= 4: 43 / 45 -> 43; c128 107 -> 93 / 104 us; Gaussian / Poisson).
template <typename T, typename I>
__global__ void __launch_bounds__(256) spectral_kernel(cpx<T> *d, const Geom g, int64_t total, int op,
                                                       double a) {
    const int64_t e0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * CEPT;
    overlap_wait();
    if (e0 >= total) return;
    cpx<T> v[CEPT];
    ld_run(d + e0, v);
    const I n = (I)g.n, half = n >> 1;
    const T inv2a2 = (T)(1.0 / (2.0 * a * a)), inva2 = (T)(1.0 / (a * a)), ta = (T)a;
    auto sgn = [&](int64_t k) { return (I)k >= half ? (I)k - n : (I)k; };
    int64_t k0, k1, k2;
    recip_k(e0, g, k0, k1, k2);
    const bool shared = g.logL >= 2;   // the CEPT elements lie in one row
    const I kp = (I)(g.dim == 2 ? k1 : k0);
    const I sb = g.dim == 2 ? 0 : sgn(k1), sc = sgn(k2), r2 = sb * sb + sc * sc;
    const I w0 = g.logVP > 0 ? 1 : (I)g.vec, w1 = g.logVP > 1 ? 2 : (I)g.vec << (1 - g.logVP);
#pragma unroll
    for (int i = 0; i < CEPT; i++) {
        I ksq;
        if (shared) {
            const I k = kp + (i & 1 ? w0 : 0) + (i & 2 ? w1 : 0), s = k >= half ? k - n : k;
            ksq = r2 + s * s;
        } else {
            recip_k(e0 + i, g, k0, k1, k2);
            const I s0 = g.dim == 2 ? 0 : sgn(k0), s1 = sgn(k1), s2 = sgn(k2);
            ksq = s0 * s0 + s1 * s1 + s2 * s2;
        }
        const T k2sum = (T)ksq;   // exact in FP64; one rounding in FP32
        T f;
        if (op == 0) f = exp(-k2sum * inv2a2);
        else if (op == 1) f = k2sum == (T)0 ? (T)0 : -inva2 / k2sum;
        else f = ta;
        v[i] = {v[i].x * f, v[i].y * f};
    }
    st_run(d + e0, v);
}

template <typename T>
static cudaError_t spectral_t(const zm_plan_s *p, void *data, int op, double a, cudaStream_t st) {
    const int threads = 256;
    const unsigned grid = (unsigned)((p->total / CEPT + threads - 1) / threads);
    cpx<T> *d = reinterpret_cast<cpx<T> *>(data);
    count_launch();
    return launch_overlapped(p->g.logN <= 14 ? spectral_kernel<T, int32_t> : spectral_kernel<T, int64_t>, grid,
                             threads, 0, st, d, p->g, p->total, op, a);
}

cudaError_t launch_spectral(const zm_plan_s *p, void *data, int op, double a, cudaStream_t st) {
    return p->dtype == 0 ? spectral_t<double>(p, data, op, a, st) : spectral_t<float>(p, data, op, a, st);
}

template <typename T>
__global__ void fill_kernel(cpx<T> *__restrict__ d, const Geom g, int64_t total, int kind, uint64_t seed) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const uint64_t gi = (uint64_t)real_gidx(e, g);
    double re, im;
    if (kind == 0) {
        re = u01(seed, gi, 0) * 2.0 - 1.0;
        im = u01(seed, gi, 1) * 2.0 - 1.0;
    } else {
        re = gauss(seed, gi, 0);
        im = gauss(seed, gi, 1);
    }
    d[e] = {(T)re, (T)im};
}

cudaError_t launch_fill(const zm_plan_s *p, void *data, int kind, uint64_t seed, cudaStream_t st) {
    const int threads = 256;
    const unsigned grid = (unsigned)((p->total + threads - 1) / threads);
    if (p->dtype == 0)
        fill_kernel<double><<<grid, threads, 0, st>>>(reinterpret_cast<cpx<double> *>(data), p->g,
                                                      p->total, kind, seed);
    else
        fill_kernel<float><<<grid, threads, 0, st>>>(reinterpret_cast<cpx<float> *>(data), p->g,
                                                     p->total, kind, seed);
    count_launch();
    return cudaGetLastError();
}

constexpr int kMaxModes = 64;
struct ModeSet {
    int n;
    double noise;
    uint64_t seed;
    int64_t kx[kMaxModes], ky[kMaxModes];
    double ar[kMaxModes], ai[kMaxModes];
};

template <typename T>
__global__ void modes_kernel(cpx<T> *__restrict__ d, const Geom g, int64_t total, const ModeSet ms) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const int64_t gi = real_gidx(e, g);
    const int64_t gr = gi >> g.logN, gc = gi & (g.n - 1);
    double re = 0.0, im = 0.0;
    for (int m = 0; m < ms.n; m++) {
        // exact phase (kx x + ky y) mod N, then one sincospi
        const int64_t ph = (ms.kx[m] * gc + ms.ky[m] * gr) & (g.n - 1);
        double s, c;
        sincospi(2.0 * (double)ph / (double)g.n, &s, &c);
        re += ms.ar[m] * c - ms.ai[m] * s;
        im += ms.ar[m] * s + ms.ai[m] * c;
    }
    if (ms.noise != 0.0) {
        re += ms.noise * gauss(ms.seed, (uint64_t)gi, 0);
        im += ms.noise * gauss(ms.seed, (uint64_t)gi, 1);
    }
    d[e] = {(T)re, (T)im};
}

cudaError_t launch_fill_modes(const zm_plan_s *p, void *data, int nmodes, const int64_t *modes,
                              const double *amps, double noise, uint64_t seed, cudaStream_t st) {
    if (nmodes < 0 || nmodes > kMaxModes || p->g.dim != 2) return cudaErrorInvalidValue;
    ModeSet ms;
    ms.n = nmodes;
    ms.noise = noise;
    ms.seed = seed;
    for (int m = 0; m < nmodes; m++) {
        // reduce to [0, N) so the device phase product stays non-negative
        ms.kx[m] = ((modes[2 * m] % p->g.n) + p->g.n) % p->g.n;
        ms.ky[m] = ((modes[2 * m + 1] % p->g.n) + p->g.n) % p->g.n;
        ms.ar[m] = amps[2 * m];
        ms.ai[m] = amps[2 * m + 1];
    }
    const int threads = 256;
    const unsigned grid = (unsigned)((p->total + threads - 1) / threads);
    if (p->dtype == 0)
        modes_kernel<double><<<grid, threads, 0, st>>>(reinterpret_cast<cpx<double> *>(data), p->g,
                                                       p->total, ms);
    else
        modes_kernel<float><<<grid, threads, 0, st>>>(reinterpret_cast<cpx<float> *>(data), p->g,
                                                      p->total, ms);
    count_launch();
    return cudaGetLastError();
}

}  // namespace zm
