// zm_batch.cuh -- what the batch kernels share: the program of a launch, the grid barrier and
// the residual step.
#pragma once

#include <cuda/atomic>
#include <cuda_runtime.h>

#include "zm_index.cuh"
#include "zm_internal.h"

namespace zm {

constexpr int kBatchThreads = 256;
constexpr int kMaxSteps = 6;
constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;   // 2 s

struct BatchField {
    Geom g;
    int64_t off;       // element offset in a batch buffer
    int64_t tile0;     // first tile of this field in a pass step's tile sequence
    const void *twN;   // the field plan's twiddle table w_N^m (tw<T> entries)
    const AxisMap *ax; // weight tables of the x and y passes (batches on the axis tiles)
    const void *twx;   // their stage twiddles
    const AxisMap *ex; // tiles of zm_batch_exact.cu: tables of x forward, y, x inverse,
    const void *exf, *exi;   // and the forward and inverse stage twiddles
    int T;             // lines per tile
    int nst_vec, nst_m;
    int rad_vec[8], rad_m[8];
};

enum BatchOp : int {
    BOP_X_FWD = 0,     // x pass forward: real layout -> REPACK layout
    BOP_Y_FWD = 1,     // y pass forward: REPACK layout -> reciprocal layout
    BOP_Y_INV = 2,     // y pass inverse
    BOP_X_INV = 3,     // x pass inverse (scale 1/N^2 when step.scale)
    BOP_Y_POISSON = 4, // y pass forward, divide by -|k|^2, y pass inverse (in place)
    BOP_RESIDUAL = 5,  // out = Lap(in) / h^2 - aux (5-point, periodic)
    BOP_FILL = 6,      // out = generator(kind, seed + field) in the real layout
    BOP_NOP = 7        // nothing (barrier probe)
};

struct BatchStep {
    int op;
    int kind;          // BOP_FILL: zm_field_kind
    int scale;         // BOP_X_INV: apply 1/N^2
    const void *in;
    void *out;
    const void *aux;
    double a;          // BOP_Y_POISSON: 2 pi / length; BOP_RESIDUAL: 1 / length
    uint64_t seed;
};

struct BatchParams {
    const BatchField *fields;
    const int *tile_field;   // field of each tile (batches on the axis tiles)
    int nfields;
    int64_t tiles;
    int nsteps;
    BatchStep step[kMaxSteps];
    unsigned *bar;     // [0] arrivals, [1] generation
    int *abort;        // this launch only: set by a barrier that timed out, the others give up
    int *err;          // sticky: set by a barrier that timed out, read and cleared by zm_batch_status
    unsigned missing;  // arrivals a barrier waits for beyond the grid (0; > 0 only in the probe)
};

ZM_DEV unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier of a cooperative launch (all CTAs resident).  Sense by generation
// count; the last CTA to arrive resets the arrival count and releases the generation.
// A wait longer than kBarrierTimeoutNs, or an abort already raised by another CTA of
// this launch, makes every waiting CTA give up: returns false and the kernel returns.
// A timeout also raises the sticky error word that zm_batch_status reports; the abort
// word is cleared before every launch, so one timeout ends only its own launch.
ZM_DEV bool grid_barrier(unsigned *bar, unsigned nblocks, int *abort, int *err, int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> cnt(bar[0]), gen(bar[1]);
        cuda::atomic_ref<int, cuda::thread_scope_device> flag(*abort), sticky(*err);
        const unsigned g0 = gen.load(cuda::memory_order_acquire);
        if (cnt.fetch_add(1u, cuda::memory_order_acq_rel) == nblocks - 1) {
            cnt.store(0u, cuda::memory_order_relaxed);
            gen.fetch_add(1u, cuda::memory_order_release);
        } else {
            const unsigned long long t0 = globaltimer_ns();
            while (gen.load(cuda::memory_order_acquire) == g0) {
                if (flag.load(cuda::memory_order_relaxed) != 0 ||
                    globaltimer_ns() - t0 > kBarrierTimeoutNs) {
                    flag.store(1, cuda::memory_order_relaxed);
                    sticky.store(1, cuda::memory_order_relaxed);
                    ok = 0;
                    break;
                }
                __nanosleep(128);
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// Odd steps walk the tiles from the last: what the step before wrote last is still in the L2
// (126 MB), so a batch larger than that reads that part from there: 29 complex128 fields of
// N = 128 .. 1024 (89 MB a buffer) forward 138 -> 120 us, Poisson call 302 -> 284 us; 16
// complex64 fields of 1024^2 (134 MB) 354 -> 347 us; 96 fields (554 MB) unchanged.  From
// buffers of 77 MB (four turns of the walk): below, everything is in the L2 either way, and a
// CTA that keeps its tile is faster (300 complex128 fields of N = 64, Poisson call 70 us, 74
// reversed).
ZM_DEV bool walks_back(const BatchParams &bp, int step) { return (step & 1) && bp.tiles > 4 * (int64_t)gridDim.x; }

// the kernel of the complex64 Poisson call with a residual (zm_batch_exact.cu)
using BatchFn = void (*)(const BatchParams);
BatchFn batch_exact_fn();
// whether its tiles hold a field of this layout, and the digits of its transforms
bool batch_exact_fits(const Geom &g);
std::vector<int> batch_exact_digits(const Geom &g, bool inverse);
// exponents of its stage twiddles (w_N^e)
void batch_exact_twiddles(const Geom &g, bool inverse, std::vector<int64_t> *exps);

// One tile of the residual step, out = Lap_h(in) - rhs over elements [e0, e0 + TP) of a
// field (5-point, periodic, h = length / N, a = 1 / length); its own function so that its
// registers do not weigh on the rest of the persistent kernel.  A tile is whole rows of
// ranks: it is read once into shared memory, where the centre, the neighbours inside a
// rank's B x B block (-L, +L in rows, -VEC, +VEC in packed columns) come from; the rows
// above and below the tile and the neighbours across a block's edge come from global memory
// through the block-cyclic maps.  (With every neighbour from global memory the step moved
// five times the field between L2 and the SMs and ran the maps in 64 bits per neighbour: the
// whole Poisson call of 29 complex128 fields of N = 128 .. 1024 332 -> 309 us, of 100 fields of
// N = 64 57 -> 49 us.)
template <typename T, int TP>
__device__ __noinline__ void residual_tile(const Geom &g, double a, const cpx<T> *in, const cpx<T> *rhs, cpx<T> *out,
                                           int64_t e0, cpx<T> *S, int tid) {
    constexpr int K = 16 / (int)sizeof(cpx<T>), NV = TP / K / kBatchThreads;   // elements, vectors per thread
    struct __align__(16) V { cpx<T> v[K]; };
    const T inv_h2 = (T)((double)g.n * a * (double)g.n * a);
    const int iL = (int)g.L, iV = (int)g.vec, bm = (int)g.b - 1, logL = g.logL, logV = g.logVEC;
    auto resid = [&](const cpx<T> &up, const cpx<T> &dn, const cpx<T> &lf, const cpx<T> &rt,
                     const cpx<T> &c, const cpx<T> &r) -> cpx<T> {
        const T lx = up.x + dn.x + lf.x + rt.x - (T)4 * c.x;
        const T ly = up.y + dn.y + lf.y + rt.y - (T)4 * c.y;
        return {lx * inv_h2 - r.x, ly * inv_h2 - r.y};
    };
    auto ld = [](const cpx<T> *q) { return *reinterpret_cast<const V *>(q); };
    in += e0;
    rhs += e0;
    out += e0;
    __syncthreads();   // the previous tile is done with S
    {
        V t[NV];
#pragma unroll
        for (int q = 0; q < NV; q++) t[q] = ld(in + (tid + q * kBatchThreads) * K);
#pragma unroll
        for (int q = 0; q < NV; q++) *reinterpret_cast<V *>(S + (tid + q * kBatchThreads) * K) = t[q];
    }
    __syncthreads();
    const int P = (int)g.p, logLL = 2 * logL, vm = iV - 1;
#pragma unroll 2
    for (int q = 0; q < NV; q++) {
        const int i = (tid + q * kBatchThreads) * K;
        const V r = ld(rhs + i), c = ld(S + i);
        const int e = (int)e0 + i, pos = e & (iL - 1), lr = (e >> logL) & (iL - 1), rank = e >> logLL;
        const int j = pos >> logV, rb = lr & bm, rid = rank >> g.logP, cid = rank & (P - 1);
        V up, dn, lf, rt, o;
        // Across a block's edge (utils.h:122-128, 166-186): the row above row 0 of a block is
        // row B - 1 of the same block cycle in the rank above, or, past the first rank, of the
        // cycle before in the last one (local row lr - 1); likewise the other way and in columns,
        // where the cycle is the packed position's low part and moves by one element.
        if (rb > 0) up = i >= iL ? ld(S + i - iL) : ld(in + i - iL);
        else up = ld(in + i + (rid > 0 ? -(P << logLL) + (bm << logL)
                                       : ((P - 1) * P << logLL) + (((lr - 1) & (iL - 1)) - lr) * iL));
        if (rb < bm) dn = i + iL < TP ? ld(S + i + iL) : ld(in + i + iL);
        else dn = ld(in + i + (rid < P - 1 ? (P << logLL) - (bm << logL)
                                           : -((P - 1) * P << logLL) + (((lr + 1) & (iL - 1)) - lr) * iL));
        // element i + k, column neighbour d = -1 / +1, one by one
        auto side = [&](int k, int d) {
            const int pk = pos + k, jk = pk >> logV, jj = pk & vm;
            if (d < 0 ? jk > 0 : jk < bm) return S[i + k + d * iV];
            const bool wrap = d < 0 ? cid == 0 : cid == P - 1;
            const int to = ((d < 0 ? bm : 0) << logV) + (wrap ? (jj + d) & vm : jj);   // packed position
            return in[i + k + ((wrap ? -d * (P - 1) : d) * (1 << logLL)) + to - pk];
        };
        if (iV >= K && j > 0) lf = ld(S + i - iV);
        else if (iV >= K && cid > 0) lf = ld(in + i - (1 << logLL) + (bm << logV));
        else
#pragma unroll
            for (int k = 0; k < K; k++) lf.v[k] = side(k, -1);
        if (iV >= K && j < bm) rt = ld(S + i + iV);
        else if (iV >= K && cid < P - 1) rt = ld(in + i + (1 << logLL) - (bm << logV));
        else
#pragma unroll
            for (int k = 0; k < K; k++) rt.v[k] = side(k, 1);
#pragma unroll
        for (int k = 0; k < K; k++) o.v[k] = resid(up.v[k], dn.v[k], lf.v[k], rt.v[k], c.v[k], r.v[k]);
        *reinterpret_cast<V *>(out + i) = o;
    }
}

}  // namespace zm
