// zm_batch.cu -- many independent 2D fields of uneven N in one persistent launch.
//
// A batch is a list of fields, each with its own (N, B, P) reference layout, packed one
// after the other in every batch buffer.  One call is one cooperative launch of
// a persistent kernel: a grid of exactly the CTAs that fit on the device at once walks a short
// program of steps (an axis pass over all fields, a fused y pass, a stencil, a
// generator ...), with a grid barrier between steps.  Inside a pass step the work items
// are tiles of TL lines of one field, TL * N = a fixed number of points per tile, so the
// same CTA shape serves every N; a tile's field comes from a table, or in batch_kernel from a
// binary search over the fields' first tile numbers.  Three kernels hold the tile code:
// batch_axis_kernel on the axis pass sized by N alone (zm_batch_axis.cuh);
// batch_exact_kernel (zm_batch_exact.cu) for the complex64 Poisson call, which keeps the
// rounding of the VEC x M split (see zm_batch_poisson); and batch_kernel on that split
// (zm_tile.cuh) for a whole batch where one field does not fit the others' tiles: complex64
// Poisson calls with a field of VEC = 1 or above 16 (its compile-time VEC = 4 tiles serve
// that field's neighbours), and complex128 batches with a field of N = 32.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <map>
#include <new>
#include <tuple>
#include <vector>

#include "zm_batch.cuh"
#include "zm_batch_axis.cuh"
#include "zm_tile.cuh"
#include "zmodel_b200.h"

namespace zm {

// largest f with fields[f].tile0 <= tile
ZM_DEV int field_of_tile(const BatchField *fields, int nfields, int64_t tile) {
    int lo = 0, hi = nfields - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (fields[mid].tile0 <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Both sub-transforms of a tile: compile-time-sized stages (LMC = log2 M) for the
// complex64 tiles with VEC = 4 and P = 2 or 4 (B = N / 8 at P = 2), or the runtime-sized stages (LMC = 0) for every other
// shape.  (LMC > 0: the column sub-transform only; the row stage runs fused with the
// vector-side sweep, tile_load_rows_v4 / tile_rows_store_v4)
template <typename T, int EPT, bool INV, int LM, typename SW>
__device__ __noinline__ void tile_transform_v4(cpx<T> *s, int tid, const tw<T> *twN) {
    tile_transform_ct<T, EPT, INV, 2, LM, kBatchThreads, SW, false>(s, tid, twN);
}
template <typename T, int EPT, bool INV, int LMC, typename SW>
ZM_DEV void batch_tile_transform(cpx<T> *s, const BatchField &f, int nthr, int tid, const tw<T> *twN) {
    if constexpr (LMC > 0) {
        tile_transform_v4<T, EPT, INV, LMC, SW>(s, tid, twN);
    } else {
        const Geom &g = f.g;
        tile_transform<T, EPT, INV>(s, g, f.rad_vec, f.nst_vec, f.rad_m, f.nst_m, nthr, tid, twN);
    }
}

// One tile of an axis-pass step: load, transform(s), store.  SW is the shared-memory
// slot permutation of the tile (SwzV4 for the compile-time VEC = 4 tiles).
template <typename T, int EPT, int LMC, typename SW, int LP = 0>
__device__ __noinline__ void batch_tile(int op, bool scale, double a, const BatchField &sf, const Tile c, cpx<T> *s,
                                        const cpx<T> *in, cpx<T> *out, int64_t l0, int nthr, int tid) {
    const Geom &g = sf.g;
    const tw<T> *twN = reinterpret_cast<const tw<T> *>(sf.twN);
    const bool xpass = op == BOP_X_FWD || op == BOP_X_INV;
    // vector-side sweeps: plain, or with the VEC = 4 row stage fused in and every size
    // fixed (LMC > 0, P = 2^LP); likewise the frequency-side sweeps
    auto load_vec = [&]() {
        if constexpr (LMC > 0) {
            if (xpass) tile_load_rows_v4<EPT, LMC, LP, true, kBatchThreads, SW>(c, s, in, tid);
            else tile_load_rows_v4<EPT, LMC, LP, false, kBatchThreads, SW>(c, s, in, tid);
        } else {
            tile_load_vec<EPT, SW>(c, g, s, in, nthr, tid);
        }
    };
    auto store_vec = [&](bool scl, T sc) {
        if constexpr (LMC > 0) {
            if (xpass) tile_rows_store_v4<EPT, LMC, LP, true, kBatchThreads, SW>(c, s, out, scl, sc, (T)0, twN, tid);
            else tile_rows_store_v4<EPT, LMC, LP, false, kBatchThreads, SW>(c, s, out, scl, sc, (T)0, twN, tid);
        } else {
            tile_store_vec<EPT, SW>(c, g, s, out, scl, sc, (T)0, nthr, tid);
        }
    };
    auto store_freq = [&]() {
        if constexpr (LMC > 0) {
            if (xpass) tile_freq_v4<EPT, LMC, LP, true, kBatchThreads, false, SW>(c, s, in, out, tid);
            else tile_freq_v4<EPT, LMC, LP, false, kBatchThreads, false, SW>(c, s, in, out, tid);
        } else {
            tile_store_freq<EPT, SW>(c, g, s, out, false, (T)1, (T)0, nthr, tid);
        }
    };
    auto load_freq = [&]() {
        if constexpr (LMC > 0) {
            if (xpass) tile_freq_v4<EPT, LMC, LP, true, kBatchThreads, true, SW>(c, s, in, out, tid);
            else tile_freq_v4<EPT, LMC, LP, false, kBatchThreads, true, SW>(c, s, in, out, tid);
        } else {
            tile_load_freq<EPT, SW>(c, g, s, in, nthr, tid);
        }
    };
    if (op == BOP_X_FWD || op == BOP_Y_FWD) {
        load_vec();
        __syncthreads();
        batch_tile_transform<T, EPT, false, LMC, SW>(s, sf, nthr, tid, twN);
        store_freq();
    } else if (op == BOP_X_INV || op == BOP_Y_INV) {
        load_freq();
        __syncthreads();
        batch_tile_transform<T, EPT, true, LMC, SW>(s, sf, nthr, tid, twN);
        const bool scl = scale && xpass;
        const T sc = (T)(1.0 / ((double)g.n * (double)g.n));
        store_vec(scl, sc);
    } else {   // BOP_Y_POISSON
        load_vec();
        __syncthreads();
        batch_tile_transform<T, EPT, false, LMC, SW>(s, sf, nthr, tid, twN);
        // slot (t, k1, k2) holds the frequency the y pass would store at rank
        // (rid = k2 / VP, cid), local row p, column pos = k1 VP + k2 % VP
        // (reciprocal_to_global, utils.h:265-268): along the transform that is
        // d_ct(rid L + d_lp(pos)) = d_ct(k2 M + k1) = k1 VEC + k2 = r, the slot position
        // itself; along the lines d_ct(cid L + d_lp(p)) of line l0 + t.  The factor
        // -1 / (a^2 |k|^2) in the working precision (|k|^2 an exact integer).
        const T a2 = (T)(a * a);
        auto divide = [&](int e, int ka, int r, int nh, int n) {
            const int sa = ka >= nh ? ka - n : ka, sb = r >= nh ? r - n : r;
            const int ksq = sa * sa + sb * sb;
            T fac;
            if constexpr (sizeof(T) == 4) fac = ksq == 0 ? 0.f : -__frcp_rn(a2 * (float)ksq);
            else fac = ksq == 0 ? 0.0 : -1.0 / (a2 * (double)ksq);
            const cpx<T> v = s[SW::f(e)];
            s[SW::f(e)] = {v.x * fac, v.y * fac};
        };
        if constexpr (LMC > 0) {
            // the same with the sizes fixed: ka = ct(cid L + lp(p)) in 32-bit constant shifts
            using G = V4Geom<LMC, LP, false>;
            constexpr int M = 1 << LMC, LVP = G::LVP, VP = G::VP;
#pragma unroll 4
            for (int e = tid; e < EPT * kBatchThreads; e += kBatchThreads) {
                const int t = e >> G::LN, r = e & (G::N - 1);
                const int l = (int)l0 + t, cid = l >> G::LL, p = l & (G::L - 1);
                const int q = (cid << G::LL) + (p >> LVP) + ((p & (VP - 1)) << LMC);
                divide(e, ((q & (M - 1)) << 2) + (q >> LMC), r, G::N / 2, G::N);
            }
        } else {
            const int tot = sf.T << g.logN;
            for (int e = tid; e < tot; e += nthr) {
                const int t = e >> g.logN, r = e & (int)(g.n - 1);
                const int64_t l = l0 + t, cid = l >> g.logL, p = l & (g.L - 1);
                divide(e, (int)d_ct(cid * g.L + d_lp(p, g), g), r, (int)(g.n >> 1), (int)g.n);
            }
        }
        __syncthreads();
        batch_tile_transform<T, EPT, true, LMC, SW>(s, sf, nthr, tid, twN);
        store_vec(false, (T)1);
    }
}

template <typename T, int EPT>
__global__ void __launch_bounds__(kBatchThreads, 4) batch_kernel(const BatchParams bp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *s = reinterpret_cast<cpx<T> *>(smem_raw);
    __shared__ int64_t s_abase[64], s_fbase[64];
    __shared__ BatchField sf;
    __shared__ int s_ok, s_f;
    const int tid = threadIdx.x, nthr = blockDim.x;

    for (int st = 0; st < bp.nsteps; st++) {
        if (st > 0 && !grid_barrier(bp.bar, gridDim.x + bp.missing, bp.abort, bp.err, &s_ok)) return;
        const BatchStep S = bp.step[st];
        if (S.op == BOP_NOP) continue;

        if (S.op == BOP_RESIDUAL || S.op == BOP_FILL) {
            // element-wise steps over the pass steps' tiles: tile `tile` of field f covers
            // elements [(tile - tile0) * TP, + TP) of the field's array (N^2 / TP tiles of a
            // field of N^2 elements), so every CTA has work whatever the field sizes
            constexpr int TP0 = kBatchThreads * EPT;
            for (int64_t tile = blockIdx.x; tile < bp.tiles; tile += gridDim.x) {
                __syncthreads();   // the previous tile is done with sf
                if (tid == 0) {
                    s_f = field_of_tile(bp.fields, bp.nfields, tile);
                    sf = bp.fields[s_f];
                }
                __syncthreads();
                const int f = s_f;
                const Geom g = sf.g;
                const bool half = g.n * g.n < TP0;   // a field smaller than a tile is a tile of its own
                const int TP = half ? TP0 / 2 : TP0;
                const int64_t e0 = (tile - sf.tile0) * TP;
                cpx<T> *out = reinterpret_cast<cpx<T> *>(S.out) + sf.off;
                if (S.op == BOP_FILL) {
                    const uint64_t seed = S.seed + (uint64_t)f;
                    for (int i = tid; i < TP; i += nthr) {
                        const int64_t e = e0 + i;
                        const uint64_t gi = (uint64_t)real_gidx(e, g);
                        double re, im;
                        if (S.kind == 0) {
                            re = u01(seed, gi, 0) * 2.0 - 1.0;
                            im = u01(seed, gi, 1) * 2.0 - 1.0;
                        } else {
                            re = gauss(seed, gi, 0);
                            im = gauss(seed, gi, 1);
                        }
                        out[e] = {(T)re, (T)im};
                    }
                    continue;
                }
                const cpx<T> *in = reinterpret_cast<const cpx<T> *>(S.in) + sf.off;
                const cpx<T> *rhs = reinterpret_cast<const cpx<T> *>(S.aux) + sf.off;
                if (half) residual_tile<T, TP0 / 2>(g, S.a, in, rhs, out, e0, s, tid);
                else residual_tile<T, TP0>(g, S.a, in, rhs, out, e0, s, tid);
            }
            continue;
        }

        // axis-pass steps: tiles of TL lines, TL * N = nthr * EPT points (complex128 N = 32: the
        // field's 32 lines, half as many)
        for (int64_t tile = blockIdx.x; tile < bp.tiles; tile += gridDim.x) {
            __syncthreads();   // the previous tile is done with sf, the bases and s
            if (tid == 0) sf = bp.fields[field_of_tile(bp.fields, bp.nfields, tile)];
            __syncthreads();
            const Geom &g = sf.g;
            const int64_t l0 = (tile - sf.tile0) * sf.T;
            const bool xpass = S.op == BOP_X_FWD || S.op == BOP_X_INV;
            const Tile c = tile_begin(g, xpass ? PASS_X2 : PASS_Y2, l0, sf.T, s_abase, s_fbase, nthr, tid);
            __syncthreads();
            const cpx<T> *in = reinterpret_cast<const cpx<T> *>(S.in) + sf.off;
            cpx<T> *out = reinterpret_cast<cpx<T> *>(S.out) + sf.off;
            // slot permutation per column length (SwzX, zm_tile.cuh)
#define ZM_BT(LMC, ...)                                                                                \
    (g.logP == 1 ? batch_tile<T, EPT, LMC, __VA_ARGS__, 1>(S.op, S.scale != 0, S.a, sf, c, s, in, out, l0, nthr, tid) \
                 : batch_tile<T, EPT, LMC, __VA_ARGS__, 2>(S.op, S.scale != 0, S.a, sf, c, s, in, out, l0, nthr, tid))
            bool done = false;
            if constexpr (sizeof(T) == 4 && EPT == 16) {
                if (g.logVEC == 2 && (g.logP == 1 || g.logP == 2)) {
                    done = true;
                    switch (g.logM) {
                    case 4: ZM_BT(4, SwzX<4, 8, 4, 6, 0>); break;
                    case 5: ZM_BT(5, SwzX<3, 9, 7, 4, 6>); break;
                    case 6: ZM_BT(6, SwzX<3, 8, 0, 4, 10>); break;
                    case 7: ZM_BT(7, SwzX<3, 4, 10, 5, 8>); break;
                    case 8: ZM_BT(8, SwzX<4, 9, 4, 6, 10>); break;
                    case 9: ZM_BT(9, SwzX<3, 10, 0, 4, 6>); break;
                    case 10: ZM_BT(10, SwzX<3, 0, 0, 4, 0>); break;
                    default: done = false; break;
                    }
                }
            }
#undef ZM_BT
            if constexpr (sizeof(T) == 8) {
                if (g.n * g.n < kBatchThreads * EPT) {
                    done = true;
                    batch_tile<T, EPT / 2, 0, SwzNone>(S.op, S.scale != 0, S.a, sf, c, s, in, out, l0, nthr, tid);
                }
            }
            if (!done) batch_tile<T, EPT, 0, SwzNone>(S.op, S.scale != 0, S.a, sf, c, s, in, out, l0, nthr, tid);
        }
    }
}

template <typename T, int TP>
__device__ __noinline__ void fill_tile(const Geom &g, int kind, uint64_t seed, cpx<T> *out, int64_t e0, int tid) {
    for (int i = tid; i < TP; i += kBatchThreads) {
        const int64_t e = e0 + i;
        const uint64_t gi = (uint64_t)real_gidx(e, g);
        double re, im;
        if (kind == 0) {
            re = u01(seed, gi, 0) * 2.0 - 1.0;
            im = u01(seed, gi, 1) * 2.0 - 1.0;
        } else {
            re = gauss(seed, gi, 0);
            im = gauss(seed, gi, 1);
        }
        out[e] = {(T)re, (T)im};
    }
}

// The same steps on the axis tiles (zm_batch_axis.cuh): every tile is 4096 points, its field
// read from a table (the index of the CTA's next tile one tile ahead) instead of searched.
// Bound by the L1 data pipe (71 % of its cycles: tile exchanges and twiddle loads), DRAM at
// 50 %.  32 + 32 + 24 + 8 complex64 fields of N = 256 .. 2048, P = 2, forward / inverse:
// 986 / 884 -> 608 / 610 us at VEC = 4 (the split's compile-time tiles), 2221 / 2163 -> 608 /
// 609 us at VEC = 16 (its runtime-sized tiles); 29 complex128 fields of N = 128 .. 1024,
// P = 4: 237 / 233 -> 120 / 115 us (136 / 120 before odd steps walked back, walks_back).
template <typename T>
__global__ void __launch_bounds__(kBatchThreads, sizeof(T) == 4 ? 4 : 2) batch_axis_kernel(const BatchParams bp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<T> *s = reinterpret_cast<cpx<T> *>(smem_raw);
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
            const int fcur = fi;
            if ((unsigned)(tile + hop) < (unsigned)ntiles) fi = __ldg(bp.tile_field + tile + hop);
            const Geom &g = f.g;
            const int64_t sub = tile - f.tile0;   // of the field
            const cpx<T> *in = reinterpret_cast<const cpx<T> *>(S.in) + f.off;
            cpx<T> *out = reinterpret_cast<cpx<T> *>(S.out) + f.off;
            if (op == BOP_RESIDUAL) {
                residual_tile<T, TP>(g, S.a, in, reinterpret_cast<const cpx<T> *>(S.aux) + f.off, out, sub * TP, s,
                                     threadIdx.x);
                continue;
            }
            if (op == BOP_FILL) {
                fill_tile<T, TP>(g, S.kind, S.seed + (uint64_t)fcur, out, sub * TP, threadIdx.x);
                continue;
            }
            const bool xpass = op == BOP_X_FWD || op == BOP_X_INV;
            const int top = op == BOP_Y_POISSON ? ATILE_POISSON
                                                : (op == BOP_X_INV || op == BOP_Y_INV ? ATILE_INV : ATILE_FWD);
            const T sc = op == BOP_X_INV && S.scale ? (T)(1.0 / ((double)g.n * (double)g.n)) : T(1);
            __syncthreads();   // the previous tile is done with the shared memory
#define ZM_AT(LN)                                                                                             \
    case LN:                                                                                                  \
        batch_axis_tile<T, LN>(top, s, in, out, g, f.ax + (xpass ? 0 : 1), f.twx, xpass,                      \
                               sub << (kBatchTileLog - LN), sc, S.a);                                         \
        break;
            switch (g.logN) {
                ZM_AT(6) ZM_AT(7) ZM_AT(8) ZM_AT(9) ZM_AT(10) ZM_AT(11) ZM_AT(12)
            default: break;
            }
#undef ZM_AT
        }
    }
}

// kernel and dynamic shared memory of a call
enum BatchTiles : int { TILES_SPLIT = 0, TILES_AXIS = 1, TILES_EXACT = 2 };
struct BatchKernel {
    BatchFn fn;
    size_t smem;
};
static BatchKernel batch_kernel_of(int dtype, int tiles) {
    constexpr size_t slots = axis_slot((1 << kBatchTileLog) - 1) + 1;
    if (tiles == TILES_EXACT) return BatchKernel{batch_exact_fn(), slots * 8};
    if (tiles == TILES_AXIS) return dtype == 0 ? BatchKernel{batch_axis_kernel<double>, slots * 16}
                                : BatchKernel{batch_axis_kernel<float>, slots * 8};
    return dtype == 0 ? BatchKernel{batch_kernel<double, 8>, kBatchThreads * 8 * 16}
                      : BatchKernel{batch_kernel<float, 16>, kBatchThreads * 16 * 8};
}

static cudaError_t launch_batch(const BatchKernel &k, const BatchParams &bp, int grid, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(bp.bar, 0, 3 * sizeof(unsigned), st);   // arrivals, generation, abort
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kBatchThreads);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k.fn, bp);
    count_launch();
    return e;
}

// resident CTAs of the device (0 on error)
static int batch_grid(const BatchKernel &k, int device) {
    int per_sm = 0, sms = 0;
    const void *fn = reinterpret_cast<const void *>(k.fn);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBatchThreads, k.smem) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    return per_sm * sms;
}

}  // namespace zm

// ================================================================== C ABI

struct zm_batch_s {
    int dtype;
    int device;
    int grid;
    std::vector<zm_plan> plans;            // distinct (N, B, P) plans (twiddle tables)
    std::vector<zm::BatchField> fields;    // host copy
    std::vector<int> field_plan;
    zm::BatchField *d_fields = nullptr;
    bool axis = false;                     // every field fits the axis tiles (zm_batch_axis.cuh)
    bool exact = false;                    // every field fits the tiles of zm_batch_exact.cu
    int axis_grid = 0, exact_grid = 0;
    int64_t axis_tiles = 0;
    const zm::BatchField *axis_fields = nullptr;   // the fields as the axis tiles count them
    const int *tile_field = nullptr;
    unsigned *d_sync = nullptr;            // [0..1] barrier, [2] abort (per launch), [3] sticky error flag
    int64_t tiles = 0, elems = 0;
};

namespace {

bool aligned16b(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_batch(zm_batch b) {
    if (!b) return zm::report_error(ZM_ERR_INVALID_ARG, "null batch");
    return ZM_OK;
}

int check_buf(const void *p, const char *name) {
    if (!p) return zm::report_error(ZM_ERR_INVALID_ARG, "%s is NULL", name);
    if (!aligned16b(p)) return zm::report_error(ZM_ERR_MISALIGNED, "%s is not 16-byte aligned", name);
    return ZM_OK;
}

bool overlap_b(const void *a, const void *b, size_t bytes) {
    const char *x = static_cast<const char *>(a), *y = static_cast<const char *>(b);
    return x < y + bytes && y < x + bytes;
}

// `tiles`: the kernel asked for; batches whose fields do not all fit it run the split tiles
int launch(zm_batch b, const zm::BatchStep *steps, int nsteps, void *stream, int tiles, unsigned missing = 0) {
    if ((tiles == zm::TILES_AXIS && !b->axis) || (tiles == zm::TILES_EXACT && !b->exact)) tiles = zm::TILES_SPLIT;
    const bool split = tiles == zm::TILES_SPLIT;
    zm::BatchParams bp = {};
    bp.missing = missing;
    bp.fields = split ? b->d_fields : b->axis_fields;
    bp.tile_field = b->tile_field;
    bp.nfields = (int)b->fields.size();
    bp.tiles = split ? b->tiles : b->axis_tiles;
    bp.nsteps = nsteps;
    for (int i = 0; i < nsteps; i++) bp.step[i] = steps[i];
    bp.bar = b->d_sync;
    bp.abort = reinterpret_cast<int *>(b->d_sync + 2);
    bp.err = reinterpret_cast<int *>(b->d_sync + 3);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int grid = split ? b->grid : tiles == zm::TILES_EXACT ? b->exact_grid : b->axis_grid;
    cudaError_t e = zm::launch_batch(zm::batch_kernel_of(b->dtype, tiles), bp, grid, st);
    if (e != cudaSuccess)
        return zm::report_error(ZM_ERR_CUDA, "batch launch: %s (%s)", cudaGetErrorName(e), cudaGetErrorString(e));
    return ZM_OK;
}

// The device tables of a batch in one allocation and one copy: the fields, and for the axis
// tiles their own field records, weight tables per plan, stage twiddles per N and the
// tile -> field table.
int device_tables(zm_batch b) {
    const size_t nf = b->fields.size();
    std::vector<unsigned char> blob(sizeof(zm::BatchField) * nf);
    auto reserve = [&blob](size_t bytes) {
        const size_t at = (blob.size() + 15) & ~size_t{15};
        blob.resize(at + bytes);
        return at;
    };
    size_t af_at = 0, tf_at = 0;
    std::vector<zm::BatchField> af;
    std::vector<size_t> map_at(b->plans.size()), tw_at(b->plans.size());
    std::vector<std::array<size_t, 3>> ex_at(b->plans.size());   // exact tiles: tables, forward and inverse twiddles
    if (b->axis) {
        std::map<int, size_t> tw_of;   // log2 N -> stage twiddles
        for (size_t i = 0; i < b->plans.size(); i++) {
            const zm::Geom &g = b->plans[i]->g;
            const int ltl = zm::kBatchTileLog - g.logN, lg = std::min(ltl, 3);
            const std::vector<int> lrs = zm::axis_digits(g.logN, 4);
            const zm::AxisMap maps[2] = {zm::axis_map(g, zm::PASS_X2, b->dtype, ltl, zm::kBatchPtsLog, lrs, lg),
                                         zm::axis_map(g, zm::PASS_Y2, b->dtype, ltl, zm::kBatchPtsLog, lrs, lg)};
            map_at[i] = reserve(sizeof maps);
            std::memcpy(&blob[map_at[i]], maps, sizeof maps);
            if (!tw_of.count(g.logN)) {
                std::vector<int64_t> exps;
                zm::axis_twiddles(g, lrs, &exps);
                tw_of[g.logN] = reserve(exps.size() * 16);
                zm::twiddle_entries(b->plans[i]->roots, b->dtype, exps, &blob[tw_of[g.logN]]);
            }
            tw_at[i] = tw_of[g.logN];
            if (!b->exact) continue;
            const std::vector<int> df = zm::batch_exact_digits(g, false), di = zm::batch_exact_digits(g, true);
            const zm::AxisMap ex[3] = {zm::axis_map(g, zm::PASS_X2, b->dtype, ltl, zm::kBatchPtsLog, df, lg),
                                       zm::axis_map(g, zm::PASS_Y2, b->dtype, ltl, zm::kBatchPtsLog, df, lg),
                                       zm::axis_map(g, zm::PASS_X2, b->dtype, ltl, zm::kBatchPtsLog, di, lg)};
            ex_at[i][0] = reserve(sizeof ex);
            std::memcpy(&blob[ex_at[i][0]], ex, sizeof ex);
            for (int inv = 0; inv < 2; inv++) {
                std::vector<int64_t> exps;
                zm::batch_exact_twiddles(g, inv, &exps);
                ex_at[i][1 + inv] = reserve(exps.size() * 16);
                zm::twiddle_entries(b->plans[i]->roots, b->dtype, exps, &blob[ex_at[i][1 + inv]]);
            }
        }
        std::vector<int> tf;
        af = b->fields;
        for (size_t i = 0; i < nf; i++) {
            af[i].T = (1 << zm::kBatchTileLog) / (int)af[i].g.n;
            af[i].tile0 = (int64_t)tf.size();
            tf.insert(tf.end(), (size_t)(af[i].g.n / af[i].T), (int)i);
        }
        b->axis_tiles = (int64_t)tf.size();
        af_at = reserve(sizeof(zm::BatchField) * nf);
        tf_at = reserve(tf.size() * sizeof(int));
        std::memcpy(&blob[tf_at], tf.data(), tf.size() * sizeof(int));
    }
    cudaError_t e = cudaMalloc(&b->d_fields, blob.size());
    if (e != cudaSuccess) return zm::report_error(ZM_ERR_NO_MEMORY, "batch tables: %s", cudaGetErrorString(e));
    unsigned char *d = reinterpret_cast<unsigned char *>(b->d_fields);
    std::memcpy(blob.data(), b->fields.data(), sizeof(zm::BatchField) * nf);
    if (b->axis) {
        for (size_t i = 0; i < nf; i++) {
            af[i].ax = reinterpret_cast<const zm::AxisMap *>(d + map_at[b->field_plan[i]]);
            af[i].twx = d + tw_at[b->field_plan[i]];
            const std::array<size_t, 3> &e = ex_at[b->field_plan[i]];
            af[i].ex = b->exact ? reinterpret_cast<const zm::AxisMap *>(d + e[0]) : nullptr;
            af[i].exf = b->exact ? d + e[1] : nullptr;
            af[i].exi = b->exact ? d + e[2] : nullptr;
        }
        std::memcpy(&blob[af_at], af.data(), sizeof(zm::BatchField) * nf);
        b->axis_fields = reinterpret_cast<const zm::BatchField *>(d + af_at);
        b->tile_field = reinterpret_cast<const int *>(d + tf_at);
    }
    e = cudaMemcpy(d, blob.data(), blob.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return zm::report_error(ZM_ERR_NO_MEMORY, "batch tables: %s", cudaGetErrorString(e));
    return ZM_OK;
}

size_t batch_bytes(zm_batch b) { return (size_t)b->elems * (b->dtype == ZM_C128 ? 16 : 8); }

}  // namespace

extern "C" {

int zm_batch_create(zm_batch *batch, int nfields, const int64_t *n, const int64_t *b, const int64_t *p,
                    int dtype) {
    if (!batch) return zm::report_error(ZM_ERR_INVALID_ARG, "batch output pointer is NULL");
    *batch = nullptr;
    if (nfields < 1 || nfields > 65536) return zm::report_error(ZM_ERR_INVALID_ARG, "nfields=%d out of range [1, 65536]", nfields);
    if (!n || !b || !p) return zm::report_error(ZM_ERR_INVALID_ARG, "n, b and p must not be NULL");
    if (dtype != ZM_C128 && dtype != ZM_C64) return zm::report_error(ZM_ERR_INVALID_ARG, "unknown dtype %d", dtype);
    const int ept = zm::ept_for(dtype);
    const int64_t tile_pts = (int64_t)zm::kBatchThreads * ept;
    zm_batch_s *B = new (std::nothrow) zm_batch_s();
    if (!B) return zm::report_error(ZM_ERR_NO_MEMORY, "host allocation failed");
    B->dtype = dtype;
    cudaGetDevice(&B->device);
    std::map<std::tuple<int64_t, int64_t, int64_t>, int> seen;
    int rc = ZM_OK;
    // an axis tile is 4096 points of one field: N = 64 and up
    B->axis = true;
    for (int i = 0; i < nfields; i++) B->axis = B->axis && n[i] >= 64;
    B->exact = B->axis && dtype == ZM_C64;
    for (int i = 0; i < nfields && rc == ZM_OK; i++) {
        if (n[i] < tile_pts / 64 || n[i] > tile_pts) {
            rc = zm::report_error(ZM_ERR_CONSTRAINT, "field %d: N=%lld outside the batch range [%lld, %lld]", i,
                                  (long long)n[i], (long long)(tile_pts / 64), (long long)tile_pts);
            break;
        }
        const auto key = std::make_tuple(n[i], b[i], p[i]);
        auto it = seen.find(key);
        int pi;
        if (it == seen.end()) {
            zm_plan pl = nullptr;
            rc = zm_plan_create(&pl, 2, n[i], b[i], p[i], dtype, 0);
            if (rc != ZM_OK) break;
            pi = (int)B->plans.size();
            B->plans.push_back(pl);
            seen.emplace(key, pi);
        } else {
            pi = it->second;
        }
        const zm_plan_s *pl = B->plans[pi];
        B->exact = B->exact && zm::batch_exact_fits(pl->g);
        zm::BatchField f = {};
        f.g = pl->g;
        f.off = B->elems;
        f.tile0 = B->tiles;
        f.twN = pl->twN;
        f.T = (int)std::min(tile_pts / n[i], n[i]);   // complex128 N = 32 has half a tile's points
        const int fept = (int)(f.T * n[i] / zm::kBatchThreads);   // points per thread, the largest radix
        f.nst_vec = zm::radix_schedule(pl->g.vec, fept, f.rad_vec);
        f.nst_m = zm::radix_schedule(pl->g.m, fept, f.rad_m);
        B->fields.push_back(f);
        B->field_plan.push_back(pi);
        B->elems += (n[i] * n[i] + 1) & ~int64_t{1};
        B->tiles += n[i] / f.T;
    }
    if (rc == ZM_OK) {
        B->grid = zm::batch_grid(zm::batch_kernel_of(dtype, zm::TILES_SPLIT), B->device);
        if (B->axis) B->axis_grid = zm::batch_grid(zm::batch_kernel_of(dtype, zm::TILES_AXIS), B->device);
        if (B->exact) B->exact_grid = zm::batch_grid(zm::batch_kernel_of(dtype, zm::TILES_EXACT), B->device);
        if (B->grid <= 0 || (B->axis && B->axis_grid <= 0) || (B->exact && B->exact_grid <= 0))
            rc = zm::report_error(ZM_ERR_CUDA, "batch kernel occupancy query failed");
    }
    if (rc == ZM_OK) rc = device_tables(B);
    if (rc == ZM_OK) {
        cudaError_t e = cudaMalloc(&B->d_sync, 4 * sizeof(unsigned));
        if (e == cudaSuccess) e = cudaMemset(B->d_sync, 0, 4 * sizeof(unsigned));
        if (e != cudaSuccess)
            rc = zm::report_error(ZM_ERR_NO_MEMORY, "batch tables: %s", cudaGetErrorString(e));
    }
    if (rc != ZM_OK) {
        zm_batch_destroy(B);
        return rc;
    }
    *batch = B;
    return ZM_OK;
}

int zm_batch_destroy(zm_batch batch) {
    int rc;
    if ((rc = check_batch(batch))) return rc;
    for (zm_plan pl : batch->plans) zm_plan_destroy(pl);
    if (batch->d_fields) cudaFree(batch->d_fields);
    if (batch->d_sync) cudaFree(batch->d_sync);
    delete batch;
    return ZM_OK;
}

int zm_batch_get_field(zm_batch batch, int i, zm_batch_field *info) {
    int rc;
    if ((rc = check_batch(batch))) return rc;
    if (!info) return zm::report_error(ZM_ERR_INVALID_ARG, "info is NULL");
    if (i < 0 || i >= (int)batch->fields.size()) return zm::report_error(ZM_ERR_INVALID_ARG, "field %d out of range", i);
    const zm::BatchField &f = batch->fields[i];
    info->n = f.g.n;
    info->b = f.g.b;
    info->p = f.g.p;
    info->offset = f.off;
    info->elems = f.g.n * f.g.n;
    return ZM_OK;
}

int zm_batch_total_elems(zm_batch batch, int64_t *elems) {
    int rc;
    if ((rc = check_batch(batch))) return rc;
    if (!elems) return zm::report_error(ZM_ERR_INVALID_ARG, "elems is NULL");
    *elems = batch->elems;
    return ZM_OK;
}

int zm_batch_fill(zm_batch batch, void *data, int kind, uint64_t first_seed, void *stream) {
    int rc;
    if ((rc = check_batch(batch)) || (rc = check_buf(data, "data"))) return rc;
    if (kind != ZM_FIELD_UNIFORM && kind != ZM_FIELD_GAUSSIAN) return zm::report_error(ZM_ERR_INVALID_ARG, "unknown kind %d", kind);
    zm::BatchStep s = {};
    s.op = zm::BOP_FILL;
    s.kind = kind;
    s.out = data;
    s.seed = first_seed;
    return launch(batch, &s, 1, stream, zm::TILES_AXIS);
}

int zm_batch_forward(zm_batch batch, const void *in, void *out, void *stream) {
    int rc;
    if ((rc = check_batch(batch)) || (rc = check_buf(in, "in")) || (rc = check_buf(out, "out"))) return rc;
    if (overlap_b(in, out, batch_bytes(batch))) return zm::report_error(ZM_ERR_INVALID_ARG, "in and out overlap");
    zm::BatchStep s[2] = {};
    s[0].op = zm::BOP_X_FWD; s[0].in = in; s[0].out = out;
    s[1].op = zm::BOP_Y_FWD; s[1].in = out; s[1].out = out;
    return launch(batch, s, 2, stream, zm::TILES_AXIS);
}

int zm_batch_inverse(zm_batch batch, const void *in, void *out, void *work, int normalise, void *stream) {
    int rc;
    if ((rc = check_batch(batch)) || (rc = check_buf(in, "in")) || (rc = check_buf(out, "out"))) return rc;
    const size_t F = batch_bytes(batch);
    if (overlap_b(in, out, F)) return zm::report_error(ZM_ERR_INVALID_ARG, "in and out overlap");
    if (work) {
        if ((rc = check_buf(work, "work"))) return rc;
        if (overlap_b(work, in, F) || overlap_b(work, out, F))
            return zm::report_error(ZM_ERR_INVALID_ARG, "work overlaps in/out");
    }
    void *tmp = work ? work : const_cast<void *>(in);
    zm::BatchStep s[2] = {};
    s[0].op = zm::BOP_Y_INV; s[0].in = in; s[0].out = tmp;
    s[1].op = zm::BOP_X_INV; s[1].in = tmp; s[1].out = out; s[1].scale = normalise ? 1 : 0;
    return launch(batch, s, 2, stream, zm::TILES_AXIS);
}

int zm_batch_poisson(zm_batch batch, const void *rhs, void *phi, void *residual, void *work, double length,
                     void *stream) {
    int rc;
    if ((rc = check_batch(batch)) || (rc = check_buf(rhs, "rhs")) || (rc = check_buf(phi, "phi")) ||
        (rc = check_buf(work, "work")))
        return rc;
    if (residual && (rc = check_buf(residual, "residual"))) return rc;
    if (!(length > 0.0) || !std::isfinite(length)) return zm::report_error(ZM_ERR_INVALID_ARG, "length must be positive");
    const size_t F = batch_bytes(batch);
    if (overlap_b(rhs, phi, F) || overlap_b(rhs, work, F) || overlap_b(phi, work, F) ||
        (residual && (overlap_b(residual, rhs, F) || overlap_b(residual, phi, F) || overlap_b(residual, work, F))))
        return zm::report_error(ZM_ERR_INVALID_ARG, "rhs, phi, residual and work must not overlap");
    zm::BatchStep s[4] = {};
    const double two_pi = 6.283185307179586476925286766559;
    s[0].op = zm::BOP_X_FWD; s[0].in = rhs; s[0].out = work;
    s[1].op = zm::BOP_Y_POISSON; s[1].in = work; s[1].out = work; s[1].a = two_pi / length;
    s[2].op = zm::BOP_X_INV; s[2].in = work; s[2].out = phi; s[2].scale = 1;
    int ns = 3;
    if (residual) {
        s[3].op = zm::BOP_RESIDUAL; s[3].in = phi; s[3].aux = rhs; s[3].out = residual; s[3].a = 1.0 / length;
        ns = 4;
    }
    // The complex64 residual is a difference of nearly equal terms: it amplifies phi's
    // rounding by about 8 N / (2 pi)^2 (2e-5 of the residual at N = 256, 2e-4 at 2048), so
    // another order of the transforms' operations is another residual field.  Complex64 calls
    // keep the rounding of the VEC x M split, on its own tiles (zm_batch_exact.cu) or, for
    // fields that these do not hold, on batch_kernel; without a residual as well, so that phi
    // does not depend on whether the residual is asked for.
    return launch(batch, s, ns, stream, batch->dtype == ZM_C128 ? zm::TILES_AXIS : zm::TILES_EXACT);
}

int zm_batch_status(zm_batch batch, int *device_error) {
    int rc;
    if ((rc = check_batch(batch))) return rc;
    if (!device_error) return zm::report_error(ZM_ERR_INVALID_ARG, "device_error is NULL");
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess)
        return zm::report_error(ZM_ERR_CUDA, "batch status: %s (%s)", cudaGetErrorName(e), cudaGetErrorString(e));
    int flag = 0;
    e = cudaMemcpy(&flag, batch->d_sync + 3, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && flag) e = cudaMemset(batch->d_sync, 0, 4 * sizeof(unsigned));
    if (e != cudaSuccess)
        return zm::report_error(ZM_ERR_CUDA, "batch status: %s (%s)", cudaGetErrorName(e), cudaGetErrorString(e));
    *device_error = flag ? 1 : 0;
    return ZM_OK;
}

int zm_batch_barrier_probe(zm_batch batch, int missing, void *stream) {
    int rc;
    if ((rc = check_batch(batch))) return rc;
    if (missing < 0 || missing > 1) return zm::report_error(ZM_ERR_INVALID_ARG, "missing must be 0 or 1");
    zm::BatchStep s[2] = {};
    s[0].op = zm::BOP_NOP;
    s[1].op = zm::BOP_NOP;
    // the kernels that this batch's calls launch: one, and for complex64 the Poisson call's
    if ((rc = launch(batch, s, 2, stream, zm::TILES_AXIS, (unsigned)missing)) || batch->dtype == ZM_C128) return rc;
    return launch(batch, s, 2, stream, zm::TILES_EXACT, (unsigned)missing);
}

int zm_batch_autotune_b(int64_t n, int64_t p, int dtype, int count, int reps, int64_t *best_b, float *best_ms) {
    if (count < 1 || reps < 1) return zm::report_error(ZM_ERR_INVALID_ARG, "count and reps must be >= 1");
    if (n <= 0 || p <= 0 || (n & (n - 1)) || (p & (p - 1)) || n % p)
        return zm::report_error(ZM_ERR_CONSTRAINT, "N and P must be powers of two with P | N");
    const int64_t L = n / p;
    int64_t best = 0;
    float best_t = 0.f;
    int rc = ZM_OK;
    for (int64_t b = 1; b <= L / p && rc == ZM_OK; b *= 2) {
        std::vector<int64_t> nv(count, n), bv(count, b), pv(count, p);
        zm_batch bt = nullptr;
        if (zm_batch_create(&bt, count, nv.data(), bv.data(), pv.data(), dtype) != ZM_OK) continue;   // B not allowed
        const size_t F = batch_bytes(bt);
        void *buf = nullptr;
        cudaError_t e = cudaMalloc(&buf, 4 * F);
        if (e != cudaSuccess) {
            zm_batch_destroy(bt);
            rc = zm::report_error(ZM_ERR_NO_MEMORY, "autotune buffers: %s", cudaGetErrorString(e));
            break;
        }
        char *c = static_cast<char *>(buf);
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        rc = zm_batch_fill(bt, c, ZM_FIELD_GAUSSIAN, 1, nullptr);
        for (int it = -1; it < reps && rc == ZM_OK; it++) {
            if (it == 0) cudaEventRecord(e0, nullptr);
            rc = zm_batch_poisson(bt, c, c + F, c + 2 * F, c + 3 * F, 1.0, nullptr);
        }
        cudaEventRecord(e1, nullptr);
        int flag = 0;
        if (rc == ZM_OK && (e = cudaEventSynchronize(e1)) != cudaSuccess)
            rc = zm::report_error(ZM_ERR_CUDA, "autotune timing: %s", cudaGetErrorString(e));
        if (rc == ZM_OK) rc = zm_batch_status(bt, &flag);
        if (rc == ZM_OK && flag) rc = zm::report_error(ZM_ERR_TIMEOUT, "autotune: batch barrier timed out");
        if (rc == ZM_OK) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            ms /= (float)reps;
            if (best == 0 || ms < best_t) {
                best = b;
                best_t = ms;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaFree(buf);
        zm_batch_destroy(bt);
    }
    if (rc != ZM_OK) return rc;
    if (best == 0) return zm::report_error(ZM_ERR_CONSTRAINT, "no B is valid for N=%lld", (long long)n);
    if (best_b) *best_b = best;
    if (best_ms) *best_ms = best_t;
    return ZM_OK;
}

}  // extern "C"
