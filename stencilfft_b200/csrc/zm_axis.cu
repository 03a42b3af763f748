// zm_axis.cu -- host side of the axis pass sized by N alone (zm_axis.cuh): tile shapes,
// weight tables and twiddle order.
#include <string.h>

#include <algorithm>
#include <cmath>

#include "zm_axis.cuh"
#include "zm_axis_tiles.h"

namespace zm {

// The tile of a plan's passes, or false when the other kernels run it.
bool axis_tile(const Geom &g, int dtype, int64_t total, int *ltl, int *lp, int *le) {
    // element offsets inside a tile are 32-bit (3D N = 2048 complex64, the one larger field that
    // a GPU holds twice, takes the VEC x M pass at VEC = 32: forward / inverse 158 / 126 ms,
    // 283 / 283 on the runtime-sized pass of its other layouts)
    if (total >= int64_t{1} << 31) return false;
    // complex64 / complex128 lines of 2^14 points at VEC = 64, M = 256 have passes of their
    // own (zm_fft3.cuh and the tensor-memory-staged tiles of zm_fft2.cuh)
    if (g.logVEC == 6 && g.logM == 8) return false;
    const int64_t nlines = total >> g.logN;
    bool found = false;
    // wide tiles when they fill the chip's 148 SMs about three times over, else the last
    // (narrowest) one listed that the field has lines for
    auto take = [&](int ln, int tl, int pts, int e) {
        if (ln != g.logN || nlines < (int64_t{1} << tl)) return;
        if (found && (nlines >> *ltl) >= 512) return;
        found = true;
        *ltl = tl;
        *lp = pts;
        *le = e;
    };
#define ZM_TAKE(LN, LTL, LP, LE) take(LN, LTL, LP, LE);
    if (dtype == 0) { ZM_AXIS_TILES_C128(ZM_TAKE) } else { ZM_AXIS_TILES_C64(ZM_TAKE) }
#undef ZM_TAKE
    return found;
}

namespace {
struct Bit { int64_t a; int i; };   // address weight, index bit

// The lanes of a warp are the five lowest address bits, in an order that can trade the banks
// one phase of a shared-memory access falls on (its 2^phase lanes) for the 128-byte lines
// that the same lanes touch in global memory; ascending addresses on ties.
void order_lanes(std::vector<Bit> &v, int nthread, int phase, int banks, int line) {
    if (nthread < 5) return;
    int best = 0, best_cost = 1 << 30;
    for (int sub = 0; sub < 32; sub++) {
        if (__builtin_popcount(sub) != phase) continue;
        unsigned seen = 0;
        int lines = 1;
        for (int b = 0; b < 5; b++)
            if ((sub >> b & 1) && v[b].a >= line) lines *= 2;
        for (int l = sub;; l = (l - 1) & sub) {
            int slot = 0;
            for (int b = 0; b < 5; b++)
                if (l >> b & 1) slot += axis_slot(1 << v[b].i);
            seen |= 1u << (slot & (banks - 1));
            if (!l) break;
        }
        const int cost = banks / __builtin_popcount(seen) + lines;
        if (cost < best_cost) {
            best_cost = cost;
            best = sub;
        }
    }
    std::vector<Bit> o;
    for (int b = 0; b < 5; b++) if (best >> b & 1) o.push_back(v[b]);
    for (int b = 0; b < 5; b++) if (!(best >> b & 1)) o.push_back(v[b]);
    std::copy(o.begin(), o.end(), v.begin());
}
}  // namespace

// `lrs`: log2 radices of the digits, high to low
AxisMap axis_map(const Geom &g, int kind, int dtype, int ltl, int lp, const std::vector<int> &lrs, int lg) {
    AxisMap m;
    memset(&m, 0, sizeof m);
    m.ltl = ltl;
    m.lp = lp;
    m.le = *std::max_element(lrs.begin(), lrs.end());
    // complex64 moves 16-byte pairs of the vector side: its lowest address bit must lie in
    // the tile, which an interleave wider than the tile's lines would break
    if (dtype != 0) lg = std::min(lg, ltl);
    m.lg = g.dim == 2 ? std::min(lg, g.logL) : 0;
    const int ln = g.logN, lnt = ln + ltl - lp, nst = (int)lrs.size(), lr = lrs[nst - 1];
    const LineAddr z = line_addr(g, kind, 0, m.lg);
    std::vector<Bit> va, fa;
    for (int j = 0; j < ltl; j++) {
        const LineAddr q = line_addr(g, kind, int64_t{1} << j, m.lg);
        va.push_back({q.a_base - z.a_base, j});
        fa.push_back({q.f_base - z.f_base, j});
    }
    for (int b = 0; b < ln; b++) {   // n = n2 M + n1, n1 = c B + j, position j VEC + n2 of chunk c
        int64_t w;
        if (b >= g.logM) w = z.a_hi << (b - g.logM);
        else if (b < g.logB) w = z.a_hi << (b + g.logVEC);
        else w = z.a_chunk << (b - g.logB);
        va.push_back({w, ltl + b});
    }
    std::vector<int64_t> digit;
    for (int b = 0; b < ln; b++) {   // k = k1 VEC + c VP + f, position k1 VP + f of chunk c
        int64_t w, pos = -1;
        if (b < g.logVP) pos = int64_t{1} << b;
        else if (b >= g.logVEC) pos = int64_t{1} << (b - g.logVEC + g.logVP);
        if (pos < 0) w = z.f_chunk << (b - g.logVP);
        else if (z.f_lg && pos < (int64_t{1} << z.f_lg)) w = pos;
        else w = z.f_lg ? (pos >> z.f_lg) * z.f_hi : pos * z.f_pos;
        // k bit -> index bit: stage s holds k bits [o, o + lr_s) at i bits [sh_s, ...)
        int o = 0, s = 0;
        while (b >= o + lrs[s]) o += lrs[s++];
        if (s == nst - 1) digit.push_back(w);
        else fa.push_back({w, ltl + (ln - o - lrs[s]) + b - o});
    }
    auto by_addr = [](const Bit &x, const Bit &y) { return x.a < y.a; };
    std::sort(va.begin(), va.end(), by_addr);
    std::sort(fa.begin(), fa.end(), by_addr);
    const int phase = dtype == 0 ? 3 : 4, banks = dtype == 0 ? 8 : 16;
    if (dtype != 0) {   // lowest address bit to register bit 0 (behind the thread bits)
        std::rotate(va.begin(), va.begin() + 1, va.begin() + 1 + lnt);
    }
    const int line = dtype == 0 ? 8 : 16;   // elements per 128 bytes
    order_lanes(va, lnt, phase, banks, line);
    order_lanes(fa, lnt, phase, banks, line);
    for (size_t q = 0; q < va.size(); q++) {
        m.va[q] = (int)va[q].a;
        m.vs[q] = axis_slot(1 << va[q].i);
    }
    for (size_t q = 0; q < fa.size(); q++) {
        m.fa[q] = (int)fa[q].a;
        m.fs[q] = axis_slot(1 << fa[q].i);
    }
    for (int q = 0; q < lr; q++) m.fr[q] = (int)digit[q];
    return m;
}

std::vector<int> axis_digits(int ln, int le) {
    std::vector<int> lrs;
    for (int s = 0; s < axis_stages(ln, le); s++) lrs.push_back(axis_lr(ln, le, s));
    return lrs;
}

// exponent e of every table entry (w_N^e): stage s, row k, column v -> w_{N_s}^{k v}
void axis_twiddles(const Geom &g, const std::vector<int> &lrs, std::vector<int64_t> *exps) {
    int sh = g.logN;
    for (size_t s = 0; s + 1 < lrs.size(); s++) {
        const int ln = g.logN, lr = lrs[s];
        sh -= lr;
        for (int64_t k = 0; k < 1 << lr; k++)
            for (int64_t v = 0; v < 1 << sh; v++)
                exps->push_back(((k * v) << (ln - lr - sh)) & (g.n - 1));
    }
}

void unit_roots(int64_t n, double *w) {
    const long double pi = 3.141592653589793238462643383279502884L;
    for (int64_t m = 0; m < n; m++) {
        const long double th = -2.0L * pi * (long double)m / (long double)n;
        w[2 * m] = (double)cosl(th);
        w[2 * m + 1] = (double)sinl(th);
    }
}

void twiddle_store(int dtype, double c, double s, void *at) {
    if (dtype == 0) {
        const double d[2] = {c, s};
        memcpy(at, d, 16);
    } else {
        const float ch = (float)c, sh = (float)s;
        const float f[4] = {ch, sh, (float)(c - (double)ch), (float)(s - (double)sh)};
        memcpy(at, f, 16);
    }
}

void twiddle_entries(const std::vector<double> &w, int dtype, const std::vector<int64_t> &exps, void *out) {
    for (size_t i = 0; i < exps.size(); i++)
        twiddle_store(dtype, w[2 * exps[i]], w[2 * exps[i] + 1], static_cast<unsigned char *>(out) + 16 * i);
}

cudaError_t launch_axis_pass(const AxisParams &p, int dtype, bool inv, int64_t nlines, cudaStream_t st) {
    if (dtype == 0) return inv ? launch_axis_c128_inv(p, nlines, st) : launch_axis_c128_fwd(p, nlines, st);
    return inv ? launch_axis_c64_inv(p, nlines, st) : launch_axis_c64_fwd(p, nlines, st);
}

}  // namespace zm
