// axis_map_check.cu -- host check of the axis pass' weight tables (zm_axis.cu): for every
// layout and tile shape, each (thread, register) of a tile must land on the element that the
// general address formula (line_addr and the chunk / position split) gives for its slot, the
// tile must be covered once, and complex64 pairs must start on 16 bytes.
#include <cstdio>
#include <vector>

#include "zm_axis.cu"

namespace zm {
void count_launch() {}
cudaError_t launch_axis_c64_fwd(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c64_inv(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c128_fwd(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c128_inv(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
}  // namespace zm
using namespace zm;

static long bad = 0, checks = 0;

static Geom geom(int dim, int ln, int lb, int lp) {
    Geom g;
    g.dim = dim;
    g.logN = ln; g.logB = lb; g.logP = lp;
    g.logL = ln - lp; g.logVEC = ln - lp - lb; g.logVP = g.logVEC - lp; g.logM = lb + lp;
    g.n = int64_t{1} << ln; g.b = int64_t{1} << lb; g.p = int64_t{1} << lp; g.L = int64_t{1} << g.logL;
    g.vec = int64_t{1} << g.logVEC; g.vp = int64_t{1} << g.logVP; g.m = int64_t{1} << g.logM;
    return g;
}

static void check(const Geom &g, int dtype, int kind, int ltl, int lp, int le, int lg) {
    const int ln = g.logN, lnt = ln + ltl - lp, nst = axis_stages(ln, le), lr = axis_lr(ln, le, nst - 1);
    const int64_t total = g.dim == 2 ? g.n * g.n : g.n * g.n * g.n, nblk = (total >> ln) >> ltl;
    const AxisMap m = axis_map(g, kind, dtype, ltl, lp, axis_digits(g.logN, le), lg);
    const int E = 1 << (ln + ltl);
    std::vector<int> index(axis_slot(E - 1) + 1, -1);
    for (int i = 0; i < E; i++) index[axis_slot(i)] = i;
    if (m.lg > lg || (int64_t{1} << m.lg) > g.L) bad++;
    const int64_t step = nblk > 5 ? (nblk / 5) | 1 : 1;
    for (int64_t blk = 0; blk < nblk; blk += step) {
        const LineAddr la = line_addr(g, kind, blk << ltl, m.lg);
        std::vector<char> seen_a(E, 0), seen_f(E, 0);
        auto slot_index = [&](int s) { return s >= 0 && s < (int)index.size() ? index[s] : -1; };
        for (int tid = 0; tid < 1 << lnt; tid++)
            for (int r = 0; r < 1 << lp; r++, checks++) {
                int64_t a = la.a_base, f = la.f_base;
                int sa = 0, sf = 0;
                for (int q = 0; q < lnt; q++)
                    if (tid >> q & 1) a += m.va[q], sa += m.vs[q], f += m.fa[q], sf += m.fs[q];
                for (int q = 0; q < lp; q++)
                    if (r >> q & 1) a += m.va[lnt + q], sa += m.vs[lnt + q];
                const int u = r >> lr, rr = r & ((1 << lr) - 1);
                for (int q = 0; q < lp - lr; q++)
                    if (u >> q & 1) f += m.fa[lnt + q], sf += m.fs[lnt + q];
                for (int q = 0; q < lr; q++)
                    if (rr >> q & 1) f += m.fr[q];
                sf += axis_slot(rr << ltl);
                const int ia = slot_index(sa), jf = slot_index(sf);
                if (ia < 0 || jf < 0 || seen_a[ia] || seen_f[jf]) { bad++; continue; }
                seen_a[ia] = seen_f[jf] = 1;
                if (dtype != 0 && r % 2 == 0 && (a & 1)) bad++;
                // vector side
                LineAddr l = line_addr(g, kind, (blk << ltl) + (ia & ((1 << ltl) - 1)), m.lg);
                const int64_t n = ia >> ltl, n1 = n & (g.m - 1), n2 = n >> g.logM;
                const int64_t ra = l.a_base + (n1 >> g.logB) * l.a_chunk + ((n1 & (g.b - 1)) * g.vec + n2) * l.a_hi;
                // frequency side: digits of the index, lowest digit of k first
                int64_t k = 0;
                for (int q = 0, o = 0; q < nst; o += axis_lr(ln, le, q), q++)
                    k |= (int64_t)((jf >> ltl >> axis_sh(ln, le, q)) & ((1 << axis_lr(ln, le, q)) - 1)) << o;
                l = line_addr(g, kind, (blk << ltl) + (jf & ((1 << ltl) - 1)), m.lg);
                const int64_t k1 = k >> g.logVEC, k2 = k & (g.vec - 1), pos = k1 * g.vp + (k2 & (g.vp - 1));
                const int64_t fo = l.f_lg ? (pos >> l.f_lg) * l.f_hi + (pos & ((1 << l.f_lg) - 1)) : pos * l.f_pos;
                const int64_t rf = l.f_base + (k2 >> g.logVP) * l.f_chunk + fo;
                if (ra != a || rf != f || a < 0 || a >= total || f < 0 || f >= total) bad++;
            }
        for (int i = 0; i < E; i++) bad += !seen_a[i] + !seen_f[i];
    }
}

int main() {
    for (int dtype = 0; dtype < 2; dtype++)
        for (int dim = 2; dim <= 3; dim++)
            for (int ln = 4; ln <= (dim == 2 ? 14 : 8); ln++)
                for (int lp = 0; lp <= 3 && 2 * lp <= ln; lp++)
                    for (int lb = 0; lb <= ln - 2 * lp; lb += ln > 9 ? 2 : 1) {
                        const Geom g = geom(dim, ln, lb, lp);
                        const int kinds[2][3] = {{PASS_X2, PASS_Y2, PASS_Y2}, {PASS_X3, PASS_Y3, PASS_Z3}};
                        const int64_t nlines = int64_t{1} << (dim - 1) * ln;
#define ZM_CHECK(LN, LTL, LP, LE) \
    if (LN == ln && (nlines >> LTL) >= 1)  \
        for (int a = 0; a < dim; a++)          \
            for (int lg = 0; lg <= (dim == 2 ? 4 : 0); lg++) check(g, dtype, kinds[dim - 2][a], LTL, LP, LE, lg);
                        if (dtype == 0) { ZM_AXIS_TILES_C128(ZM_CHECK) } else { ZM_AXIS_TILES_C64(ZM_CHECK) }
                        // the tile that plans take exists and fits the field
                        int ltl = -1, pts = -1, le = -1;
                        const bool any = axis_tile(g, dtype, nlines << ln, &ltl, &pts, &le);
                        const bool own = (g.logVEC == 6 && g.logM == 8) || (dtype == 0 && ln > 13);
                        if (any == own || (any && (nlines >> ltl) < 1)) bad++;
                    }
    std::printf("%ld mismatches in %ld points\n", bad, checks);
    return bad != 0;
}
