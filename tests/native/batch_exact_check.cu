// batch_exact_check.cu -- host check of the split-digit tiles (zm_batch_exact.cu): their stage
// tables and digit orders, run in FP64 on the host, are the DFT and its inverse, and the weight
// tables of both digit orders land on the general addresses.
#include <cmath>
#include <complex>
#include <cstdio>
#include <vector>

#include "zm_axis.cu"
#include "zm_batch_exact.cu"

namespace zm {
void count_launch() {}
cudaError_t launch_axis_c64_fwd(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c64_inv(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c128_fwd(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_axis_c128_inv(const AxisParams &, int64_t, cudaStream_t) { return cudaSuccess; }
}  // namespace zm
using namespace zm;
using Z = std::complex<double>;

static double worst = 0;
static long bad = 0;

static Geom geom(int ln, int lv, int lp) {
    Geom g;
    g.dim = 2;
    g.logN = ln; g.logP = lp; g.logVEC = lv; g.logL = ln - lp; g.logB = g.logL - lv; g.logVP = lv - lp; g.logM = ln - lv;
    g.n = int64_t{1} << ln; g.b = int64_t{1} << g.logB; g.p = int64_t{1} << lp; g.L = int64_t{1} << g.logL;
    g.vec = int64_t{1} << lv; g.vp = int64_t{1} << g.logVP; g.m = int64_t{1} << g.logM;
    return g;
}

// the stage on digit s over all elements: DFT of the digit, sign -1 / +1
template <typename D> static void digit_dft(std::vector<Z> &x, int s, double sign) {
    const int R = 1 << D::lr(s), sh = D::sh(s), N = (int)x.size();
    for (int i = 0; i < N; i++) {
        if ((i >> sh) & (R - 1)) continue;
        std::vector<Z> y(R);
        for (int k = 0; k < R; k++)
            for (int r = 0; r < R; r++) y[k] += x[i + (r << sh)] * std::polar(1.0, sign * 2 * M_PI * k * r / R);
        for (int k = 0; k < R; k++) x[i + (k << sh)] = y[k];
    }
}
template <typename D, int s> static void twiddle(std::vector<Z> &x, const std::vector<int64_t> &e, double sign) {
    const int N = (int)x.size(), lr = D::lr(s), sh = D::sh(s);
    for (int i = 0; i < N; i++) {
        const int r = (i >> sh) & ((1 << lr) - 1), iv = ((i >> (sh + lr)) << sh) | (i & ((1 << sh) - 1));
        if (r >= D::r0(s)) x[i] *= std::polar(1.0, sign * 2 * M_PI * (double)e.at(D::tw(s) + (r << D::row(s)) + D::template col<s>(iv)) / N);
    }
}
template <typename D, int s> static void forward(std::vector<Z> &x, const std::vector<int64_t> &e) {
    digit_dft<D>(x, s, -1);
    if constexpr (s + 1 < D::NST) {
        twiddle<D, s>(x, e, -1);
        forward<D, s + 1>(x, e);
    }
}
template <typename D, int s> static void inverse(std::vector<Z> &x, const std::vector<int64_t> &e) {
    if constexpr (s + 1 < D::NST) twiddle<D, s>(x, e, 1);
    digit_dft<D>(x, s, 1);
    if constexpr (s > 0) inverse<D, s - 1>(x, e);
}

template <int LN, int LV> static void check() {
    constexpr int LM = LN - LV, N = 1 << LN;
    using DF = SplitDigits<LV, LM, false>;
    using DI = SplitDigits<LV, LM, true>;
    const Geom g = geom(LN, LV, LV > 1 ? 1 : 0);
    std::vector<int64_t> ef, ei;
    batch_exact_twiddles(g, false, &ef);
    batch_exact_twiddles(g, true, &ei);
    bad += (int)ef.size() != DF::tw(DF::NST - 1) || (int)ei.size() != DI::tw(DI::NST - 1);
    for (int64_t v : ef) bad += v < 0 || v >= N;
    for (int64_t v : ei) bad += v < 0 || v >= N;
    std::vector<Z> x(N), spec(N);
    for (int i = 0; i < N; i++) x[i] = Z(std::sin(1 + 3.7 * i * i), std::cos(2.1 * i));
    std::vector<Z> y = x;
    forward<DF, 0>(y, ef);
    // index after the forward: digits of k, lowest first at the top
    std::vector<char> seen(N, 0);
    for (int k = 0; k < N; k++) {
        const int at = inverse_index<DF>(k), to = inverse_index<DI>(k);
        bad += at < 0 || at >= N || to < 0 || to >= N || seen[to]++;
        spec[to] = y[at];
        if (k % 7 == 0 || k < 64) {
            Z ref = 0;
            for (int i = 0; i < N; i++) ref += x[i] * std::polar(1.0, -2 * M_PI * (double)((int64_t)i * k % N) / N);
            worst = std::fmax(worst, std::abs(ref - y[at]) / N);
        }
    }
    inverse<DI, DI::NST - 1>(spec, ei);
    for (int i = 0; i < N; i++) worst = std::fmax(worst, std::abs(spec[i] / (double)N - x[i]));
    // weight tables: frequency side of both digit orders, vector side
    for (int lp = 0; lp <= 2 && lp <= LV && LV + lp <= LN; lp++) {
        const Geom q = geom(LN, LV, lp);
        const int ltl = kBatchTileLog - LN, E = 1 << kBatchTileLog;
        for (int inv = 0; inv < 2; inv++)
            for (int kind : {PASS_X2, PASS_Y2}) {
                const std::vector<int> lrs = batch_exact_digits(q, inv);
                const AxisMap m = axis_map(q, kind, 1, ltl, kBatchPtsLog, lrs, std::min(ltl, 3));
                const int nst = (int)lrs.size(), lr = lrs[nst - 1], lnt = kBatchTileLog - kBatchPtsLog;
                std::vector<int> index(axis_slot(E - 1) + 1, -1);
                for (int i = 0; i < E; i++) index[axis_slot(i)] = i;
                const int64_t blk = (q.n >> ltl) - 1;
                const LineAddr la = line_addr(q, kind, blk << ltl, m.lg);
                std::vector<char> sa(E, 0), sf(E, 0);
                for (int tid = 0; tid < 1 << lnt; tid++)
                    for (int r = 0; r < 1 << kBatchPtsLog; r++) {
                        int64_t a = la.a_base, f = la.f_base;
                        int va = 0, vf = 0;
                        for (int b = 0; b < lnt; b++)
                            if (tid >> b & 1) a += m.va[b], va += m.vs[b], f += m.fa[b], vf += m.fs[b];
                        for (int b = 0; b < kBatchPtsLog; b++)
                            if (r >> b & 1) a += m.va[lnt + b], va += m.vs[lnt + b];
                        const int u = r >> lr, rr = r & ((1 << lr) - 1);
                        for (int b = 0; b < kBatchPtsLog - lr; b++)
                            if (u >> b & 1) f += m.fa[lnt + b], vf += m.fs[lnt + b];
                        for (int b = 0; b < lr; b++)
                            if (rr >> b & 1) f += m.fr[b];
                        vf += axis_slot(rr << ltl);
                        if (va >= (int)index.size() || vf >= (int)index.size() || index[va] < 0 || index[vf] < 0 ||
                            sa[index[va]]++ || sf[index[vf]]++) { bad++; continue; }
                        const int ia = index[va], jf = index[vf];
                        LineAddr l = line_addr(q, kind, (blk << ltl) + (ia & ((1 << ltl) - 1)), m.lg);
                        const int64_t n = ia >> ltl, n1 = n & (q.m - 1), n2 = n >> q.logM;
                        bad += a != l.a_base + (n1 >> q.logB) * l.a_chunk + ((n1 & (q.b - 1)) * q.vec + n2) * l.a_hi;
                        int64_t k = 0;
                        for (int s = 0, o = 0, sh = LN; s < nst; s++) {
                            sh -= lrs[s];
                            k |= (int64_t)((jf >> ltl >> sh) & ((1 << lrs[s]) - 1)) << o;
                            o += lrs[s];
                        }
                        l = line_addr(q, kind, (blk << ltl) + (jf & ((1 << ltl) - 1)), m.lg);
                        const int64_t k1 = k >> q.logVEC, k2 = k & (q.vec - 1), pos = k1 * q.vp + (k2 & (q.vp - 1));
                        const int64_t fo = l.f_lg ? (pos >> l.f_lg) * l.f_hi + (pos & ((1 << l.f_lg) - 1)) : pos * l.f_pos;
                        bad += f != l.f_base + (k2 >> q.logVP) * l.f_chunk + fo || f < 0 || f >= q.n * q.n || a < 0 || a >= q.n * q.n;
                    }
            }
    }
}
template <int LN> static void check_n() { check<LN, 1>(), check<LN, 2>(), check<LN, 3>(), check<LN, 4>(); }

int main() {
    check_n<6>(), check_n<7>(), check_n<8>(), check_n<9>(), check_n<10>(), check_n<11>(), check_n<12>();
    std::printf("%ld mismatches, largest deviation %.2e\n", bad, worst);
    return bad != 0 || !(worst < 1e-11);
}
