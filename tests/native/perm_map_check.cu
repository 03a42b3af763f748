// perm_map_check.cu -- host check of the converters' bit permutations (zm_layout.cu): for
// every layout, each (block, thread, register) must read the input element whose natural or
// interleaved partner (the index maps of zm_index.cuh) its shared-memory slot is written to,
// every element once, with complex64 pairs on 16 bytes.
#include <cstdio>
#include <vector>

#include "zm_layout.cu"

namespace zm {
void count_launch() {}
}  // namespace zm
using namespace zm;

static long bad = 0, checks = 0;

static void check(const Geom &g, int dtype, bool recip, bool to_nat) {
    const PermMap m = perm_map(g, dtype, recip, to_nat);
    const int64_t total = g.dim == 2 ? g.n * g.n : g.n * g.n * g.n;
    const int E = 1 << m.le;
    const bool pair = dtype != 0 && m.le > 8;
    std::vector<int64_t> at(perm_slot(E - 1) + 1);
    std::vector<char> seen(total, 0);
    for (int64_t blk = 0; blk < total >> m.le; blk++) {
        int64_t bi = 0, bo = 0;
        for (int f = 0; f < m.nf; f++) {
            bi += (int64_t)((unsigned)blk & m.fmask[f]) << m.fin[f];
            bo += (int64_t)(((unsigned)blk & m.fmask[f]) >> m.flow[f]) << m.fout[f];
        }
        std::fill(at.begin(), at.end(), int64_t{-1});
        for (int x = 0; x < E; x++) {   // list positions as bits of x
            int64_t a = bi;
            int s = 0;
            for (int q = 0; q < m.le; q++)
                if (x >> q & 1) a += int64_t{1} << m.ia[q], s += m.is[q];
            if (a < 0 || a >= total || s < 0 || s >= (int)at.size() || at[s] >= 0) { bad++; continue; }
            at[s] = a;
        }
        for (int x = 0; x < E; x++, checks++) {
            int64_t o = bo;
            int s = 0;
            for (int q = 0; q < m.le; q++)
                if (x >> q & 1) o += int64_t{1} << m.oa[q], s += m.os[q];
            if (o < 0 || o >= total || seen[o] || s < 0 || s >= (int)at.size() || at[s] < 0) { bad++; continue; }
            seen[o] = 1;
            const int64_t inter = to_nat ? at[s] : o, nat = to_nat ? o : at[s];
            bad += (recip ? recip_gidx(inter, g) : real_gidx(inter, g)) != nat;
        }
    }
    if (pair) bad += (m.ia[0] != 0) + (m.oa[0] != 0);
    for (char s : seen) bad += !s;
}

int main() {
    for (int dim = 2; dim <= 3; dim++)
        for (int ln = 1; ln <= (dim == 2 ? 9 : 6); ln++)
            for (int lp = 0; lp <= 3 && 2 * lp <= ln; lp++)
                for (int lb = 0; lb <= ln - 2 * lp; lb++) {
                    Geom g;
                    g.dim = dim;
                    g.logN = ln; g.logB = lb; g.logP = lp;
                    g.logL = ln - lp; g.logVEC = ln - lp - lb; g.logVP = g.logVEC - lp; g.logM = lb + lp;
                    g.n = int64_t{1} << ln; g.b = int64_t{1} << lb; g.p = int64_t{1} << lp;
                    g.L = int64_t{1} << g.logL; g.vec = int64_t{1} << g.logVEC;
                    g.vp = int64_t{1} << g.logVP; g.m = int64_t{1} << g.logM;
                    for (int f = 0; f < 8; f++) check(g, f & 1, f & 2, f & 4);
                }
    std::printf("%ld mismatches in %ld elements\n", bad, checks);
    return bad != 0;
}
