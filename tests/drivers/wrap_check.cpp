// Host check of the ghost-free periodic step: from one state whose ghosts
// repeat their sources, stream and mix with ghost copies after every step, and
// without ghosts plus one exchange at the end, and compare every slot.  The
// "collision" is an arbitrary cell-local map, so equality is exact.
#include "../../lbm3_b200/csrc/builder.h"
#include "../../lbm3_b200/csrc/lattice.h"

#include <vector>

using namespace lbm;

namespace {

struct Box {
    const HostLevel& L;
    int n, nx, nxy, m[3];
    explicit Box(const HostLevel& l)
        : L(l), n(l.info.cellCount), nx(l.info.nx), nxy(l.info.nx * l.info.ny),
          m{l.info.nx - 2, l.info.ny - 2, l.info.nz - 2} {}
    int next(int c) const { return c + 1 < n ? c + 1 : 0; }
    int nbr(int c, int which) const {
        if (which & 4) c = L.kPlus[c];
        if (which & 2) c = L.jPlus[c];
        return which & 1 ? next(c) : c;
    }
    // image shift of direction d at cell c, and its index distance
    void shift(int c, int d, int (&s)[3]) const {
        const int at[3] = {c % nx, c / nx % L.info.ny, c / nxy}, v[3] = {cx(d), cy(d), cz(d)};
        for (int a = 0; a < 3; ++a) s[a] = v[a] > 0 && at[a] == 1 ? m[a] : v[a] < 0 && at[a] == m[a] ? -m[a] : 0;
    }
    int dist(const int (&s)[3]) const { return s[0] + s[1] * nx + s[2] * nxy; }
};

using Field = std::vector<double>;  // [27][n]

void mix(double (&f)[27]) {
    double s = 0.0;
    for (int d = 0; d < 27; ++d) s += f[d] * (1.0 + 0.1 * d);
    for (int d = 0; d < 27; ++d) f[d] = 0.75 * f[d] + 0.01 * (d % 5) * s;
}

int pre(bool F, int d) { return F ? inv(d) : d; }

void copyGhosts(const Box& b, Field& f, bool F) {
    for (size_t q = 0; q < b.L.perIndex.size(); ++q)
        for (int d = 0; d < 27; ++d)
            f[size_t(pre(F, d)) * b.n + b.nbr(b.L.perIndex[q], preNbr(d))] =
                f[size_t(pre(F, d)) * b.n + b.nbr(b.L.perSource[q], preNbr(d))];
}

}  // namespace

// 0: the fields agree; 1: they differ; 2: the level does not qualify
extern "C" int lbm_wrap_check(const lbm_case* c, int steps, long long* skipped) {
    HostDomain d;
    buildDomain(*c, d);
    const HostLevel& L = d.levels[0];
    *skipped = 0;
    if (!L.wrapped) return 2;
    for (uint32_t w : L.wrapSkip) *skipped += __builtin_popcount(w);
    const Box b(L);
    Field a(size_t(27) * b.n), w;
    uint32_t x = 12345u;
    for (double& v : a) v = (x = x * 1664525u + 1013904223u) * 1e-10;
    bool F = L.info.esotwistFlipper;
    copyGhosts(b, a, F);
    w = a;
    std::vector<char> ghost(b.n, 0);
    for (int q : L.perIndex) ghost[q] = 1;
    for (int s = 0; s < steps; ++s, F = !F) {
        for (int cell = 0; cell < b.n; ++cell) {
            double f[27];
            for (int q = 0; q < 27; ++q) f[q] = a[size_t(pre(F, q)) * b.n + b.nbr(cell, preNbr(q))];
            mix(f);
            for (int q = 0; q < 27; ++q) a[size_t(pre(!F, q)) * b.n + b.nbr(cell, postNbr(q))] = f[q];
            if (ghost[cell]) continue;
            for (int q = 0; q < 27; ++q) {
                int sh[3];
                b.shift(cell, q, sh);
                f[q] = w[size_t(pre(F, q)) * b.n + b.nbr(cell, preNbr(q)) + b.dist(sh)];
            }
            mix(f);
            for (int q = 0; q < 27; ++q) w[size_t(pre(!F, q)) * b.n + b.nbr(cell, postNbr(q))] = f[q];
        }
        copyGhosts(b, a, !F);
    }
    // the exchange after the last step
    const Field last = w;
    for (size_t q = 0; q < L.perIndex.size(); ++q) {
        const int g = L.perIndex[q], src = L.perSource[q];
        const int gap[3] = {g % b.nx - src % b.nx, g / b.nx % L.info.ny - src / b.nx % L.info.ny, g / b.nxy - src / b.nxy};
        for (int k = 0; k < 27; ++k) {
            int sh[3];
            b.shift(src, k, sh);
            const bool here = sh[0] == gap[0] && sh[1] == gap[1] && sh[2] == gap[2];
            w[size_t(pre(F, k)) * b.n + b.nbr(here ? src : g, preNbr(k))] =
                last[size_t(pre(F, k)) * b.n + b.nbr(src, preNbr(k)) + b.dist(sh)];
        }
    }
    return a == w ? 0 : 1;
}
