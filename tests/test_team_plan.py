"""The FP64 plan over random bases, on the host: shells of up to 20 primitives
that share exponents, in any order, with zero coefficients, up to f.  Every
surviving pair of super pairs is covered once, by tasks whose batches fit the
shared memory that their launch asks for, and the two builders of primitive
pairs agree on their number."""
import native_driver

DRIVER = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include "hfx_engine.hpp"
using namespace hfx;

static Basis random_basis(std::mt19937& g)
{
    auto U = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); };
    auto I = [&](int a, int b) { return std::uniform_int_distribution<int>(a, b)(g); };
    std::vector<double> centres, alpha, coeff, norm;
    std::vector<int> lmn, off{0};
    const int atoms = I(1, 4);
    for (int a = 0; a < atoms; ++a) {
        const double R[3] = {U(-4, 4), U(-4, 4), U(-4, 4)};
        std::vector<double> pool(I(1, 20));
        for (double& x : pool) x = std::exp(U(-3, 9));
        const int shells = I(1, 6);
        for (int s = 0; s < shells; ++s) {
            const int L = I(0, 10) < 4 ? 0 : I(0, 3), n = (int)pool.size();
            const int np = I(0, 3) == 0 ? 1 : I(1, I(0, 4) == 0 ? n : std::min(n, 6)), first = I(0, n - np);
            std::vector<double> e(pool.begin() + first, pool.begin() + first + np), c;
            if (I(0, 2) == 0)
                for (double& x : e) x *= U(0.9, 1.1);
            if (I(0, 3) == 0) std::shuffle(e.begin(), e.end(), g);
            const bool none = I(0, 9) == 0;
            for (int k = 0; k < np; ++k) c.push_back(none || I(0, 4) == 0 ? 0.0 : U(-1, 1));
            for (int x = 0; x < ncart(L); ++x) {
                int l, m, k;
                component(L, x, l, m, k);
                lmn.insert(lmn.end(), {l, m, k});
                centres.insert(centres.end(), R, R + 3);
                alpha.insert(alpha.end(), e.begin(), e.end());
                coeff.insert(coeff.end(), c.begin(), c.end());
                norm.insert(norm.end(), np, 1.0);
                off.push_back((int)alpha.size());
            }
        }
    }
    return basis_from_functions(hfx_functions{(int)off.size() - 1, centres.data(), lmn.data(), off.data(), alpha.data(),
                                              coeff.data(), norm.data()});
}

int main(int argc, char** argv)
{
    int bad = 0;
    auto fail = [&](int seed, const char* what, long long a, long long b) {
        if (++bad < 20) std::printf("seed %d: %s: %lld, %lld\n", seed, what, a, b);
    };
    for (int seed = 0; seed < std::atoi(argv[1]); ++seed) {
        std::mt19937 g(seed);
        const Basis b = random_basis(g);
        const Fragments fr = single_fragment(b);
        const SuperData sd = build_super_data(b, fr);
        const PairData pd = build_pair_data(b, fr, seed % 2);
        for (size_t p = 0; p < sd.pairs.size(); ++p)
            for (size_t k = 0; k < sd.members[p].size(); ++k)
                if (sd.member_npp[p][k] != pd.hpairs[sd.members[p][k]].npp)
                    fail(seed, "primitive pairs", sd.member_npp[p][k], pd.hpairs[sd.members[p][k]].npp);
        auto U = [&](double a, double c) { return std::uniform_real_distribution<double>(a, c)(g); };
        std::vector<double> q(sd.pairs.size());
        for (double& x : q) x = U(0, 1) < 0.05 ? 0.0 : std::exp(U(-12, 1));
        const double cut = U(0, 1) < 0.3 ? -1.0 : std::exp(U(-20, 0));
        const int nsm = U(0, 1) < 0.5 ? 152 : 4;
        for (bool diagonal : {false, true}) {
            const TeamPlanHost plan = diagonal ? build_team_diagonal(sd, nsm) : build_team_plan(sd, q, cut, nsm);
            std::map<std::pair<int, int>, long long> rows;      // covered bra primitive pairs of (bra, ket)
            size_t tasks = 0;
            for (const TeamGroup& gr : plan.groups) {
                tasks += gr.n;
                // 227 KB per CTA, less the kernel's header
                if ((gr.L < 0 ? 4 * 456 + 64 : 16) + 8 * (long long)gr.slice > 232448) fail(seed, "slice", gr.slice, gr.L);
                for (size_t x = gr.off; x < gr.off + gr.n; ++x) {
                    const TeamTask& t = plan.tasks[x];
                    const SuperPair &k = sd.pairs[t.ket], &b0 = sd.pairs[plan.order[t.b0]];
                    const int L = b0.L + k.L;
                    if (gr.L != (L > kTeamMaxRegL ? -1 : L)) fail(seed, "angular momentum", gr.L, L);
                    const int need = team_slice(b0.L, k.L, b0.nA, b0.nB, k.nA, k.nB, t.nr, t.nkb, t.nw, t.slots, t.nb, t.parts, k.nmem);
                    if (need > gr.slice) fail(seed, "shared memory", need, gr.slice);
                    if (!t.nr || !t.nkb || !t.slots || !t.parts || !t.nb) fail(seed, "empty batch", t.nr, t.nkb);
                    if (t.nb == 1) {
                        if (t.i0 >= t.i1 || t.i1 > b0.npp || t.nw < std::min<int>(t.nr, t.i1 - t.i0)) fail(seed, "rows", t.i0, t.i1);
                        rows[{plan.order[t.b0], t.ket}] += t.i1 - t.i0;
                        continue;
                    }
                    int sum = 0, most = 0;
                    for (int y = 0; y < t.nb; ++y) {
                        const int p = plan.order[t.b0 + y];
                        const SuperPair& s = sd.pairs[p];
                        sum += s.npp;
                        most = std::max(most, s.npp);
                        rows[{p, t.ket}] += s.npp;
                        if (s.type != b0.type || s.nA != b0.nA || s.nB != b0.nB || s.nmem != b0.nmem) fail(seed, "class", p, t.ket);
                    }
                    if (t.i0 != 0 || t.i1 != sum || sum > t.nr || k.npp > t.nkb || t.slots * most > t.nw) fail(seed, "batch", sum, most);
                }
            }
            if (tasks != plan.tasks.size()) fail(seed, "tasks", tasks, plan.tasks.size());
            for (int x = 0; x < (int)sd.pairs.size(); ++x)
                for (int y = diagonal ? x : 0; y <= x; ++y) {
                    const bool on = diagonal ? sd.pairs[x].npp > 0
                                             : sd.pairs[x].npp && sd.pairs[y].npp && (cut < 0.0 || (q[x] > 0.0 && q[y] > 0.0 && q[x] * q[y] >= cut));
                    int whole = 0, part = 0;
                    for (const auto& o : {std::make_pair(x, y), std::make_pair(y, x)}) {
                        if (!rows.count(o) || (x == y && whole + part)) continue;
                        (rows[o] == sd.pairs[o.first].npp ? whole : part) += 1;
                    }
                    if (whole != on || part) fail(seed, "coverage", whole, part);
                }
        }
    }
    std::printf("%d\n", bad);
}
"""


def test_plans_of_random_bases_cover_every_quartet_once(tmp_path):
    assert native_driver.run_driver(DRIVER, tmp_path / "plan", 60) == "0\n"
