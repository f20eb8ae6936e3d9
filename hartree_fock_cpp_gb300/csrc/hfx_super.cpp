// hfx_super.cpp -- host side of the team kernel: super shells and super pairs
// of a basis, and the plan of the surviving super quartets.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <unordered_map>

#include "hfx_engine.hpp"
#include "hfx_team.hpp"

namespace hfx {

namespace {

struct SuperShell {
    std::vector<int> shells;            // indices in the basis, ascending
    std::vector<double> exps;           // union, in the order of the longest member
    std::vector<std::vector<int>> at;   // per member: primitive of the shell for each exponent, or -1
    int nfn = 0, L = 0, sig = 0;
};

// Shells of one centre, longest contraction first: a shell joins the first
// super shell whose exponents contain all of its own, if the angular momenta
// agree (general contraction) or the exponent sets are the same (SP shells),
// up to kSuperMaxFn functions.
std::vector<SuperShell> make_super_shells(const Basis& b, int s0, int s1)
{
    std::vector<int> idx(s1 - s0);
    std::iota(idx.begin(), idx.end(), s0);
    std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) { return b.shells[x].nprim() > b.shells[y].nprim(); });
    std::vector<SuperShell> out;
    std::map<std::vector<double>, std::vector<int>> centres;
    for (int s : idx) {
        const Shell& sh = b.shells[s];
        std::vector<int>& here = centres[{sh.x, sh.y, sh.z}];
        const int nc = ncart(sh.L);
        bool placed = false;
        for (int o : here) {
            SuperShell& g = out[o];
            if (g.nfn + nc > kSuperMaxFn) continue;
            std::vector<int> at(g.exps.size(), -1);
            int found = 0;
            for (int i = 0; i < sh.nprim(); ++i)
                for (size_t e = 0; e < g.exps.size(); ++e)
                    if (g.exps[e] == sh.exps[i] && at[e] < 0) {
                        at[e] = i;
                        ++found;
                        break;
                    }
            if (found != sh.nprim()) continue;
            bool one_l = true;
            for (int m : g.shells) one_l = one_l && b.shells[m].L == sh.L;
            if (!one_l && found != (int)g.exps.size()) continue;
            g.shells.push_back(s);
            g.at.push_back(at);
            g.nfn += nc;
            g.L = std::max(g.L, sh.L);
            placed = true;
            break;
        }
        if (placed) continue;
        SuperShell g;
        g.shells = {s};
        g.exps = sh.exps;
        std::vector<int> at(sh.nprim());
        std::iota(at.begin(), at.end(), 0);
        g.at = {at};
        g.nfn = nc;
        g.L = sh.L;
        here.push_back((int)out.size());
        out.push_back(g);
    }
    for (SuperShell& g : out) {
        std::vector<int> o(g.shells.size());
        std::iota(o.begin(), o.end(), 0);
        std::sort(o.begin(), o.end(), [&](int x, int y) { return g.shells[x] < g.shells[y]; });
        SuperShell t = g;
        for (size_t k = 0; k < o.size(); ++k) {
            g.shells[k] = t.shells[o[k]];
            g.at[k] = t.at[o[k]];
        }
    }
    return out;
}

// Coefficient tables of the 16 ordered (la, lb) classes.
struct TeamClass {
    int off, ncoef;
    std::vector<int> first, count;   // per component pair
};
struct TeamClasses {
    TeamClass c[kMaxL + 1][kMaxL + 1];
    std::vector<short> codes;
};
const TeamClasses& team_classes()
{
    static const TeamClasses tc = [] {
        TeamClasses t;
        for (int la = 0; la <= kMaxL; ++la)
            for (int lb = 0; lb <= kMaxL; ++lb) {
                TeamClass& c = t.c[la][lb];
                c.off = (int)t.codes.size();
                int k = 0;
                for (int a = 0; a < ncart(la); ++a)
                    for (int b = 0; b < ncart(lb); ++b) {
                        int ax, ay, az, bx, by, bz;
                        component(la, a, ax, ay, az);
                        component(lb, b, bx, by, bz);
                        c.first.push_back(k);
                        for (int x = 0; x <= ax + bx; ++x)
                            for (int y = 0; y <= ay + by; ++y)
                                for (int z = 0; z <= az + bz; ++z, ++k)
                                    t.codes.push_back((short)(herm_index(x, y, z) | (((x + y + z) & 1) << 14)));
                        c.count.push_back(k - c.first.back());
                    }
                c.ncoef = k;
            }
        return t;
    }();
    return tc;
}

}  // namespace

const std::vector<short>& team_codes() { return team_classes().codes; }

const TeamRidx& team_ridx()
{
    static const TeamRidx tab = [] {
        TeamRidx r;
        auto list = [](int L) {
            std::vector<int> v;
            for (int s = 0; s <= L; ++s)
                for (int t = 0; t <= s; ++t)
                    for (int u = 0; u <= s - t; ++u) v.push_back(t * 256 + u * 16 + s - t - u);
            return v;
        };
        for (int L1 = 0; L1 <= 2 * kMaxL; ++L1)
            for (int L2 = 0; L2 <= 2 * kMaxL; ++L2) {
                r.at[L1 * 7 + L2] = (int)(r.words.size() / 4);
                const std::vector<int> a = list(L1), b = list(L2);
                const int H1 = (int)a.size(), J = team_tuv_group(H1);
                for (int x : b)
                    for (int g = 0; g < H1; g += J) {
                        unsigned w[4] = {0, 0, 0, 0};
                        for (int j = 0; j < J && g + j < H1; ++j) {
                            const int y = a[g + j] + x;
                            w[j >> 1] |= (unsigned)herm_index(y >> 8, (y >> 4) & 15, y & 15) << (16 * (j & 1));
                        }
                        r.words.insert(r.words.end(), w, w + 4);
                    }
            }
        return r;
    }();
    return tab;
}

SuperData build_super_data(const Basis& b, const Fragments& fr)
{
    const TeamClasses& tc = team_classes();
    SuperData sd;
    std::map<std::vector<int>, int> sigs, types, classes;
    std::vector<std::vector<int>> sig_ls;
    struct Item {
        int f, x, y, id;
    };
    std::vector<std::vector<SuperShell>> sup(fr.count());
    std::vector<Item> items;
    for (int f = 0; f < fr.count(); ++f) {
        sup[f] = make_super_shells(b, fr.sh[f], fr.sh[f + 1]);
        for (SuperShell& s : sup[f]) {
            std::vector<int> key;
            for (int m : s.shells) key.push_back(b.shells[m].L);
            std::vector<int> ls = key;
            key.push_back(-1 - (int)s.exps.size());
            auto it = sigs.emplace(key, (int)sigs.size());
            if (it.second) sig_ls.push_back(ls);
            s.sig = it.first->second;
        }
        sd.pbase.push_back((int)items.size());
        for (int x = 0; x < (int)sup[f].size(); ++x)
            for (int y = 0; y <= x; ++y) items.push_back(Item{f, x, y, (int)items.size()});
    }
    sd.pbase.push_back((int)items.size());
    const int np = (int)items.size();
    sd.pairs.resize(np);
    sd.members.resize(np);
    sd.member_at.resize(np);
    sd.cls.resize(np);
    // types and classes first (serial: their numbering is the pairs' order)
    std::vector<std::pair<int, int>> sides(np);
    for (int p = 0; p < np; ++p) {
        const Item& it = items[p];
        int x = it.x, y = it.y;
        const std::vector<SuperShell>& ss = sup[it.f];
        if (ss[x].sig < ss[y].sig) std::swap(x, y);
        sides[p] = {x, y};
        const SuperShell &A = ss[x], &B = ss[y];
        SuperPair& d = sd.pairs[p];
        std::memset(&d, 0, sizeof(d));
        std::vector<int> key = sig_ls[A.sig];
        key.push_back(-1);
        key.insert(key.end(), sig_ls[B.sig].begin(), sig_ls[B.sig].end());
        auto ty = types.find(key);
        if (ty == types.end()) {
            const int off = (int)sd.types.size();
            ty = types.emplace(key, off).first;
            const std::vector<int>&la = sig_ls[A.sig], &lb = sig_ls[B.sig];
            for (size_t ma = 0; ma < la.size(); ++ma)
                for (int a = 0; a < ncart(la[ma]); ++a)
                    for (size_t mb = 0; mb < lb.size(); ++mb)
                        for (int c = 0; c < ncart(lb[mb]); ++c) {
                            const TeamClass& k = tc.c[la[ma]][lb[mb]];
                            const int ab = a * ncart(lb[mb]) + c;
                            sd.types.push_back((int)(ma * lb.size() + mb) | k.first[ab] << 8 | k.count[ab] << 20);
                        }
            for (int pass = 0; pass < 2; ++pass)
                for (int l0 : la)
                    for (int l1 : lb) sd.types.push_back(pass ? tc.c[l0][l1].ncoef : tc.c[l0][l1].off);
        }
        d.type = reinterpret_cast<const int*>((size_t)ty->second);
        d.nmem = (int)(A.shells.size() * B.shells.size());
        d.nA = A.nfn;
        d.nB = B.nfn;
        d.L = A.L + B.L;
        d.same = x == y;
        d.kdim = fr.K(it.f);
        d.frag = it.f;
        d.moff = fr.moff[it.f];
        d.id = p;
        d.shA = x;
        d.shB = y;
        d.pbase = sd.pbase[it.f];
        sd.cls[p] = classes.emplace(std::vector<int>{A.sig, B.sig}, (int)classes.size()).first->second;
        const int sb = fr.sh[it.f], pb = fr.pbase[it.f];
        for (size_t ia = 0; ia < A.shells.size(); ++ia)
            for (size_t ib = 0; ib < B.shells.size(); ++ib) {
                const int ma = A.shells[ia], mb = B.shells[ib];
                if (d.same && ma < mb) continue;
                sd.members[p].push_back(pb + shell_pair_id(ma - sb, mb - sb));
                sd.member_at[p].push_back((int)(ia * B.shells.size() + ib));
            }
    }
    sd.ncls = (int)classes.size();
    // per pair: primitive pairs, lists and coefficients, on host threads;
    // appended in pair order, so the tables do not depend on the thread count
    struct Out {
        std::vector<double> hdr, coef;
        std::vector<int> tab, npp;
    };
    std::vector<Out> outs(np);
    host_parallel_for((np + 15) / 16, [&](int unit) {
        std::vector<double> E[3];
        for (int p = unit * 16; p < std::min(np, unit * 16 + 16); ++p) {
            const Item& it = items[p];
            const SuperShell &A = sup[it.f][sides[p].first], &B = sup[it.f][sides[p].second];
            const Shell &cA = b.shells[A.shells[0]], &cB = b.shells[B.shells[0]];
            const bool same = sides[p].first == sides[p].second;
            const int nm = (int)(A.shells.size() * B.shells.size()), nb = (int)B.shells.size();
            const int nq = (int)(A.exps.size() * B.exps.size());
            const int nt = A.L + B.L + 1;
            std::vector<std::vector<double>> cf(nm);    // per member: all primitive pairs' coefficients
            std::vector<std::vector<double>> big(nm);   // and each one's largest
            std::vector<std::vector<double>> own(nm);   // the same, (i, j) and (j, i) of one super shell apart
            std::vector<std::vector<char>> has(nm);
            for (int m = 0; m < nm; ++m) {
                const int la = b.shells[A.shells[m / nb]].L, lb = b.shells[B.shells[m % nb]].L;
                cf[m].assign((size_t)nq * tc.c[la][lb].ncoef, 0.0);
                big[m].assign(nq, 0.0);
                own[m].assign(nq, -1.0);
                has[m].assign(nq, 0);
            }
            const double ox[3] = {cA.x, cA.y, cA.z}, px[3] = {cB.x, cB.y, cB.z};
            std::vector<double> geo((size_t)nq * 4, 0.0);
            for (int i = 0; i < (int)A.exps.size(); ++i)
                for (int j = 0; j < (int)B.exps.size(); ++j) {
                    // on one super shell (i, j) and (j, i) are one Gaussian: one entry, weights added
                    const int q = same && i < j ? j * (int)B.exps.size() + i : i * (int)B.exps.size() + j;
                    const double al = A.exps[i], be = B.exps[j], pe = al + be;
                    for (int d = 0; d < 3; ++d) hermite_1d(A.L, B.L, al, be, ox[d], px[d], E[d]);
                    geo[4 * q] = pe;
                    for (int d = 0; d < 3; ++d) geo[4 * q + 1 + d] = (al * ox[d] + be * px[d]) / pe;
                    auto e = [&](int d, int x, int y, int t) { return E[d][((size_t)x * (B.L + 1) + y) * nt + t]; };
                    for (int m = 0; m < nm; ++m) {
                        const int ia = A.at[m / nb][i], jb = B.at[m % nb][j];
                        const Shell &sa = b.shells[A.shells[m / nb]], &sb = b.shells[B.shells[m % nb]];
                        if (ia < 0 || jb < 0 || (same && A.shells[m / nb] < B.shells[m % nb])) continue;
                        const bool folded = has[m][q] != 0;   // the second order of one Gaussian
                        has[m][q] = 1;
                        const TeamClass& k = tc.c[sa.L][sb.L];
                        double* c = cf[m].data() + (size_t)q * k.ncoef;
                        double mx = 0.0;
                        for (int a = 0; a < ncart(sa.L); ++a)
                            for (int g = 0; g < ncart(sb.L); ++g) {
                                int ax, ay, az, bx, by, bz;
                                component(sa.L, a, ax, ay, az);
                                component(sb.L, g, bx, by, bz);
                                const double w = sa.w[(size_t)a * sa.nprim() + ia] * sb.w[(size_t)g * sb.nprim() + jb];
                                for (int t = 0; t <= ax + bx; ++t)
                                    for (int u = 0; u <= ay + by; ++u)
                                        for (int v = 0; v <= az + bz; ++v, ++c) {
                                            const double x = w * e(0, ax, bx, t) * e(1, ay, by, u) * e(2, az, bz, v);
                                            mx = std::max(mx, std::fabs(x));
                                            *c += x;
                                        }
                            }
                        own[m][i * (int)B.exps.size() + j] = mx;
                        if (folded) {
                            c -= k.ncoef;
                            mx = 0.0;
                            for (int x = 0; x < k.ncoef; ++x) mx = std::max(mx, std::fabs(c[x]));
                        }
                        big[m][q] = mx;
                    }
                }
            // a member's primitive pairs below kPrimPairCut of its largest are left out
            std::vector<char> keep(nq, 0);
            for (int m = 0; m < nm; ++m) {
                double mx = 0.0;
                for (int q = 0; q < nq; ++q) mx = std::max(mx, big[m][q]);
                for (int q = 0; q < nq; ++q) {
                    if (has[m][q] && big[m][q] < kPrimPairCut * mx) has[m][q] = 0;
                    if (has[m][q]) keep[q] = 1;
                }
            }
            Out& o = outs[p];
            // primitive pairs of more members first: a short member's list
            // then lies in the first batches of a long ket loop
            std::vector<int> place(nq, -1), seq;
            for (int q = 0; q < nq; ++q)
                if (keep[q]) seq.push_back(q);
            std::vector<int> uses(nq, 0);
            for (int m = 0; m < nm; ++m)
                for (int q = 0; q < nq; ++q) uses[q] += has[m][q] != 0;
            std::stable_sort(seq.begin(), seq.end(), [&](int x, int y) { return uses[x] > uses[y]; });
            int n = 0;
            for (int q : seq) {
                place[q] = n++;
                o.hdr.insert(o.hdr.end(), geo.begin() + 4 * (size_t)q, geo.begin() + 4 * (size_t)q + 4);
                o.hdr.push_back(5.914967172795613 / geo[4 * (size_t)q]);   // sqrt(2 pi^{5/2}) / p
                o.hdr.push_back(0.0);
            }
            o.tab.assign(3 * nm, 0);
            for (const SuperShell* s : {&A, &B})
                for (int m : s->shells)
                    for (int c = 0; c < ncart(b.shells[m].L); ++c) o.tab.push_back(b.shells[m].bf0 - fr.bf[it.f] + c);
            {
                // component pairs by decreasing work: (member, coefficients) as in the type table
                std::vector<std::pair<int, int>> w;
                for (size_t ma = 0; ma < A.shells.size(); ++ma)
                    for (int a = 0; a < ncart(b.shells[A.shells[ma]].L); ++a)
                        for (size_t mb = 0; mb < B.shells.size(); ++mb)
                            for (int c = 0; c < ncart(b.shells[B.shells[mb]].L); ++c) {
                                const int m = (int)(ma * B.shells.size() + mb);
                                int n = 0;
                                for (int q = 0; q < nq; ++q) n += has[m][q] != 0;
                                const int lb = b.shells[B.shells[mb]].L;
                                n *= tc.c[b.shells[A.shells[ma]].L][lb].count[a * ncart(lb) + c];
                                w.emplace_back(-n, (int)w.size());
                            }
                std::sort(w.begin(), w.end());
                for (const auto& x : w) o.tab.push_back(x.second);
            }
            for (int m = 0; m < nm; ++m) {
                const TeamClass& k = tc.c[b.shells[A.shells[m / nb]].L][b.shells[B.shells[m % nb]].L];
                o.tab[m] = (int)o.tab.size();
                o.tab[2 * nm + m] = (int)o.coef.size();
                for (int q : seq) {
                    if (!has[m][q]) continue;
                    o.tab.push_back(place[q]);
                    o.coef.insert(o.coef.end(), cf[m].begin() + (size_t)q * k.ncoef,
                                  cf[m].begin() + (size_t)(q + 1) * k.ncoef);
                    ++o.tab[nm + m];
                }
                if (!same || A.shells[m / nb] >= B.shells[m % nb]) {
                    // primitive pairs of the shell pair by itself, as build_pair_data keeps them
                    double mx = 0.0;
                    for (double v : own[m]) mx = std::max(mx, v);
                    int n = 0;
                    for (double v : own[m]) n += v >= 0.0 && v >= kPrimPairCut * mx;
                    o.npp.push_back(n);
                }
            }
        }
    });
    std::vector<double> nnz(sd.ncls, 0.0), prim(sd.ncls, 0.0);
    size_t nh = 0, nc = 0, nt = 0;
    for (const Out& o : outs) {
        nh += o.hdr.size();
        nc += o.coef.size();
        nt += o.tab.size();
    }
    sd.hdr.reserve(nh);
    sd.coef.reserve(nc);
    sd.tab.reserve(nt);
    for (int p = 0; p < np; ++p) {
        Out& o = outs[p];
        SuperPair& d = sd.pairs[p];
        d.npp = (int)(o.hdr.size() / kTeamHdr);
        d.hdr = reinterpret_cast<const double*>(sd.hdr.size());
        d.coef = reinterpret_cast<const double*>(sd.coef.size());
        d.tab = reinterpret_cast<const int*>(sd.tab.size());
        nnz[sd.cls[p]] += (double)o.coef.size();
        prim[sd.cls[p]] += (double)d.npp;
        sd.hdr.insert(sd.hdr.end(), o.hdr.begin(), o.hdr.end());
        sd.coef.insert(sd.coef.end(), o.coef.begin(), o.coef.end());
        sd.tab.insert(sd.tab.end(), o.tab.begin(), o.tab.end());
        sd.member_npp.push_back(std::move(o.npp));
        o = Out();
    }
    sd.cls_work.assign(sd.ncls, {});
    sd.cls_npp.assign(sd.ncls, 0);
    for (int p = 0; p < np; ++p) {
        const SuperPair& d = sd.pairs[p];
        if (d.npp <= sd.cls_npp[sd.cls[p]]) continue;
        sd.cls_npp[sd.cls[p]] = d.npp;
        std::vector<int>& w = sd.cls_work[sd.cls[p]];
        w.clear();
        const int *tab = sd.tab.data() + (size_t)d.tab, *ty = sd.types.data() + (size_t)d.type;
        const int* order = tab + 3 * d.nmem + d.nA + d.nB;
        for (int x = 0; x < d.nA * d.nB; ++x) w.push_back(tab[d.nmem + (ty[order[x]] & 255)] * ((unsigned)ty[order[x]] >> 20));
    }
    sd.cls_nnz.resize(sd.ncls);
    for (int c = 0; c < sd.ncls; ++c) sd.cls_nnz[c] = prim[c] > 0 ? nnz[c] / prim[c] : 1.0;
    return sd;
}

namespace {

// FP64 instructions of one primitive quartet's Boys function and R recursion.
double team_r_cost(int L) { return 36.0 + 3.0 * L + 1.7 * team_nherm(L) * (L + 3) / 4.0 * (L > 0); }

struct Geometry {
    int nr, nkb, slots, nw, slice, parts;
};

// FP64 instructions of the steps of one quartet class: per primitive quartet's
// R; the component pairs' work on either side, decreasing, for pairs of
// `nket` / `nbra` primitive pairs.
struct StepCosts {
    double r;
    const std::vector<int>*ket, *bra;
    int nket, nbra;
};

// Batch sizes of a task on teams of `lanes` threads, with the slice within
// `cap` doubles where the smallest batch allows it.  One bra pair: the rows
// per batch with the fewest instructions per row; the threads of a round take
// items in decreasing work, so a round costs as much as its first one.
Geometry geometry(int L1, int L2, const SuperPair& bra, const SuperPair& ket, int rows, int npk, int nb, int maxrows, int lanes, int cap,
                  const StepCosts& c)
{
    const int nab = bra.nA * bra.nB, ncd = ket.nA * ket.nB, nmk = ket.nmem;
    auto slice_of = [&](int nr, int nkb, int nw, int slots, int parts) {
        return team_slice(L1, L2, bra.nA, bra.nB, ket.nA, ket.nB, nr, nkb, nw, slots, nb, parts, nmk);
    };
    Geometry g;
    auto group = [&](int n) { return n >= team_cd_group(ncd) * lanes ? team_cd_group(ncd) : 1; };
    if (nb > 1) {
        // several bra pairs: every primitive quartet of the task in one R
        // batch; rounds of as many bra pairs as the slice holds; the rows of
        // a bra pair shared by several threads where its block alone leaves
        // threads idle
        auto parts = [&](int slots) {
            int p = 1;
            while (2 * p <= std::min(maxrows, 16) && p * slots * nab * ncd < 2 * lanes) p *= 2;
            return p;
        };
        g.nr = rows;
        g.nkb = npk;
        g.slots = 1;
        auto fits = [&](int s) {
            return slice_of(rows, npk, s * maxrows, s, parts(s)) <= cap;
        };
        while (g.slots < nb && fits(g.slots + 1)) ++g.slots;
        const int rounds = (nb + g.slots - 1) / g.slots;
        g.slots = (nb + rounds - 1) / rounds;
        g.nw = g.slots * maxrows;
        g.parts = parts(g.slots);
    } else {
        const int H1 = team_nherm(L1), J = H1 == 1 ? 1 : team_tuv_group(H1), ng = (H1 + J - 1) / J;
        double least = -1.0;
        g.slots = 1;
        for (int nblk = 1; nblk <= npk; nblk = nblk < 4 ? nblk + 1 : nblk * 3 / 2) {
            const int nkb = (npk + nblk - 1) / nblk;
            const bool last = nblk * 3 / 2 > npk;
            for (int r = 1; r <= std::min(rows, 64); ++r) {
                bool fits = false;
                for (int p = 1; p <= std::min(r, 8); p *= 2) {
                    const int size = slice_of(r, nkb, r, 1, p);
                    if (size > cap && !(last && r == 1 && least < 0.0)) break;
                    fits = true;
                    double w = nblk * ((double)((r * nkb + lanes - 1) / lanes) * c.r + 20.0);
                    for (int x = 0; x < ncd * r * ng; x += lanes)
                        w += (double)J * (*c.ket)[x / (r * ng)] * npk / c.nket + 2.0 * nblk;
                    const int JC = group(nab * ncd * p), per = ncd / JC * p;
                    for (int x = 0; x < nab * per; x += lanes)
                        w += (double)JC * (*c.bra)[x / per] / c.nbra * ((r + p - 1) / p) + 2.0;
                    w = w * ((rows + r - 1) / r) + (double)(p - 1) * ((nab * ncd + lanes - 1) / lanes);
                    if (least < 0.0 || w < 0.995 * least) {
                        least = w;
                        g.nr = g.nw = r;
                        g.nkb = nkb;
                        g.parts = p;
                    }
                }
                if (!fits) break;
            }
            if (nblk > 40 && least > 0.0) break;
        }
        if (least < 0.0) {
            g.nr = g.nw = g.parts = 1;
            g.nkb = 1;
        }
    }
    g.slice = slice_of(g.nr, g.nkb, g.nw, g.slots, g.parts);
    return g;
}

template <typename U, typename F>
void group_tasks(TeamPlanHost& plan, const SuperData& sd, const std::vector<U>& units, F&& total_L)
{
    // launch groups: (compiled L, team, slice tier); tasks by decreasing cost
    static const int tiers[] = {1024, 1536, 2048, 3072, 4096, 5120, 8192, 12800, 28000};
    struct Ref {
        int unit, at;
    };
    std::map<std::tuple<int, int, int>, std::pair<std::vector<Ref>, int>> groups;
    for (size_t ui = 0; ui < units.size(); ++ui) {
        const auto& u = units[ui];
        int L = total_L(u);
        if (L > kTeamMaxRegL) L = -1;
        for (size_t x = 0; x < u.t.size(); ++x) {
            const int sl = std::abs(u.slice[x]);
            int tier = 0;
            while (tiers[tier] < sl && tier < 8) ++tier;
            auto& g = groups[{L, u.slice[x] < 0 ? 128 : 32, tier}];
            g.first.push_back(Ref{(int)ui, (int)x});
            g.second = std::max(g.second, sl);
        }
    }
    std::vector<std::tuple<double, const std::tuple<int, int, int>*, std::pair<std::vector<Ref>, int>*>> list;
    for (auto& kv : groups) {
        double c = 0.0;
        for (const Ref& r : kv.second.first) c += units[r.unit].cost[r.at];
        list.emplace_back(c, &kv.first, &kv.second);
    }
    std::stable_sort(list.begin(), list.end(), [](const auto& x, const auto& y) { return std::get<0>(x) > std::get<0>(y); });
    for (auto& e : list) {
        TeamGroup g{};
        g.L = std::get<0>(*std::get<1>(e));
        g.team = std::get<1>(*std::get<1>(e));
        g.slice = std::get<2>(e)->second;
        g.off = plan.tasks.size();
        std::vector<Ref>& refs = std::get<2>(e)->first;
        g.n = refs.size();
        g.cost = std::get<0>(e);
        std::vector<double> cost(refs.size());
        for (size_t x = 0; x < refs.size(); ++x) cost[x] = units[refs[x].unit].cost[refs[x].at];
        for (size_t x : order_by_cost_desc(cost)) {
            const TeamTask& t = units[refs[x].unit].t[refs[x].at];
            g.prims += (double)(t.i1 - t.i0) * sd.pairs[t.ket].npp;
            plan.tasks.push_back(t);
        }
        plan.groups.push_back(g);
    }
}

}  // namespace

TeamPlanHost build_team_plan(const SuperData& sd, const std::vector<double>& q, double cut, int nsm)
{
    TeamPlanHost plan;
    const int np = (int)sd.pairs.size();
    std::vector<int> cL(sd.ncls, 0), cab(sd.ncls, 0), sample(sd.ncls, 0);
    for (int p = 0; p < np; ++p) {
        cL[sd.cls[p]] = sd.pairs[p].L;
        cab[sd.cls[p]] = sd.pairs[p].nA * sd.pairs[p].nB;
        sample[sd.cls[p]] = p;
    }
    // per (molecule, class): its pairs by decreasing bound
    const int F = (int)sd.pbase.size() - 1;
    std::vector<int> start((size_t)F * sd.ncls + 1, 0);
    for (int p = 0; p < np; ++p)
        if (sd.pairs[p].npp > 0 && (q[p] > 0.0 || cut < 0.0))
            ++start[(size_t)sd.pairs[p].frag * sd.ncls + sd.cls[p] + 1];
    for (size_t i = 1; i < start.size(); ++i) start[i] += start[i - 1];
    plan.order.resize(start.back());
    {
        std::vector<int> at(start.begin(), start.end() - 1);
        for (int p = 0; p < np; ++p)
            if (sd.pairs[p].npp > 0 && (q[p] > 0.0 || cut < 0.0))
                plan.order[at[(size_t)sd.pairs[p].frag * sd.ncls + sd.cls[p]]++] = p;
        for (size_t c = 0; c + 1 < start.size(); ++c)
            std::stable_sort(plan.order.begin() + start[c], plan.order.begin() + start[c + 1],
                             [&](int x, int y) { return q[x] > q[y]; });
    }
    // calls f(bra class, ket class, first bra, bras, ket) for every ket
    auto kets = [&](int fr, int cb, int ck, auto&& f) {
        const int b0 = start[(size_t)fr * sd.ncls + cb], b1 = start[(size_t)fr * sd.ncls + cb + 1];
        const int k0 = start[(size_t)fr * sd.ncls + ck], k1 = start[(size_t)fr * sd.ncls + ck + 1];
        int n = b1 - b0;   // surviving bras: shrinks as the ket bound falls
        for (int k = k0; k < k1 && n > 0; ++k) {
            const int ket = plan.order[k];
            if (cut >= 0.0)
                while (n > 0 && q[plan.order[b0 + n - 1]] * q[ket] < cut) --n;
            const int m = cb == ck ? std::min(n, k - k0 + 1) : n;
            if (m > 0) f(b0, m, ket);
        }
    };
    struct Unit {
        int fr, cb, ck;
        std::vector<TeamTask> t;
        std::vector<double> cost;
        std::vector<int> slice;   // negative: team of 128
        double total = 0.0;
    };
    std::vector<Unit> units;
    // cost of a primitive quartet, a bra primitive pair and a quartet
    auto costs = [&](const Unit& u, double* prim, double* row, double* quartet) {
        *prim = team_r_cost(cL[u.cb] + cL[u.ck]) + sd.cls_nnz[u.ck] * team_nherm(cL[u.cb]);
        *row = sd.cls_nnz[u.cb] * cab[u.ck];
        *quartet = 8.0 * cab[u.cb] * cab[u.ck];
    };
    for (int fr = 0; fr < F; ++fr)
        for (int i = 0; i < sd.ncls; ++i)
            for (int j = 0; j <= i; ++j) {
                const size_t b = (size_t)fr * sd.ncls + i, k = (size_t)fr * sd.ncls + j;
                if (start[b + 1] == start[b] || start[k + 1] == start[k]) continue;
                // the ket transform costs (ket coefficients) x (bra Hermite
                // functions) per primitive quartet, the bra transform (bra
                // coefficients) x (ket component pairs) per bra primitive
                // pair: the sides that cost less for the longest pairs
                Unit u, v;
                u.fr = v.fr = fr;
                u.cb = v.ck = i;
                u.ck = v.cb = j;
                auto whole = [&](const Unit& x) {
                    double cp, cr, cq;
                    costs(x, &cp, &cr, &cq);
                    return (double)sd.cls_npp[x.cb] * (sd.cls_npp[x.ck] * cp + cr);
                };
                units.push_back(whole(v) < whole(u) ? v : u);
            }
    // starting a thread costs 20-30 us: small molecules are planned on this one
    const int threads = np < 128 ? 1 : np < 256 ? 4 : 16;
    host_parallel_for((int)units.size(), [&](int i) {
        Unit& u = units[i];
        double cp, cr, cq;
        costs(u, &cp, &cr, &cq);
        kets(u.fr, u.cb, u.ck, [&](int b0, int m, int ket) {
            double rows = 0.0;
            for (int s = 0; s < m; ++s) rows += sd.pairs[plan.order[b0 + s]].npp;
            u.total += rows * sd.pairs[ket].npp * cp + rows * cr + m * cq;
        });
    }, threads);
    double total = 0.0;
    for (const Unit& u : units) total += u.total;
    // about 24 tasks for each of eight warps per SM, none below 40000
    // instructions (1250 per lane)
    const double target = std::max(4.0e4, total / (nsm * 8.0 * 24.0));
    const bool few = total < nsm * 8.0 * 6.0 * 6.0e4;   // small systems: teams of 128 for latency
    host_parallel_for((int)units.size(), [&](int i) {
        Unit& u = units[i];
        double cp, cr, cq;
        costs(u, &cp, &cr, &cq);
        const int L1 = cL[u.cb], L2 = cL[u.ck], nab = cab[u.cb], ncd = cab[u.ck], nout = nab * ncd;
        const SuperPair &bra = sd.pairs[sample[u.cb]], &ket = sd.pairs[sample[u.ck]];
        const int HS = team_nherm(L1 + L2) | 1, H1 = team_nherm(L1);
        const long long maxR = L1 + L2 > kTeamMaxRegL ? 3072 : 6144;
        // primitive quartets of a task of several bra pairs, and of the bra
        // pairs that get a task of their own: more where R is short
        const int batch = HS <= 11 && !few ? 128 : 64, alone = HS <= 11 && !few ? 96 : 40;
        const StepCosts sc{team_r_cost(L1 + L2), &sd.cls_work[u.ck], &sd.cls_work[u.cb], sd.cls_npp[u.ck], sd.cls_npp[u.cb]};
        // batch sizes repeat within a class pair: kept by the lengths they follow from
        std::unordered_map<unsigned long long, std::pair<Geometry, int>> known;
        auto pick = [&](int rows, int npk, int nb, int maxrows, double cost, int* team) {
            const bool large = cost > 1.5 * target;
            const unsigned long long key = (unsigned long long)rows << 40 | (unsigned long long)npk << 24 |
                                           (unsigned long long)nb << 17 | (unsigned long long)maxrows << 1 | large;
            auto it = known.find(key);
            if (it == known.end()) {
                const int cap32 = std::max(2800, 34 * HS + ncd * H1 + nout + 200);
                std::pair<Geometry, int> v(geometry(L1, L2, bra, ket, rows, npk, nb, maxrows, 32, cap32, sc), 32);
                if (v.first.slice > 4096 || few || large)
                    v = {geometry(L1, L2, bra, ket, rows, npk, nb, maxrows, 128, 9000, sc), 128};
                it = known.emplace(key, v).first;
            }
            *team = it->second.second;
            return it->second.first;
        };
        kets(u.fr, u.cb, u.ck, [&](int b0, int m, int ket) {
            const int npk = sd.pairs[ket].npp;
            int s = 0;
            while (s < m) {
                const int npb = sd.pairs[plan.order[b0 + s]].npp;
                TeamTask t{};
                t.ket = ket;
                t.b0 = b0 + s;
                int team;
                if ((long long)npb * npk >= alone || (long long)HS * npb * npk > maxR || npb * ncd * H1 > 4096) {
                    // one bra pair, its rows tiled to the target cost
                    const double one = (double)npk * cp + cr;
                    int per = (int)std::min<double>(npb, std::max(1.0, (target - cq) / one));
                    const int tiles = (npb + per - 1) / per;
                    per = (npb + tiles - 1) / tiles;
                    const Geometry g = pick(per, npk, 1, per, per * one + cq, &team);
                    per = std::min(npb, (per + g.nr - 1) / g.nr * g.nr);
                    t.nb = 1;
                    t.nr = (unsigned short)g.nr;
                    t.nkb = (unsigned short)g.nkb;
                    t.slots = 1;
                    t.nw = (unsigned short)g.nw;
                    t.parts = (unsigned short)g.parts;
                    for (int r = 0; r < npb; r += per) {
                        t.i0 = (unsigned short)r;
                        t.i1 = (unsigned short)std::min(npb, r + per);
                        u.t.push_back(t);
                        u.cost.push_back((t.i1 - t.i0) * one + cq);
                        u.slice.push_back(team == 32 ? g.slice : -g.slice);
                    }
                    ++s;
                    continue;
                }
                // several bra pairs in one task
                int n = 0, rows = 0, maxrows = 0;
                double cost = 0.0;
                while (s + n < m && n < 64) {
                    const int r = sd.pairs[plan.order[b0 + s + n]].npp;
                    if (n > 0 && ((rows + r) * npk > batch || (long long)HS * (rows + r) * npk > maxR || cost > target ||
                                  (long long)r * npk >= alone || r * ncd * H1 > 4096))
                        break;
                    rows += r;
                    maxrows = std::max(maxrows, r);
                    cost += r * npk * cp + r * cr + cq;
                    ++n;
                }
                const Geometry g = pick(rows, npk, n, maxrows, cost, &team);
                t.nb = (unsigned short)n;
                t.i0 = 0;
                t.i1 = (unsigned short)rows;
                t.nr = (unsigned short)g.nr;
                t.nkb = (unsigned short)g.nkb;
                t.slots = (unsigned short)g.slots;
                t.nw = (unsigned short)g.nw;
                t.parts = (unsigned short)g.parts;
                u.t.push_back(t);
                u.cost.push_back(cost);
                u.slice.push_back(team == 32 ? g.slice : -g.slice);
                s += n;
            }
        });
    }, threads);
    group_tasks(plan, sd, units, [&](const Unit& u) { return cL[u.cb] + cL[u.ck]; });
    return plan;
}

TeamPlanHost build_team_diagonal(const SuperData& sd, int nsm)
{
    TeamPlanHost plan;
    const int np = (int)sd.pairs.size();
    plan.order.resize(np);
    std::iota(plan.order.begin(), plan.order.end(), 0);
    plan.first.assign(1, 0);
    struct Unit {
        int L;
        std::vector<TeamTask> t;
        std::vector<double> cost;
        std::vector<int> slice;
    };
    std::vector<Unit> units(2 * kMaxLTot + 1);
    std::vector<double> one(np);
    double total = 0.0;
    for (int p = 0; p < np; ++p) {
        const SuperPair& d = sd.pairs[p];
        const double nnz = sd.cls_nnz[sd.cls[p]];
        one[p] = d.npp * (team_r_cost(2 * d.L) + nnz * team_nherm(d.L)) + nnz;
        total += one[p] * d.npp;
    }
    const double target = std::max(4.0e4, total / (nsm * 8.0 * 4.0));
    for (int p = 0; p < np; ++p) {
        const SuperPair& d = sd.pairs[p];
        const double nnz = sd.cls_nnz[sd.cls[p]];
        const int nab = d.nA * d.nB, HS = team_nherm(2 * d.L) | 1;
        Unit& u = units[2 * d.L];
        u.L = 2 * d.L;
        int per = (int)std::min<double>(d.npp, std::max(1.0, target / one[p]));
        const int c = sd.cls[p];
        const StepCosts sc{team_r_cost(2 * d.L), &sd.cls_work[c], &sd.cls_work[c], sd.cls_npp[c], sd.cls_npp[c]};
        int team = 32;
        Geometry g = geometry(d.L, d.L, d, d, per, d.npp, 1, per, 32,
                              std::max(2800, 34 * HS + nab * team_nherm(d.L) + nab * nab + 200), sc);
        if (g.slice > 4096 || one[p] > target) {
            team = 128;
            g = geometry(d.L, d.L, d, d, per, d.npp, 1, per, 128, 9000, sc);
        }
        per = std::min(d.npp, (per + g.nr - 1) / g.nr * g.nr);
        TeamTask t{};
        t.ket = t.b0 = p;
        t.nb = t.slots = 1;
        t.nr = t.nw = (unsigned short)g.nr;
        t.nkb = (unsigned short)g.nkb;
        t.parts = (unsigned short)g.parts;
        int out = plan.first.back();
        for (int r = 0; r < d.npp; r += per) {
            t.i0 = (unsigned short)r;
            t.i1 = (unsigned short)std::min(d.npp, r + per);
            t.out = out;
            out += nab;
            u.t.push_back(t);
            u.cost.push_back((t.i1 - t.i0) * one[p]);
            u.slice.push_back(team == 32 ? g.slice : -g.slice);
        }
        plan.first.push_back(out);
    }
    group_tasks(plan, sd, units, [](const Unit& u) { return u.L; });
    return plan;
}

const std::vector<double>& team_boys_host()
{
    static const std::vector<double> tab = [] {
        constexpr int M = kTeamBoysMaxL + 5;
        std::vector<double> v((size_t)(kTeamBoysMaxL + 1) * kTeamBoysN * 8, 0.0);
        std::vector<long double> F(M + 1);
        for (int k = 0; k < kTeamBoysN; ++k) {
            const long double T = (long double)k / kTeamBoysInv, e = expl(-T);
            // F_M by its ascending series (positive terms), then downward
            long double term = 1.0L / (2 * M + 1), sum = term;
            for (int i = 1; i < 400 && term > 1e-22L * sum; ++i) {
                term *= 2.0L * T / (2 * M + 2 * i + 1);
                sum += term;
            }
            F[M] = e * sum;
            for (int m = M - 1; m >= 0; --m) F[m] = (2.0L * T * F[m + 1] + e) / (2 * m + 1);
            for (int L = 0; L <= kTeamBoysMaxL; ++L) {
                double* r = &v[((size_t)L * kTeamBoysN + k) * 8];
                long double fac = 1.0L;
                for (int j = 0; j < 6; ++j) {
                    r[j] = (double)(F[L + j] / fac);
                    fac *= j + 1;
                }
                r[6] = (double)e;
            }
        }
        return v;
    }();
    return tab;
}

}  // namespace hfx
