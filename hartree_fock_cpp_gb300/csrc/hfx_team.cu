// hfx_team.cu -- FP64 Fock build over super shells: one team of threads (a
// warp, or a CTA of 128) per task of one ket super pair and one or several
// bra super pairs.
//
// What bounds it: the FP64 pipe of this GPU issues one warp instruction every
// 16 cycles per SM, 1/64 of the FP32 rate, while shared memory, integer and
// load instructions run at full rate.  So the kernel spends everything else
// freely to execute as few FP64 instructions as possible, each with all 32
// lanes: index arithmetic is generic (any angular momenta and contractions,
// through tables), and each of the four steps lays its own outputs over the
// threads:
//   1. R_tuv of every (bra, ket) primitive quartet of a batch, one per thread
//      (up to kTeamMaxRegL in registers, every index a compile-time constant;
//      beyond that level by level over the team)
//   2. W[row][cd][tuv] = sum over the ket primitive pairs: outputs ordered so
//      that a warp's lanes share cd, hence trip count and coefficients
//   3. (ab|cd) += bra coefficients x W
//   4. digestion: each J / K element that the quartet touches is summed over
//      the block and added with one atomic
// Fock builds against the FP64 shell-quartet kernels before it (ms): benzene /
// cc-pVDZ 17.9 -> 7.7, n-decane / 6-31G* 16.7 -> 14.0, NaCl / cc-pVTZ 19.7 ->
// 3.3, water / cc-pVTZ UHF 8.1 -> 0.89 (there one warp evaluated a whole
// contracted f quartet); 114 M FP64 warp instructions for benzene, 21 of 32
// lanes active (R 34 M at 23 lanes, step 2 47 M at 22, step 3 21 M at 18, the
// digestion 12 M at 15).  Schwarz pass of NaCl / cc-pVTZ 35 -> 0.9 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "hfx_class.cuh"
#include "hfx_smem.hpp"
#include "hfx_team.hpp"

namespace hfx {

namespace {

constexpr int kNb = 456;          // recursion neighbours (ints; general form only)
// shared-memory header: the work-queue box, in the general form the neighbours
__host__ __device__ constexpr int team_header(int LC) { return LC < 0 ? 4 * kNb + 64 : 16; }

template <int TEAM>
__device__ __forceinline__ void team_sync()
{
    if constexpr (TEAM == 32)
        __syncwarp();
    else
        __syncthreads();
}

// o / n for 0 <= o < 2^20: inv = 1/n rounded, one correction either way
__device__ __forceinline__ int fdiv(int o, int n, float inv)
{
    int q = (int)((float)o * inv);
    const int r = o - q * n;
    q += (r >= n) - (r < 0);
    return q;
}

// +-v for an odd flag: the sign bit flipped on the integer pipe
__device__ __forceinline__ double flip(double v, int odd)
{
    return __hiloint2double(__double2hiint(v) ^ (odd << 31), __double2loint(v));
}

// v * 2^n, n in 0..3, on the integer pipe (zero and denormals by multiplication)
__device__ __forceinline__ double times_pow2(double v, int n)
{
    const int hi = __double2hiint(v);
    if ((hi & 0x7ff00000) == 0) return v * (double)(1 << n);
    return __hiloint2double(hi + (n << 20), __double2loint(v));
}

// T's table cell k = round(64 T) and nd = T_k - T without conversions
// (adding 1.5 2^52 leaves the rounded integer in the low word)
__device__ __forceinline__ int boys_cell(double T, double& nd)
{
    const double magic = 6755399441055744.0;
    const double t = fma(T, (double)kTeamBoysInv, magic);
    nd = fma(t - magic, 1.0 / kTeamBoysInv, -T);
    return __double2loint(t);
}

// F_L(T) and e^{-T} (only needed for L > 0) from the table row of (L, k)
template <bool EXP>
__device__ __forceinline__ void boys_row(const double* __restrict__ row, double nd, double& F, double& e)
{
    const double2* r2 = reinterpret_cast<const double2*>(row);
    const double2 c0 = __ldg(r2), c1 = __ldg(r2 + 1), c2 = __ldg(r2 + 2);
    double r = c2.y;
    r = fma(r, nd, c2.x);
    r = fma(r, nd, c1.y);
    r = fma(r, nd, c1.x);
    r = fma(r, nd, c0.y);
    F = fma(r, nd, c0.x);
    if constexpr (EXP) {
        double x = 1.0 / 720.0;
        x = fma(x, nd, 1.0 / 120.0);
        x = fma(x, nd, 1.0 / 24.0);
        x = fma(x, nd, 1.0 / 6.0);
        x = fma(x, nd, 0.5);
        x = fma(x, nd, 1.0);
        x = fma(x, nd, 1.0);
        e = __ldg(row + 6) * x;
    }
}

__device__ __forceinline__ bool beyond_table(double T)
{
    return __double2hiint(T) >= 0x40480000;   // T >= 48 (T >= 0)
}
static_assert(kTeamBoysTMax == 48, "beyond_table compares with the high word of 48.0");

struct Prim {
    double X, Y, Z, R2, rho, T, pref;
};
__device__ __forceinline__ Prim prim_quartet(const double* __restrict__ b, const double* __restrict__ k)
{
    const double2 b0 = __ldg((const double2*)b), b1 = __ldg((const double2*)b + 1), b2 = __ldg((const double2*)b + 2);
    const double2 k0 = __ldg((const double2*)k), k1 = __ldg((const double2*)k + 1), k2 = __ldg((const double2*)k + 2);
    Prim p;
    p.X = b0.y - k0.y;
    p.Y = b1.x - k1.x;
    p.Z = b1.y - k1.y;
    const double rs = rsqrt(b0.x + k0.x);
    p.rho = b0.x * k0.x * (rs * rs);
    p.R2 = fma(p.Z, p.Z, fma(p.Y, p.Y, p.X * p.X));
    p.T = p.rho * p.R2;
    p.pref = b2.x * k2.x * rs;   // 2 pi^{5/2} / (p q sqrt(p + q))
    return p;
}

// (2L-1)!! / 2^{L+1} sqrt(pi): F_L(T) = this / T^{L+1/2} beyond the table
__host__ __device__ constexpr double boys_far(int L)
{
    double v = 0.88622692545275801365;
    for (int m = 0; m < L; ++m) v *= 0.5 * (2 * m + 1);
    return v;
}

// Seeds s_m = pref (-2 rho)^m F_m(T), m = 0..L, downward from F_L:
// s_m = (pref e^{-T} (-2 rho)^m - R^2 s_{m+1}) / (2m+1), both terms of one
// sign.  Beyond the table F_L is asymptotic and e^{-T} < 2e-21 is left out;
// only F_L is behind the branch (lanes of a warp mostly differ in it).
template <int L>
__device__ __forceinline__ void seeds(const Prim& p, const double* __restrict__ tab, double (&s)[L + 1])
{
    double F, e = 0.0;
    if (!beyond_table(p.T)) {
        double nd;
        const int k = boys_cell(p.T, nd);
        boys_row<(L > 0)>(tab + ((size_t)L * kTeamBoysN + k) * 8, nd, F, e);
    } else {
        const double rs = rsqrt(p.T), r2 = rs * rs;
        F = boys_far(L) * rs;
#pragma unroll
        for (int m = 0; m < L; ++m) F *= r2;
    }
    if constexpr (L == 0) {
        s[0] = p.pref * F;
    } else {
        const double m2r = -2.0 * p.rho;
        double pe[L];
        pe[0] = p.pref * e;
        double pw = p.pref * m2r;
#pragma unroll
        for (int m = 1; m < L; ++m) {
            pe[m] = pe[m - 1] * m2r;
            pw *= m2r;
        }
        s[L] = pw * F;
#pragma unroll
        for (int m = L - 1; m >= 0; --m) s[m] = fma(-p.R2, s[m + 1], pe[m]) * (1.0 / (2 * m + 1));
    }
}

__constant__ double c_team_inv_odd[12] = {1.0,      1.0 / 3,  1.0 / 5,  1.0 / 7,  1.0 / 9,  1.0 / 11,
                                          1.0 / 13, 1.0 / 15, 1.0 / 17, 1.0 / 19, 1.0 / 21, 1.0 / 23};

// Seeds for a runtime L into S[m * stride]; beyond the table with e^{-T}.
__device__ void seeds_any(const Prim& p, int L, const double* __restrict__ tab, double* S, int stride)
{
    const double m2r = -2.0 * p.rho;
    if (!beyond_table(p.T)) {
        double nd, F, e;
        const int k = boys_cell(p.T, nd);
        boys_row<true>(tab + ((size_t)L * kTeamBoysN + k) * 8, nd, F, e);
        double pw = p.pref;
        for (int m = 0; m < L; ++m) {
            S[m * stride] = pw * e;
            pw *= m2r;
        }
        double s = pw * F;
        S[L * stride] = s;
        for (int m = L - 1; m >= 0; --m) {
            s = fma(-p.R2, s, S[m * stride]) * c_team_inv_odd[m];
            S[m * stride] = s;
        }
    } else {
        const double rs = rsqrt(p.T), e = exp(-p.T), inv2T = 0.5 * rs * rs;
        double F = 0.88622692545275801365 * rs, pw = p.pref;
        S[0] = pw * F;
        for (int m = 0; m < L; ++m) {
            F = ((2 * m + 1) * F - e) * inv2T;
            pw *= m2r;
            S[(m + 1) * stride] = pw * F;
        }
    }
}

__device__ __forceinline__ long long tri(int a, int b)
{
    const int hi = a > b ? a : b, lo = a > b ? b : a;
    return (long long)hi * (hi + 1) / 2 + lo;
}

// First entry of a sorted list of n primitive indices that is not below v.
__device__ __forceinline__ int first_at_least(const int* __restrict__ list, int n, int v)
{
    int lo = 0;
    while (lo < n) {
        const int mid = (lo + n) >> 1;
        if (__ldg(list + mid) < v)
            lo = mid + 1;
        else
            n = mid;
    }
    return lo;
}

// LC: compiled total angular momentum, or -1 for any L.
template <int LC, int TEAM>
__global__ void __launch_bounds__(TEAM, TEAM == 32 ? 16 : 4) k_team(TeamArgs a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    int* box = reinterpret_cast<int*>(smem);
    int* nbt = reinterpret_cast<int*>(smem + 64);
    const int tid = threadIdx.x;
    double* sl = reinterpret_cast<double*>(smem + team_header(LC));
    if constexpr (LC < 0) {
        // recursion neighbours: axis, the two lower entries, the second one's factor
        for (int e = threadIdx.x; e < 455; e += blockDim.x) {
            int s = 0;
            while (team_nherm(s) <= e) ++s;
            int o = e - (s == 0 ? 0 : team_nherm(s - 1)), t = 0;
            while (o >= s - t + 1) {
                o -= s - t + 1;
                ++t;
            }
            const int u = o, v = s - t - u;
            int w = 0;
            if (s > 0) {
                const int d = t > 0 ? 0 : u > 0 ? 1 : 2;
                const int c = (d == 0 ? t : d == 1 ? u : v) - 1;
                const int i1 = herm_index(t - (d == 0), u - (d == 1), v - (d == 2));
                const int i2 = c > 0 ? herm_index(t - 2 * (d == 0), u - 2 * (d == 1), v - 2 * (d == 2)) : 0;
                w = d | i1 << 2 | i2 << 11 | c << 20;
            }
            nbt[e] = w;
        }
        __syncthreads();
    }

    while (true) {
        int tk = 0;
        if (TEAM == 32) {
            if (tid == 0) tk = atomicAdd(a.counter, 1);
            tk = __shfl_sync(0xffffffffu, tk, 0);
        } else {
            __syncthreads();
            if (tid == 0) *box = atomicAdd(a.counter, 1);
            __syncthreads();
            tk = *box;
        }
        if (tk >= a.ntasks) break;
        const TeamTask t = a.tasks[tk];
        const SuperPair& ket = a.pairs[t.ket];
        if (a.active && !__ldg(a.active + ket.frag)) continue;
        const SuperPair& bra0 = a.pairs[a.order[t.b0]];
        const int L1 = bra0.L, L2 = ket.L, L = LC >= 0 ? LC : L1 + L2;
        const int HL = team_nherm(L), HS = HL | 1, H1 = team_nherm(L1);
        const int nA = bra0.nA, nB = bra0.nB, nC = ket.nA, nD = ket.nB, nab = nA * nB, ncd = nC * nD, nout = nab * ncd;
        const int nmb = bra0.nmem, nmk = ket.nmem, npk = ket.npp, nfb = nA + nB;
        const int As = nout | 1;                        // odd strides of bra blocks and W rows: no bank conflicts
        double* acc = sl;
        double* W = acc + t.parts * t.slots * As;
        double* R = W + team_w(H1, nA, nB, nC, nD, t.nw, t.slots);
        double* R2 = R + t.nr * t.nkb * HS;                                     // second buffer and seeds (general L)
        double* S = R2 + (LC < 0 && L > kTeamMaxRegL ? t.nr * t.nkb * HS : 0);
        int* rowd = reinterpret_cast<int*>(S + (LC < 0 && L > kTeamMaxRegL ? (L + 1) * t.nr * t.nkb : 0));
        int* rstart = rowd + t.nr;
        int* bid = rstart + t.nb + 1;              // pair of each bra
        int* kmem = bid + t.nb;                    // ket members: list start, length, coefficients, class | count << 16,
                                                   // first and last list entry
        int* kfn = kmem + 6 * nmk;                 // ket function indices
        int* border = kfn + nC + nD;               // component pairs by decreasing work
        int* korder = border + nab;
        int* bfn = korder + ncd;                   // function indices of the round's bra pairs
        const bool single = t.nb == 1;
        {
            const int* tab = ket.tab;
            const int* ty = ket.type + ncd;
            for (int m = tid; m < nmk; m += TEAM) {
                const int ls = __ldg(tab + m), lc = __ldg(tab + nmk + m);
                kmem[6 * m] = ls;
                kmem[6 * m + 1] = lc;
                kmem[6 * m + 2] = __ldg(tab + 2 * nmk + m);
                kmem[6 * m + 3] = __ldg(ty + m) | __ldg(ty + nmk + m) << 16;
                kmem[6 * m + 4] = lc > 0 ? __ldg(tab + ls) : 0;
                kmem[6 * m + 5] = lc > 0 ? __ldg(tab + ls + lc - 1) : -1;
            }
            for (int m = tid; m < nC + nD; m += TEAM) kfn[m] = __ldg(tab + 3 * nmk + m);
            for (int m = tid; m < t.nb; m += TEAM) bid[m] = a.order[t.b0 + m];
        }

        // Component pairs in use, by decreasing work: those of the members
        // that can reach the cut with the task's largest bra pair (the first)
        // resp. with the ket pair (single bra pair).  The others' integrals
        // stay zero: each is below the cut.
        const double cut = a.mode == kTeamDiag ? -1.0 : a.mixed ? ket.cut32 : a.thr;
        auto in_use = [&](const SuperPair& s, int nfn, int n, double other, double cut, int step, int* list) {
            const int* seq = s.tab + 3 * s.nmem + nfn;
            int got = 0;
            for (int x0 = 0; x0 < n; x0 += 32) {
                const int x = x0 + (tid & 31), v = x < n ? __ldg(seq + x) : 0;
                const bool use = x < n && (cut <= 0.0 || __ldg(s.mq + (__ldg(s.type + v) & 255)) * other >= cut);
                const unsigned m = __ballot_sync(0xffffffffu, use);
                if (use) list[got + __popc(m & ((1u << (tid & 31)) - 1u))] = v;
                got += __popc(m);
            }
            // up to a whole group of `step` component pairs, with ones not in use
            for (int x = 0; x < n && got % step; ++x) {
                const int v = __ldg(seq + x);
                if (cut > 0.0 && __ldg(s.mq + (__ldg(s.type + v) & 255)) * other < cut) list[got++] = v;
            }
            return got;
        };
        const int nce = in_use(ket, nC + nD, ncd, bra0.qmax, cut, team_cd_group(ncd), korder);
        const int nae = in_use(bra0, nfb, nab, ket.qmax, single ? cut : -1.0, 1, border);
        const int Ws = (nce * H1) | 1;
        if (nce < ncd || nae < nab)
            for (int x = tid; x < t.parts * t.slots * As; x += TEAM) acc[x] = 0.0;

        // rows of the task: (bra slot, bra primitive pair); a bra pair whose
        // quartet the density screen drops gets no rows
        auto negligible = [&](const SuperPair& b) {
            if (!a.dscreen) return false;
            const double* D = a.Dsh + ket.pbase;
            double d = fmax(a.Dsh[b.id], a.Dsh[ket.id]);
            d = fmax(d, D[shell_pair_id(b.shA, ket.shA)]);
            d = fmax(d, D[shell_pair_id(b.shA, ket.shB)]);
            d = fmax(d, D[shell_pair_id(b.shB, ket.shA)]);
            d = fmax(d, D[shell_pair_id(b.shB, ket.shB)]);
            return b.qmax * ket.qmax * d < a.dthr;
        };
        int nrows;
        if (single) {
            team_sync<TEAM>();
            if (negligible(bra0)) continue;
            nrows = t.i1 - t.i0;
        } else {
            team_sync<TEAM>();
            if (tid < 32) {
                int at = 0;
                for (int s0 = 0; s0 < t.nb; s0 += 32) {
                    const int s = s0 + tid;
                    int n = 0;
                    if (s < t.nb) {
                        const SuperPair& b = a.pairs[bid[s]];
                        n = negligible(b) ? 0 : b.npp;
                    }
                    int incl = n;
                    for (int d = 1; d < 32; d <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, incl, d);
                        if (tid >= d) incl += v;
                    }
                    if (s < t.nb) {
                        rstart[s] = at + incl - n;
                        for (int r = 0; r < n; ++r) rowd[at + incl - n + r] = s << 16 | r;
                    }
                    at += __shfl_sync(0xffffffffu, incl, 31);
                }
                if (tid == 0) rstart[t.nb] = at;
            }
            team_sync<TEAM>();
            nrows = rstart[t.nb];
            if (nrows == 0) {
                team_sync<TEAM>();   // rstart is read before the next task writes it
                continue;
            }
        }

        const double* khdr = ket.hdr;
        const int* ktab = ket.tab;
        const double* kcoef = ket.coef;
        const int* ktype = ket.type;
        const int* btype = bra0.type;
        const double* bhdr0 = bra0.hdr;
        const uint4* ridx = a.ridx + a.ridx_at[L1 * 7 + L2];

        // step 1: R of rows [r0, r0 + nr) against ket primitive pairs [k0, k0 + nk)
        auto make_R = [&](int r0, int nr, int k0, int nk) {
            const int n = nr * nk;
            const float ink = 1.0f / nk;
            for (int x = tid; x < n; x += TEAM) {
                const int row = fdiv(x, nk, ink), kl = x - row * nk;
                const double* bh;
                if (single) {
                    bh = bhdr0 + (size_t)(t.i0 + r0 + row) * kTeamHdr;
                } else {
                    const int d = rowd[row];
                    bh = a.pairs[bid[d >> 16]].hdr + (size_t)(d & 0xffff) * kTeamHdr;
                }
                const Prim p = prim_quartet(bh, khdr + (size_t)(k0 + kl) * kTeamHdr);
                if constexpr (LC >= 0) {
                    double sd[LC + 1], Rr[c_nh(LC)];
                    seeds<LC>(p, a.boys, sd);
                    hermite_R<double, LC>(p.X, p.Y, p.Z, sd, Rr);
                    double* o = R + x * HS;
#pragma unroll
                    for (int e = 0; e < c_nh(LC); ++e) o[e] = Rr[e];
                } else {
                    seeds_any(p, L, a.boys, S + x, n);
                }
            }
            if constexpr (LC < 0) {
                // level by level: buffers alternate so that the last level lands in R
                team_sync<TEAM>();
                double* cur = (L & 1) ? R : R2;
                double* nxt = (L & 1) ? R2 : R;
                for (int m = L; m >= 0; --m) {
                    const int cnt = team_nherm(L - m);
                    const float icnt = 1.0f / cnt;
                    for (int o = tid; o < n * cnt; o += TEAM) {
                        const int x = fdiv(o, cnt, icnt), e = o - x * cnt;
                        double v;
                        if (e == 0) {
                            v = S[m * n + x];
                        } else {
                            const int w = nbt[e];
                            const int d = w & 3, i1 = (w >> 2) & 511, i2 = (w >> 11) & 511, c = (w >> 20) & 15;
                            const int row = fdiv(x, nk, ink), kl = x - row * nk;
                            const double* bh;
                            if (single) {
                                bh = bhdr0 + (size_t)(t.i0 + r0 + row) * kTeamHdr;
                            } else {
                                const int q = rowd[row];
                                bh = a.pairs[bid[q >> 16]].hdr + (size_t)(q & 0xffff) * kTeamHdr;
                            }
                            const double xd = __ldg(bh + 1 + d) - __ldg(khdr + (size_t)(k0 + kl) * kTeamHdr + 1 + d);
                            v = xd * cur[x * HS + i1];
                            if (c) v = fma((double)c, cur[x * HS + i2], v);
                        }
                        nxt[x * HS + e] = v;
                    }
                    team_sync<TEAM>();
                    double* sw = cur;
                    cur = nxt;
                    nxt = sw;
                }
            }
            team_sync<TEAM>();
        };

        // step 2: W of batch rows [w0, w0 + nw) (stored from W's first row on)
        // from ket primitive pairs [k0, k0 + nk); first: store, else add.
        // A thread computes JT consecutive tuv of one (row, cd): the term's
        // coefficient and R offsets are read once for JT independent sums.
        auto make_W_j = [&](auto jt, int w0, int nw, int k0, int nk, bool first) {
            constexpr int JT = decltype(jt)::value;
            const int ng = (H1 + JT - 1) / JT;             // groups per row
            const int n = nce * nw * ng;
            const float ing = 1.0f / ng, inw = 1.0f / nw;
            for (int o = tid; o < n; o += TEAM) {
                const int q = fdiv(o, ng, ing), g = o - q * ng, cw = fdiv(q, nw, inw), row = q - cw * nw;
                const int cd = korder[cw];
                const unsigned fw = __ldg(ktype + cd);
                const int m = fw & 255, ko = (fw >> 8) & 4095, nc = fw >> 20;
                const int lc = kmem[6 * m + 1], cls = kmem[6 * m + 3] & 0xffff, nco = kmem[6 * m + 3] >> 16;
                const double* cf = kcoef + kmem[6 * m + 2] + ko;
                const int* list = ktab + kmem[6 * m];
                const short* codes = a.kcode + cls + ko;
                const double* Rr = R + (size_t)(w0 + row) * nk * HS;
                double s[JT];
#pragma unroll
                for (int j = 0; j < JT; ++j) s[j] = 0.0;
                const bool all = lc == npk;
                int e0 = k0, e1 = k0 + nk;
                if (!all) {
                    const int lo = kmem[6 * m + 4], hi = kmem[6 * m + 5];
                    e0 = lo >= k0 ? 0 : hi < k0 ? lc : first_at_least(list, lc, k0);
                    e1 = hi < k0 + nk ? lc : lo >= k0 + nk ? 0 : first_at_least(list, lc, k0 + nk);
                }
#pragma unroll 2
                for (int k = 0; k < nc; ++k) {
                    const int code = __ldg(codes + k), odd = (code >> 14) & 1, tnp = code & 16383;
                    const double* c = cf + (size_t)e0 * nco + k;
                    int ri[JT];
                    if constexpr (JT == 1) {
                        ri[0] = tnp;
                    } else {
                        const uint4 x = __ldg(ridx + tnp * ng + g);
                        const unsigned xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int j = 0; j < JT; ++j) ri[j] = (xs[j >> 1] >> (16 * (j & 1))) & 0xffff;
                    }
                    if (all) {
                        const double* Rk = Rr;
#pragma unroll 4
                        for (int e = e0; e < e1; ++e, c += nco, Rk += HS) {
                            const double cv = flip(__ldg(c), odd);
#pragma unroll
                            for (int j = 0; j < JT; ++j) s[j] = fma(cv, Rk[ri[j]], s[j]);
                        }
                    } else {
#pragma unroll 2
                        for (int e = e0; e < e1; ++e, c += nco) {
                            const double cv = flip(__ldg(c), odd);
                            const double* Rk = Rr + (__ldg(list + e) - k0) * HS;
#pragma unroll
                            for (int j = 0; j < JT; ++j) s[j] = fma(cv, Rk[ri[j]], s[j]);
                        }
                    }
                }
                double* w = W + row * Ws + g * JT * nce + cw;
#pragma unroll
                for (int j = 0; j < JT; ++j)
                    if (g * JT + j < H1) w[j * nce] = first ? s[j] : w[j * nce] + s[j];
            }
        };
        auto make_W = [&](int w0, int nw, int k0, int nk, bool first) {
            if (H1 == 1)
                make_W_j(CInt<1>{}, w0, nw, k0, nk, first);
            else if (team_tuv_group(H1) == 4)
                make_W_j(CInt<4>{}, w0, nw, k0, nk, first);
            else
                make_W_j(CInt<5>{}, w0, nw, k0, nk, first);
        };

        // step 3: bra transform of one bra pair's `rows` rows from W row w0
        // on, its primitive pairs [ij0, ij0 + rows), into JC consecutive
        // component pairs cd of one ab; first: store, else add
        auto bra_j = [&](auto jc, const SuperPair& bra, double* out, int ab, int cw, int w0, int ij0, int rows,
                         bool first, int part, int parts) {
            constexpr int JC = decltype(jc)::value;
            const unsigned fw = __ldg(btype + ab);
            const int m = fw & 255, ko = (fw >> 8) & 4095, nc = fw >> 20;
            const int* tab = bra.tab;
            const int ls = __ldg(tab + m), lc = __ldg(tab + nmb + m);
            const int cls = __ldg(btype + nab + m), nco = __ldg(btype + nab + nmb + m);
            const double* cf = bra.coef + __ldg(tab + 2 * nmb + m) + ko;
            const short* codes = a.kcode + cls + ko;
            const int* list = tab + ls;
            const bool all = lc == bra.npp;
            int e0 = all ? ij0 : 0, e1 = all ? ij0 + rows : lc;
            if (!all && rows < bra.npp) {
                e0 = first_at_least(list, lc, ij0);
                e1 = first_at_least(list, lc, ij0 + rows);
            }
            double s[JC];
#pragma unroll
            for (int j = 0; j < JC; ++j) s[j] = 0.0;
            for (int e = e0 + part; e < e1; e += parts) {
                const int r = (all ? e : __ldg(list + e)) - ij0;
                const double* w = W + (w0 + r) * Ws + cw;
                const double* c = cf + (size_t)e * nco;
#pragma unroll 4
                for (int k = 0; k < nc; ++k) {
                    const double cv = __ldg(c + k);
                    const double* wk = w + (__ldg(codes + k) & 16383) * nce;
#pragma unroll
                    for (int j = 0; j < JC; ++j) s[j] = fma(cv, wk[j], s[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < JC; ++j) {
                double* v = out + ab * ncd + korder[cw + j];
                *v = first ? s[j] : *v + s[j];
            }
        };
        // the bra transform of `ns` bra pairs (slots s0..) over the team
        auto make_acc = [&](int s0, int ns, int w0, bool first, int r0, int nr) {
            auto run = [&](auto jc) {
                constexpr int JC = decltype(jc)::value;
                // ab slowest: a warp's lanes share the bra coefficients' pattern
                const int ng = nce / JC, ngp = ng * t.parts, per = ns * ngp, n = nae * per;
                const float iper = 1.0f / per, ingp = 1.0f / ngp, ing = 1.0f / ng;
                for (int x = tid; x < n; x += TEAM) {
                    const int aw = fdiv(x, per, iper), y = x - aw * per, ab = border[aw];
                    const int s = fdiv(y, ngp, ingp), z = y - s * ngp, part = fdiv(z, ng, ing), g = z - part * ng;
                    const SuperPair& bra = single ? bra0 : a.pairs[bid[s0 + s]];
                    const int w = single ? 0 : rstart[s0 + s] - w0;
                    const int ij0 = single ? t.i0 + r0 : 0;
                    const int rows = single ? nr : rstart[s0 + s + 1] - rstart[s0 + s];
                    bra_j(jc, bra, acc + (part * t.slots + s) * As, ab, g * JC, w, ij0, rows, first, part, t.parts);
                }
            };
            // several component pairs per thread where that leaves no thread idle
            const int n = ns * nae * nce * t.parts;
            const int step = team_cd_group(ncd);
            if (step == 4 && n >= 4 * TEAM)
                run(CInt<4>{});
            else if (step == 3 && n >= 3 * TEAM)
                run(CInt<3>{});
            else
                run(CInt<1>{});
        };

        // step 4: weights, screen and digestion of `ns` bra pairs from slot s0 on
        const int K = ket.kdim;
        const long long moff = ket.moff;
        const double* __restrict__ Dj = a.Dj + moff;
        const double* __restrict__ Qb = ket.Qbf;
        const float* __restrict__ Qf = ket.Qbf32;
        const int ketsame = ket.same, ketid = t.ket;
        auto digest = [&](int s0, int ns) {
            const float inout = 1.0f / nout, incd = 1.0f / ncd;
            for (int x = tid; x < ns * nfb; x += TEAM) {
                const int s = x / nfb;
                bfn[x] = __ldg(a.pairs[bid[s0 + s]].tab + 3 * nmb + x - s * nfb);
            }
            team_sync<TEAM>();
            // per function pair of the round (bra pairs by slot, then the ket
            // pair): member bound, Schwarz bound (negative: not a unique
            // pair), pair index | (i != j) << 31
            double* pm = W;     // W is not needed any more
            float* pq = reinterpret_cast<float*>(pm + ns * nab + ncd);
            unsigned* pp = reinterpret_cast<unsigned*>(pq + ns * nab + ncd);
            const float inab = 1.0f / nab;
            for (int x = tid; x < ns * nab + ncd; x += TEAM) {
                const bool isket = x >= ns * nab;
                const int s = isket ? 0 : fdiv(x, nab, inab), e = isket ? x - ns * nab : x - s * nab;
                const int b = isket ? ketid : bid[s0 + s], n = isket ? nD : nB, u = e / n;
                const int* f = isket ? kfn : bfn + s * nfb;
                const int i = f[u], j = f[(isket ? nC : nA) + e - u * n];
                const unsigned q = (unsigned)tri(i, j);
                const float v = __ldg(Qf + q);
                pq[x] = i < j && a.pairs[b].same ? -1.0f : v;
                pp[x] = q | (i != j ? 0x80000000u : 0u);
                if (a.mixed) pm[x] = __ldg(a.pairs[b].mq + (__ldg((isket ? ktype : btype) + e) & 255));
            }
            team_sync<TEAM>();
            for (int x = tid; x < ns * nout; x += TEAM) {
                const int s = fdiv(x, nout, inout), o = x - s * nout, ab = fdiv(o, ncd, incd), cd = o - ab * ncd;
                const int xb = s * nab + ab, xk = ns * nab + cd;
                const float qb = pq[xb], qk = pq[xk];
                const unsigned eb = pp[xb], ek = pp[xk], pij = eb & 0x7fffffffu, pkl = ek & 0x7fffffffu;
                bool skip = qb < 0.0f || qk < 0.0f || (pij < pkl && bid[s0 + s] == ketid);
                if (a.mixed) skip = skip || pm[xb] * pm[xk] < ket.cut32;
                if (a.screen) {
                    // decided in float away from the threshold, in double near it
                    const float f = qb * qk;
                    if (f < a.thr_hi) skip = skip || f < a.thr_lo || __ldg(Qb + pij) * __ldg(Qb + pkl) < a.thr;
                }
                double* v = acc + s * As + o;
                for (int part = 1; part < t.parts; ++part) *v += v[part * t.slots * As];
                *v = skip ? 0.0 : times_pow2(*v, (int)(eb >> 31) + (int)(ek >> 31) + (pij != pkl));
            }
            team_sync<TEAM>();
            // The six blocks of function pairs that a quartet touches, per bra
            // pair: AB, CD, then per exchange matrix AC, BD, AD, BC.  Their
            // densities go to shared memory in one pass (one load latency;
            // with the loads inside the sums the digestion took 5.8 of the
            // 17.1 ms of n-decane/6-31G*'s launches); then one thread sums
            // each element of J and K over the opposite block.
            const int nac = nA * nC, nbd = nB * nD, nad = nA * nD, nbc = nB * nC, nx = nac + nbd + nad + nbc;
            const int per = nab + ncd + a.nk * nx, Ds = per | 1;
            const float ins = 1.0f / ns;
            double* Dl = W;
            // row and column of element o of bra pair s, and its matrix (0: J, 1, 2: exchange)
            auto element = [&](int o, int s, int& r, int& c) {
                const int* fb = bfn + s * nfb;
                if (o < nab) {
                    const int ia = o / nB;
                    r = fb[ia]; c = fb[nA + o - ia * nB];
                    return 0;
                }
                if ((o -= nab) < ncd) {
                    const int ic = o / nD;
                    r = kfn[ic]; c = kfn[nC + o - ic * nD];
                    return 0;
                }
                o -= ncd;
                const int sp = o >= nx;
                o -= sp ? nx : 0;
                const bool b = o >= nac && (o < nac + nbd || o >= nac + nbd + nad);     // row from B
                const bool dd = o >= nac && o < nac + nbd + nad;                         // column from D
                o -= o < nac ? 0 : o < nac + nbd ? nac : o < nac + nbd + nad ? nac + nbd : nac + nbd + nad;
                const int n = dd ? nD : nC, x = o / n;
                r = fb[b ? nA + x : x]; c = kfn[dd ? nC + o - x * n : o - x * n];
                return 1 + sp;
            };
            // bra pair fastest: a warp's lanes sum blocks of one shape
            for (int x = tid; x < ns * per; x += TEAM) {
                const int o = fdiv(x, ns, ins), s = x - o * ns;
                int r, c;
                const int m = element(o, s, r, c);
                const double* D = m == 0 ? Dj : (m == 1 ? a.Dk : a.Dk2) + moff;
                Dl[s * Ds + o] = __ldg(D + (long long)r * K + c);
            }
            team_sync<TEAM>();
            for (int x = tid; x < ns * per; x += TEAM) {
                int o = fdiv(x, ns, ins);
                const int s = x - o * ns;
                int r, c;
                const int m = element(o, s, r, c);
                const double* v = acc + s * As;
                const double* D = Dl + s * Ds;
                int n1, n2, s1, s2;                   // the opposite block and its strides in the quartet's
                if (o < nab) {                        // J_ij += D_kl
                    v += o * ncd;
                    D += nab;
                    n1 = 1; n2 = ncd; s1 = 0; s2 = 1;
                } else if ((o -= nab) < ncd) {        // J_kl += D_ij
                    v += o;
                    n1 = 1; n2 = nab; s1 = 0; s2 = ncd;
                } else {
                    o -= ncd;
                    D += nab + ncd;
                    if (o >= nx) {
                        o -= nx;
                        D += nx;
                    }
                    if (o < nac) {                    // K_ik += D_jl
                        const int x1 = o / nC;
                        v += x1 * nB * ncd + (o - x1 * nC) * nD;
                        D += nac;
                        n1 = nB; n2 = nD; s1 = ncd; s2 = 1;
                    } else if ((o -= nac) < nbd) {    // K_jl += D_ik
                        const int x1 = o / nD;
                        v += x1 * ncd + o - x1 * nD;
                        n1 = nA; n2 = nC; s1 = nB * ncd; s2 = nD;
                    } else if ((o -= nbd) < nad) {    // K_il += D_jk
                        const int x1 = o / nD;
                        v += x1 * nB * ncd + o - x1 * nD;
                        D += nac + nbd + nad;
                        n1 = nB; n2 = nC; s1 = ncd; s2 = nD;
                    } else {                          // K_jk += D_il
                        o -= nad;
                        const int x1 = o / nC;
                        v += x1 * ncd + (o - x1 * nC) * nD;
                        D += nac + nbd;
                        n1 = nA; n2 = nD; s1 = nB * ncd; s2 = 1;
                    }
                }
                double sum = 0.0;
                for (int x1 = 0; x1 < n1; ++x1, v += s1, D += n2) {
#pragma unroll 4
                    for (int x2 = 0; x2 < n2; ++x2) sum = fma(D[x2], v[x2 * s2], sum);
                }
                if (__double_as_longlong(sum) << 1) {
                    double* M = m == 0 ? a.J : m == 1 ? a.Kx : a.Kx2;
                    atomicAdd(M + moff + (long long)r * K + c, sum);
                }
            }
        };

        // kTeamEri: the unique, unscreened integrals of `ns` bra pairs; a
        // quartet split over several tasks adds its parts
        auto store = [&](int s0, int ns, bool part) {
            const float inout = 1.0f / nout, incd = 1.0f / ncd;
            for (int x = tid; x < ns * nout; x += TEAM) {
                const int s = fdiv(x, nout, inout), o = x - s * nout, ab = fdiv(o, ncd, incd), cd = o - ab * ncd;
                const int b = bid[s0 + s];
                const SuperPair& bra = a.pairs[b];
                const int* fb = bra.tab + 3 * nmb;
                const int i = __ldg(fb + ab / nB), j = __ldg(fb + nA + ab % nB);
                const int k = kfn[cd / nD], l = kfn[nC + cd % nD];
                const long long pij = tri(i, j), pkl = tri(k, l);
                if ((i < j && bra.same) || (k < l && ketsame) || (b == ketid && pij < pkl)) continue;
                if (a.screen && __ldg(Qb + pij) * __ldg(Qb + pkl) < a.thr) continue;
                const long long hi = pij > pkl ? pij : pkl, lo = pij > pkl ? pkl : pij;
                double* e = a.out + hi * (hi + 1) / 2 + lo;
                double v = acc[s * As + o];
                for (int q = 1; q < t.parts; ++q) v += acc[(q * t.slots + s) * As + o];
                if (part)
                    atomicAdd(e, v);
                else
                    *e = v;
            }
        };

        if (single) {
            for (int r0 = 0; r0 < nrows; r0 += t.nr) {
                const int nr = min((int)t.nr, nrows - r0);
                for (int k0 = 0; k0 < npk; k0 += t.nkb) {
                    const int nk = min((int)t.nkb, npk - k0);
                    make_R(r0, nr, k0, nk);
                    make_W(0, nr, k0, nk, k0 == 0);
                    team_sync<TEAM>();
                }
                if (a.mode == kTeamDiag) {
                    for (int x = tid; x < nab; x += TEAM)
                        bra_j(CInt<1>{}, bra0, acc, korder[x], x, 0, t.i0 + r0, nr, r0 == 0, 0, 1);
                } else {
                    make_acc(0, 1, 0, r0 == 0, r0, nr);
                }
                team_sync<TEAM>();
            }
            if (a.mode == kTeamFock) {
                digest(0, 1);
            } else if (a.mode == kTeamEri) {
                store(0, 1, nrows < bra0.npp);
            } else {
                for (int ab = tid; ab < nab; ab += TEAM) a.out[t.out + ab] = acc[ab * ncd + ab];
            }
            team_sync<TEAM>();
        } else {
            make_R(0, nrows, 0, npk);
            for (int s0 = 0; s0 < t.nb; s0 += t.slots) {
                const int ns = min((int)t.slots, t.nb - s0);
                const int w0 = rstart[s0], nw = rstart[s0 + ns] - w0;
                if (nw == 0) continue;
                make_W(w0, nw, 0, npk, true);
                team_sync<TEAM>();
                make_acc(s0, ns, w0, true, 0, 0);
                team_sync<TEAM>();
                if (a.mode == kTeamFock)
                    digest(s0, ns);
                else
                    store(s0, ns, false);
                team_sync<TEAM>();
            }
            team_sync<TEAM>();   // rstart is read before the next task writes it
        }
    }
}

// BF-pair Schwarz bounds sqrt((ab|ab)): the partial sums of a super pair's
// tasks added in order.
__global__ void k_team_bounds(const SuperPair* pairs, int npairs, const int* first, const double* part,
                              const long long* qoff, double* Q, float* Q32)
{
    const int p = blockIdx.x;
    const SuperPair& s = pairs[p];
    const int* f = s.tab + 3 * s.nmem;
    const int nab = s.nA * s.nB;
    for (int ab = threadIdx.x; ab < nab; ab += blockDim.x) {
        const int i = f[ab / s.nB], j = f[s.nA + ab % s.nB];
        if (s.same && i < j) continue;
        double v = 0.0;
        for (int x = first[p]; x < first[p + 1]; x += nab) v += part[x + ab];
        v = sqrt(v > 0.0 ? v : 0.0);
        const long long q = qoff[s.frag] + tri(i, j);
        Q[q] = v;
        Q32[q] = (float)v;
    }
}

__global__ void k_team_rebase(TeamTask* t, long long n, int dpair, int dorder)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        t[i].ket += dpair;
        t[i].b0 += dorder;
    }
}
__global__ void k_team_rebase_order(int* o, long long n, int dpair)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        o[i] += dpair;
}

// Dsh[p] = largest |D| in the function block of super pair p (D2 may be null)
__global__ void k_team_density(const SuperPair* pairs, int npairs, const double* D1, const double* D2, double* Dsh)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    const SuperPair& s = pairs[p];
    const int* f = s.tab + 3 * s.nmem;
    double m = 0.0;
    for (int i = 0; i < s.nA; ++i)
        for (int j = 0; j < s.nB; ++j) {
            const long long e = s.moff + (long long)f[i] * s.kdim + f[s.nA + j];
            m = fmax(m, fabs(D1[e]));
            if (D2) m = fmax(m, fabs(D2[e]));
        }
    Dsh[p] = m;
}

template <int TEAM>
const void* team_kernel(int L)
{
    switch (L) {
    case 0: return (const void*)k_team<0, TEAM>;
    case 1: return (const void*)k_team<1, TEAM>;
    case 2: return (const void*)k_team<2, TEAM>;
    case 3: return (const void*)k_team<3, TEAM>;
    case 4: return (const void*)k_team<4, TEAM>;
    case 5: return (const void*)k_team<5, TEAM>;
    case 6: return (const void*)k_team<6, TEAM>;
    default: return (const void*)k_team<-1, TEAM>;
    }
}

}  // namespace

static KernelSpec team_strided_spec(const void* f, long long n)
{
    KernelSpec s;
    s.func = f;
    s.grid = dim3((unsigned)std::max(1LL, std::min((n + 255) / 256, 1024LL)));
    s.block = dim3(256);
    return s;
}
KernelSpec team_rebase_spec(long long n) { return team_strided_spec((const void*)k_team_rebase, n); }
KernelSpec team_rebase_order_spec(long long n) { return team_strided_spec((const void*)k_team_rebase_order, n); }

KernelSpec team_bounds_spec(int npairs)
{
    KernelSpec s;
    s.func = (const void*)k_team_bounds;
    s.grid = dim3((unsigned)npairs);
    s.block = dim3(64);
    return s;
}

KernelSpec team_density_spec(int npairs)
{
    KernelSpec s;
    s.func = (const void*)k_team_density;
    s.grid = dim3((unsigned)((npairs + 127) / 128));
    s.block = dim3(128);
    return s;
}

// Persistent grid: as many CTAs as fit the GPU, or as the tasks need.
cudaError_t team_spec(const TeamGroup& g, int nsm, KernelSpec* s)
{
    s->func = g.team == 32 ? team_kernel<32>(g.L) : team_kernel<128>(g.L);
    s->block = dim3((unsigned)g.team);
    s->smem = team_header(g.L) + sizeof(double) * (size_t)g.slice;
    cudaError_t e = allow_max_smem(s->func);
    if (e != cudaSuccess) return e;
    int per = 1;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, s->func, g.team, s->smem);
    if (e != cudaSuccess) return e;
    s->grid = dim3((unsigned)std::min<long long>((long long)g.n, (long long)nsm * std::max(1, per)));
    return cudaSuccess;
}

}  // namespace hfx
