// hfx_team.hpp -- the FP64 Fock build over super shells: data layout, launch
// arguments and the host-side plan of the team kernel (hfx_team.cu).
//
// A super shell gathers shells of one centre that share primitive exponents:
// the general contractions of the correlation-consistent sets (carbon
// cc-pVDZ: three s shells over nine exponents), the SP shells of the Pople
// sets.  A super pair is a pair of super shells; it holds one list of
// primitive pairs over the union of the exponents, and every Hermite Coulomb
// table R_tuv is computed once per pair of primitive pairs for all the member
// shells, where a shell-by-shell build computes it once per contracted
// quartet (benzene/cc-pVDZ: 1.0e8 primitive quartets become 1.4e7).
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <vector>

#include "hfx_device.cuh"
#include "hfx_internal.hpp"

namespace hfx {

// Most functions of a super shell of several shells: the Cartesian block of a
// quartet of such is at most 36 x 36, 10 KB of shared memory.  A single shell
// may have up to ten functions (f): 100 x 100, 80 KB, in slices of up to 19452
// doubles (152 KB, NaCl/cc-pVTZ).
constexpr int kSuperMaxFn = 6;

// Primitive-pair header: p, Px, Py, Pz, sqrt(2 pi^{5/2}) / p, and a word that
// keeps its three 16-byte loads aligned.
constexpr int kTeamHdr = 6;

// Boys table of the team kernel: one row of 8 doubles per (L, k), T_k = k/64:
// F_L, F_{L+1}, F_{L+2}/2!, ... F_{L+5}/5!, exp(-T_k), 0, for T < 48.
constexpr int kTeamBoysInv = 64;
constexpr int kTeamBoysTMax = 48;
constexpr int kTeamBoysN = kTeamBoysTMax * kTeamBoysInv + 1;
constexpr int kTeamBoysMaxL = 12;

// A super pair on the device.  tab: per member shell pair the start and the
// length of its primitive list, then the offset of its coefficients (3 nmem
// ints); the nA + nB basis-function indices; the nA nB component pairs by
// decreasing work (list length x coefficients), the order in which the lanes
// of a warp take them; the lists.  coef: per member and
// list entry the non-zero Hermite->Cartesian products (weights included) in
// the class order of hfx_device.cuh.
struct __align__(16) SuperPair {
    const double* hdr;
    const double* coef;
    const int* tab;
    const double* Qbf;      // the molecule's BF-pair Schwarz bounds and their float copy
    const float* Qbf32;
    const double* mq;       // Schwarz bound of each member shell pair
    double qmax;            // the largest of them
    double cut32;           // FP32 cut of a mixed-precision job
    long long moff;         // first element of the molecule's matrices
    const int* type;        // the type's table
    int npp, nmem, L, nA, nB;
    int kdim, frag, same;   // same: both sides are one super shell
    int id, shA, shB, pbase;
};

// Type table (ints), shared by all super pairs of one (A, B) composition: per
// component pair  member | first coefficient << 8 | coefficients << 20;  per
// member the offset of its class in the coefficient tables, then its
// coefficients per primitive pair.

// One unit of work: one ket super pair against nb bra super pairs
// (order[b0..b0+nb)), or (nb = 1) the bra primitive pairs [i0, i1) of one.
struct __align__(16) TeamTask {
    int ket, b0;
    unsigned short nb, i0, i1;
    unsigned short nr;      // bra primitive pairs per R batch
    unsigned short nkb;     // ket primitive pairs per R batch
    unsigned short slots;   // bra pairs per round (nb > 1)
    unsigned short nw;      // bra primitive pairs per round
    unsigned short parts;   // threads that share a bra pair's rows in the bra transform
    int out;                // kTeamDiag: first element of the task's partial sums
};

// What a launch does with its quartets' integrals.
enum TeamMode {
    kTeamFock = 0,   // digest them into J and K
    kTeamDiag = 1,   // Schwarz pass: (ab|ab) of every super pair with itself, partial sums per task
    kTeamEri = 2     // store the unique ones in the packed eri_index order
};

struct TeamArgs {
    const SuperPair* pairs;
    const int* order;
    const TeamTask* tasks;
    int ntasks;
    int* counter;
    const short* kcode;     // per coefficient: packed Hermite index | parity << 14
    const uint4* ridx;      // R offsets of tuv + tnp, groups of team_tuv_group tuv (8 shorts each)
    int ridx_at[49];        // first entry of (L1, L2) at L1 * 7 + L2
    const double* boys;
    double thr;
    float thr_lo, thr_hi;   // the threshold's surroundings: decided in double between them
    int screen;             // thr >= 0
    int dscreen;            // density screening (dthr)
    const double* Dj;
    const double* Dk;
    const double* Dk2;
    double* J;
    double* Kx;
    double* Kx2;
    const double* Dsh;      // per super pair max |D| (density screening), or null
    double dthr;
    const unsigned char* active;
    int mode;               // TeamMode
    double* out;            // kTeamDiag: partial sums; kTeamEri: packed integrals
    int nk;                 // exchange matrices (1 or 2)
    int mixed;              // leave out the member quartets below the pairs' cut32: FP32 launches have them
};

__host__ __device__ constexpr int team_nherm(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// largest total angular momentum whose R table a thread keeps in registers
constexpr int kTeamMaxRegL = 6;

// W's part of a slice (doubles): nw rows, or the function pairs and the density
// blocks of a round of the digestion, which take its place.
__host__ __device__ inline int team_w(int H1, int nA, int nB, int nC, int nD, int nw, int slots)
{
    const int w = nw * ((nC * nD * H1) | 1), d = slots * ((nA * nB + nC * nD + 2 * (nA + nB) * (nC + nD)) | 1);
    const int p = 2 * (slots * nA * nB + nC * nD);
    return w > d ? (w > p ? w : p) : (d > p ? d : p);
}
// Shared-memory slice of a task (doubles): Cartesian blocks, ket-transformed
// Hermite integrals, R tables (two and the seeds beyond kTeamMaxRegL), row
// descriptors.
__host__ __device__ inline int team_slice(int L1, int L2, int nA, int nB, int nC, int nD, int nr, int nkb, int nw, int slots, int nb,
                                          int parts, int nmk)
{
    const int L = L1 + L2, HS = team_nherm(L) | 1;
    const int nab = nA * nB, ncd = nC * nD;
    int n = parts * slots * (nab * ncd | 1) + team_w(team_nherm(L1), nA, nB, nC, nD, nw, slots) + nr * nkb * HS;
    if (L > kTeamMaxRegL) n += nr * nkb * HS + (L + 1) * nr * nkb;
    // ints: rows, row starts, bra pairs, ket members and functions, bra
    // functions, the two orders of component pairs
    n += (nr + 2 * nb + 1 + 6 * nmk + 20 + 20 * slots + nab + ncd + 1) / 2;
    return (n + 3) & ~1;
}
// Component pairs cd that one thread of step 3 computes where they are many.
__host__ __device__ constexpr int team_cd_group(int ncd) { return ncd % 4 == 0 ? 4 : ncd % 3 == 0 ? 3 : 1; }
// Consecutive tuv that one thread of step 2 computes (H1 > 1).
__host__ __device__ constexpr int team_tuv_group(int H1) { return H1 == 10 || H1 == 20 || H1 == 35 ? 5 : 4; }

// One launch: the tasks of one register-R angular momentum (or the general
// form), team size and slice tier.
struct TeamGroup {
    int L;               // compiled total angular momentum, -1: general
    int team;            // threads per team, one team per CTA
    int slice;           // doubles per team
    size_t off, n;
    double cost;         // estimated FP64 instructions
    double prims;        // primitive quartets whose R the tasks compute
};

// Host image of a job's super pairs.
struct SuperData {
    std::vector<SuperPair> pairs;       // hdr / coef / tab hold offsets into the pools below until uploaded
    std::vector<double> hdr, coef;
    std::vector<int> tab;
    std::vector<int> types;
    std::vector<int> cls;               // per pair: its class (composition and primitive counts)
    std::vector<double> cls_nnz;        // per class: coefficients per primitive pair
    std::vector<std::vector<int>> cls_work;   // per class, of its longest pair: list length x coefficients, decreasing
    std::vector<int> cls_npp;           // and its primitive pairs
    int ncls = 0;
    std::vector<std::vector<int>> members;   // per pair: ids of its member shell pairs
    std::vector<std::vector<int>> member_at; // and their member numbers
    std::vector<std::vector<int>> member_npp;   // and the primitive pairs of each shell pair by itself (build statistics)
    std::vector<int> pbase;             // per molecule: first super pair
};

// Per coefficient of the 16 ordered (la, lb) classes, concatenated: packed
// Hermite index | parity << 14.
const std::vector<short>& team_codes();
// TeamArgs::ridx and ridx_at.
struct TeamRidx {
    std::vector<unsigned> words;    // four per entry
    int at[49];
};
const TeamRidx& team_ridx();

struct Fragments;
SuperData build_super_data(const Basis& b, const Fragments& fr);

struct TeamPlanHost {
    std::vector<TeamGroup> groups;
    std::vector<TeamTask> tasks;
    std::vector<int> order;
    std::vector<int> first;     // diagonal plan: first partial sum of every pair (one more at the end)
};
// The diagonal quartets of every super pair (kTeamDiag).
TeamPlanHost build_team_diagonal(const SuperData& sd, int nsm);
// The bra and ket super pairs of every surviving quartet (bound >= cut).
TeamPlanHost build_team_plan(const SuperData& sd, const std::vector<double>& q, double cut, int nsm);

// Boys table of the team kernel, built once per process.
const std::vector<double>& team_boys_host();

// Shift the pair indices of task and order lists copied into a session's lists.
KernelSpec team_rebase_spec(long long n);   // k_team_rebase(tasks, n, pair shift, order shift)
KernelSpec team_rebase_order_spec(long long n);   // k_team_rebase_order(order, n, pair shift)
// k_team_bounds(pairs, npairs, first, partial sums, qoff, Q, Q32): BF-pair Schwarz bounds
KernelSpec team_bounds_spec(int npairs);
KernelSpec team_density_spec(int npairs);   // k_team_density(pairs, npairs, D1, D2, Dsh)
cudaError_t team_spec(const TeamGroup& g, int nsm, KernelSpec* s);   // k_team(TeamArgs)

}  // namespace hfx
