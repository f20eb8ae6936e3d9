// hfx_engine.hpp -- the device-resident job: pair data, Schwarz tables,
// screened shell-quartet work lists, and the Fock-build entry points.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <map>
#include <memory>
#include <tuple>
#include <vector>

#include "hfx_device.cuh"
#include "hfx_internal.hpp"
#include "hfx_team.hpp"

namespace hfx {

// device launch helpers (hfx_kernels.cu)
// symmetrisation of packed accumulators: one grid row (blockIdx.y) per
// molecule, Kmax = the largest molecule's K
KernelSpec finish_rhf_spec(int Kmax, int nfrag);   // k_finish_rhf(Jacc, Kacc, G, fk, fmoff, active)
KernelSpec finish_uhf_spec(int Kmax, int nfrag);   // k_finish_uhf(Jacc, Ka, Kb, J, Kao, Kbo, fk, fmoff, active)
KernelSpec add_spec(long long n);    // k_add(A, B, C, n)
KernelSpec to_float_spec(long long n);   // k_to_float(A, B, n)
KernelSpec density_blocks_spec(int npairs);   // k_density_blocks(pairs, npairs, D1, D2, Dsh)
KernelSpec rebase_tasks_spec(long long n);    // k_rebase_tasks(tasks, n, delta): bra, ket += delta
cudaError_t small_spec_f32(int pcb, int pck, int nk, int ntasks, KernelSpec* s);   // k_small(SmallArgs<float>)
cudaError_t warp_spec(int nk, int grid, int warps_per_cta, int slice, KernelSpec* s);   // k_warp_quartet(WarpArgs<float>)
// shared-memory slice (elements) of a warp task; the lane-parallel R mode (L <= 6,
// ket npp >= lane_min_npp, 0: never) needs 32 R vectors, the level-parallel one a round
int warp_slice_elems(int l0b, int l1b, int l0k, int l1k, int npp_ket, int lane_min_npp);
constexpr int kDefaultLaneMinNpp = 6;
bool is_small_class(int pcb, int pck);
// Boys table of the kernels ([kBoysN][kBoysM], last column exp(-T_k)), built once per process.
const std::vector<double>& boys_table_host();
// The FP32 kernels' Boys table: 8 floats per (L <= kBoys32MaxL, k), see hfx_device.cuh.
const std::vector<float>& boys_table32_host();

void cuda_check(cudaError_t e, const char* what);

// cudaMemcpyAsync between host and device, its bytes counted
// (hfx_debug_copied_bytes).
void copy_async(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t st, const char* what);
void copied_bytes(double* h2d, double* d2h);

// Caching device allocator: freed blocks (rounded up to a power of two, up to
// 256 MB) are kept for reuse instead of being returned with cudaFree, whose
// implicit device synchronisation would stall every other job in flight when
// one job of the request server finishes.  Larger blocks are allocated and
// freed directly.  Callers free a block only after the work using it has
// completed (a job synchronises its streams before its buffers go).
void* pool_alloc(size_t bytes);
void pool_free(void* p, size_t bytes);
size_t pool_cached_bytes();

// Owning device buffer.
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { reset(); }
    void reset()
    {
        if (p) pool_free(p, n * sizeof(T));
        p = nullptr;
        n = 0;
    }
    void alloc(size_t count)
    {
        if (count == n && p) return;
        reset();
        if (count == 0) return;
        p = static_cast<T*>(pool_alloc(count * sizeof(T)));
        n = count;
    }
    // The copy may still read v when this returns (pageable memory that the
    // GPU reaches directly is not staged): v lives until the stream is waited for.
    void upload(std::vector<T>&&, cudaStream_t) = delete;
    void upload(const std::vector<T>& v, cudaStream_t st)
    {
        alloc(v.size());
        if (!v.empty()) copy_async(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st, "upload");
    }
};

// The team kernel's Boys table on the current device, shared by the jobs and
// sessions alive there and freed with the last of them.
std::shared_ptr<DevBuf<double>> team_boys_device(int device, cudaStream_t st);

struct HostPair {
    int frag;         // molecule of a packed job
    int s0, s1;       // shells (s0 has the higher L), indices in the concatenated basis
    int l0, l1;
    int npp;
    long long e_off;
    int pp0;
    bool same;
};

// Host image of the per-job pair data (built on the CPU, then uploaded).
struct PairData {
    std::vector<HostPair> hpairs;
    std::vector<DPair> dpairs;
    std::vector<PairGeo> geo;
    std::vector<double> epool;
    std::vector<double> rec;   // class-kernel primitive-pair records
};

// Per pair class: component-pair / coefficient layout of the records.
struct ClassTables {
    std::vector<PairClassTab> tab;
    std::vector<int> ab_start;
    std::vector<short> k_herm, k_lin;
};
const ClassTables& class_tables();

// One kernel launch of a Fock build.
struct LaunchGroup {
    int kind;            // 0: small-class kernel, 1: warp kernel
    int pcb, pck;        // small-class kernel class
    bool fp32;
    int slice;           // warp kernel: per-warp slice (elements)
    int warps_per_cta;
    int lane_min_npp;    // warp kernel: lane-parallel R threshold the slice was sized for
    int grid;
    size_t off, n;       // task range in the concatenated list
    double flops, prims;
};
// Molecules of a packed job (one entry for a plain job): molecule f owns
// shells [sh[f], sh[f+1]) and basis functions [bf[f], bf[f+1]) of the
// concatenated basis, shell pairs [pbase[f], pbase[f+1]), the K_f x K_f
// block at moff[f] of every packed matrix buffer and the BF-pair bounds at
// qoff[f].
struct Fragments {
    std::vector<int> sh, bf, pbase;
    std::vector<long long> moff, qoff;
    int count() const { return (int)sh.size() - 1; }
    int K(int f) const { return bf[f + 1] - bf[f]; }
    long long nmat() const { return moff.back(); }
};
// Concatenate molecules' bases (shell bf0 shifted to the concatenated order)
// and describe the blocks.
Basis concat_basis(const std::vector<Basis>& mols, Fragments& fr);
Fragments single_fragment(const Basis& b);

// Records of the FP32 kernels; `dense`: also the primitive pairs' geometry and
// dense E blocks (hfx_debug_pair_data).
PairData build_pair_data(const Basis& b, const Fragments& fr, bool dense = true);
// Primitive-pair counts of `pd`'s records into a list of the same shell pairs.
void take_record_counts(std::vector<HostPair>& pairs, const PairData& pd);

// Primitive pairs below this fraction of their shell pair's largest
// coefficient are left out (build_pair_data, build_super_data).
constexpr double kPrimPairCut = 1e-18;

// f(i) for i in [0, n) on up to `most` (and 16) host threads.
void host_parallel_for(int n, const std::function<void(int)>& f, int most = 16);
// Indices by decreasing cost (counting sort on 1/16-octave bins, stable); with
// `shape`, equal bins are ordered by shape.
std::vector<size_t> order_by_cost_desc(const std::vector<double>& cost,
                                       const std::vector<unsigned short>* shape = nullptr);

// Screening thresholds of a launch (density screening off at dthr = 0).
void team_thresholds(TeamArgs& a, double thr, double dthr);

// A team-kernel plan on the device.
struct TeamPlanDev {
    std::vector<TeamGroup> groups;
    std::vector<KernelSpec> specs;    // per group, kept: an eager build would query the occupancy 40 times
    DevBuf<TeamTask> tasks;
    DevBuf<int> order;
    void upload(TeamPlanHost&&, int, cudaStream_t) = delete;   // as DevBuf::upload
    void upload(const TeamPlanHost& h, int nsm, cudaStream_t st);
    void make_specs(int nsm);
};

// The launch plan of one precision mode.
struct GroupSet {
    std::vector<LaunchGroup> groups;
    DevBuf<Task> tasks;
    // FP64 quartets: tasks of the team kernel over super pairs
    TeamPlanDev team;
    size_t launches() const { return groups.size() + team.groups.size(); }
    int ntasks = 0, nquartets = 0;
    double flops64 = 0.0, flops32 = 0.0, prims = 0.0, quartets32 = 0.0;
};

// Streams of a build beside the main one, and how many of all of them the FP64
// launches of a mixed build share (an FP64 build uses all): its 30-40 launches
// end in tails of a few CTAs that only other launches can fill. 3 + all
// against 11 + 8, ms: water/cc-pVTZ 1.14 / 0.92, NaCl/cc-pVTZ 3.73 / 3.4,
// benzene/cc-pVDZ 8.10 / 7.84, n-decane/6-31G* mixed 3.20 / 3.02.
constexpr int kAuxLanes = 11, kFp64Lanes = 8;
// Copies of the J/K accumulators of a build with FP32 launches (a power of
// two; CTAs spread over them, the symmetrisation adds them up): with one, the
// reductions of the FP32 kernels crowd in a few L2 slices; with four the
// busiest is 58-62% occupied and the average one 38-40% in (ps|ss) and (dp|ps)
// of n-decane/6-31G*.  1 / 2 / 4 / 8 copies, ms: n-decane mixed at an FP32 cut
// of 0.1 3.05 / 2.90 / 2.86 / 2.84, tree of 16 heavy atoms in 6-31G* at 0.03
// 14.3 / 13.8 / 13.7 / 13.6, tree of 12 in cc-pVDZ UHF at 0.1 33.6 / 32.6 /
// 32.0 / 31.7. FP64 builds reduce in the kernel first (1-4%) and keep one.
constexpr int kAccCopies = 4;

// Destination of a Fock build's device work.  Lane 0 is the job's main
// stream, lanes 1..n its auxiliary streams; fork() makes every auxiliary lane
// wait for what lane 0 has issued so far, join() makes lane 0 wait for all of
// them.  StreamSink issues the work on the streams as it comes; GraphSink
// records it as the nodes and edges of a CUDA graph, built node by node
// rather than by stream capture, so other threads' CUDA calls (allocations,
// module loads, library handles of concurrent jobs) cannot invalidate it.
class OpSink {
public:
    virtual ~OpSink() = default;
    virtual void zero(int lane, void* p, size_t bytes) = 0;
    virtual void kernel(int lane, const KernelSpec& s, void** params) = 0;
    virtual void fork() = 0;
    virtual void join() = 0;
};

class StreamSink final : public OpSink {
public:
    StreamSink(cudaStream_t main, const std::vector<cudaStream_t>& aux, cudaEvent_t fork_ev,
               const std::vector<cudaEvent_t>& aux_ev);
    void zero(int lane, void* p, size_t bytes) override;
    void kernel(int lane, const KernelSpec& s, void** params) override;
    void fork() override;
    void join() override;

private:
    cudaStream_t stream(int lane) const { return lane == 0 ? main_ : aux_[lane - 1]; }
    cudaStream_t main_;
    const std::vector<cudaStream_t>& aux_;
    cudaEvent_t fork_ev_;
    const std::vector<cudaEvent_t>& aux_ev_;
};

class GraphSink final : public OpSink {
public:
    explicit GraphSink(int lanes);
    ~GraphSink() override;
    void zero(int lane, void* p, size_t bytes) override;
    void kernel(int lane, const KernelSpec& s, void** params) override;
    void fork() override;
    void join() override;
    cudaGraphExec_t instantiate();

private:
    cudaGraph_t graph_ = nullptr;
    std::vector<std::vector<cudaGraphNode_t>> deps_;   // per lane: the nodes its next node depends on
};

// FP32 class kernels of a build with at least this many algorithmic flops run
// before everything that uses shared memory.  They live on the L1 cache, whose
// size an SM sets by the shared memory of what it runs and changes only when it
// is idle: beside FP64 or warp CTAs they keep the small one to their end. Beside
// / before, ms, mixed builds at the FP32 cut given: tree of 12 heavy atoms,
// cc-pVDZ UHF 0.1 (6e11 flops) 45.6 / 31.9, tree of 16, 6-31G* UHF 0.1 (1.5e11)
// 18.1 / 13.9, tree of 12, 6-31G* UHF 0.1 (8e10) 9.9 / 8.1.  Below it the overlap
// of both pipes is worth as much: benzene/cc-pVDZ RHF 0.03 (2e10) 4.76 / 4.95,
// n-decane/6-31G* RHF 0.1 (2.4e10) 2.85 / 2.63, NaCl/6-31G* RHF 0.03 (4e8) 0.34 / 0.36.
constexpr double kClassesFirstFlops = 4e10;

// Issues the launches of a build, which has forked, on `lanes` lanes, the lane
// chosen for each: put(lane, true, i) for the i-th FP64 launch, put(lane, false,
// i) for the i-th FP32 one.
void place_launches(OpSink& sk, size_t nteam, const std::vector<LaunchGroup>& groups, int lanes,
                    const std::function<void(int, bool, size_t)>& put);

// What the device SCF needs from a Fock builder: a job of its own, or one
// molecule's share of a packed job (hfx_batch.cpp).  Builds are synchronous
// with respect to stream().
class FockSource {
public:
    virtual ~FockSource() = default;
    virtual int K() const = 0;
    virtual cudaStream_t stream() const = 0;
    virtual bool mixed() const = 0;
    virtual void fock_rhf_device_ex(const double* dP, double* dG, bool mixed, double dthr) = 0;
    virtual void fock_uhf_device_ex(const double* dPa, const double* dPb, double* dJ, double* dKa, double* dKb,
                                    bool mixed, double dthr) = 0;
    virtual double last_build_ms() const = 0;   // device time of the last build
};

class FockSession;

class Job final : public FockSource {
    friend class FockSession;   // reads the device pair tables and plans of its members

public:
    Job(Basis b, const hfx_options& opt);
    // Packed job over several molecules: shell pairs and quartets never mix
    // molecules, and every Fock build works on packed buffers holding each
    // molecule's K_f x K_f matrices back to back (the blocks of fragments()).
    Job(const std::vector<Basis>& mols, const hfx_options& opt);
    ~Job();

    const Fragments& fragments() const { return frags_; }
    long long nmat() const { return frags_.nmat(); }
    // packed jobs: molecules whose flag is 0 are skipped by the next builds
    void set_active(const unsigned char* flags);

    int K() const override { return basis_.K; }
    int device() const { return device_; }
    const Basis& basis() const { return basis_; }

    void schwarz_host(std::vector<double>& Qbf) const;
    // device-pointer Fock builds (synchronous)
    void fock_rhf_device(const double* dP, double* dG);
    // Builds with an explicit precision plan (mixed = false: every quartet in
    // FP64) and density-weighted screening threshold (0: none; used by the
    // incremental builds of the mixed-precision SCF).
    void fock_rhf_device_ex(const double* dP, double* dG, bool mixed, double dthr) override;
    void fock_uhf_device_ex(const double* dPa, const double* dPb, double* dJ, double* dKa, double* dKb, bool mixed,
                            double dthr) override;
    double last_build_ms() const override { return stats.ms; }
    void fock_rhf_ex(const double* P, double* G, bool mixed, double dthr);
    void fock_uhf_ex(const double* Pa, const double* Pb, double* J, double* Ka, double* Kb, bool mixed, double dthr);
    bool mixed() const override { return opt_.precision == HFX_PREC_MIXED; }
    double fp32_threshold() const { return opt_.fp32_threshold; }
    double screening_threshold() const { return opt_.screening_threshold; }
    // Pick the FP32 threshold: for each candidate (largest first) build G in
    // mixed precision at density P and keep the largest tau whose energy
    // change 1/2 sum P (G_tau - G_fp64) stays within target_dE; the job is
    // switched to mixed precision at that tau.  Returns tau (0 if none fits).
    double autotune_fp32_threshold(const double* P, double target_dE, double* dE_out, double* ms_fp64,
                                   double* ms_mixed);
    // RHF build whose scratch (J/K accumulators, work-queue counters) is
    // supplied by the caller; allocates nothing.  Jacc/Kacc hold K*K doubles,
    // counters num_launch_groups() ints.
    void fock_rhf_device_scratch(const double* dP, double* dG, double* Jacc, double* Kacc, int* counters);
    // launch shape of the plans (chunk sizes, warps per CTA); setting it rebuilds the plans
    const hfx_launch_shape& launch_shape() const { return shape_; }
    void set_launch_shape(const hfx_launch_shape& s);
    // pick the launch shape by timing builds at density P (host, K x K); returns the best build ms
    double autotune_launch_shape(const double* P, int builds, hfx_launch_shape* out);
    int num_launch_groups() const { return (int)plan(true).launches(); }
    // launch groups of a plan (FP64 or, for a mixed job, mixed)
    const std::vector<LaunchGroup>& plan_groups(bool mixed_plan) const { return plan(mixed_plan).groups; }
    const std::vector<TeamGroup>& plan_team(bool mixed_plan) const { return plan(mixed_plan).team.groups; }
    int team_grid(bool mixed_plan, size_t g) const { return (int)plan(mixed_plan).team.specs[g].grid.x; }
    void fock_uhf_device(const double* dPa, const double* dPb, double* dJ, double* dKa, double* dKb);
    void fock_rhf(const double* P, double* G);
    void fock_uhf(const double* Pa, const double* Pb, double* J, double* Ka, double* Kb);
    void eri_unique(double thr, double* out);

    hfx_build_stats stats{};
    cudaStream_t stream() const override { return stream_; }

private:
    void init(const hfx_options& opt);
    void build_pairs();
    void compute_schwarz();
    TeamArgs team_args(const TeamPlanDev& plan, const TeamGroup& g, int* counter) const;
    void run_team(const TeamPlanDev& plan, int mode, double thr, double* out);
    void record_stats(int launches);

    Basis basis_;
    hfx_options opt_;
    int device_ = 0;
    int nsm_ = 1;
    cudaStream_t stream_ = nullptr;
    cudaEvent_t ev0_ = nullptr, ev1_ = nullptr, evk0_ = nullptr, evk1_ = nullptr;

    void build_jk_groups(bool mixed, GroupSet& gs);
    void build_super();
    void count_quartets(GroupSet& gs) const;
    void build_fp32_groups(GroupSet& gs);
    void launch_jk(OpSink& sk, int nk, const double* Dj, const double* Dk, const double* Dk2, double* J, double* Kx,
                   double* Kx2, int* counters = nullptr, bool mixed_plan = false, double dthr = 0.0, int ncopy = 1,
                   long long cstride = 0);
    int acc_copies(bool mixed_plan) const;
    long long acc_stride(bool mixed_plan) const;
    void alloc_acc(int nk, bool mixed_plan);
    const GroupSet& plan(bool mixed_plan) const { return mixed_plan && mixed() ? gs_mixed_ : gs_fp64_; }
    void record_stats_plan(int launches, const GroupSet& gs);
    StreamSink stream_sink() { return StreamSink(stream_, aux_, fork_ev_, aux_ev_); }
    int max_fragment_K() const;
    void enqueue_finish_rhf(OpSink& sk, const double* Jacc, const double* Kacc, double* dG, int ncopy = 1, long long cstride = 0);
    void enqueue_rhf(OpSink& sk, const double* dP, double* dG, bool mixed_plan, double dthr);
    void enqueue_uhf(OpSink& sk, const double* dPa, const double* dPb, double* dJ, double* dKa, double* dKb, bool mixed_plan,
                     double dthr);
    cudaGraphExec_t graph_for(int nk, bool mixed_plan, double dthr);
    void clear_graphs();
    struct GraphEntry {
        cudaGraphExec_t exec = nullptr;
        int eager_runs = 0;
    };
    std::map<std::tuple<int, bool, double>, GraphEntry> graphs_;
    bool no_graphs_ = false;
    DevBuf<double> d_gin_, d_gin2_, d_gout_, d_gout2_, d_gout3_;
    Fragments frags_;
    DevBuf<int> d_fk_;              // per molecule K_f
    DevBuf<long long> d_fmoff_;     // per molecule matrix offset
    DevBuf<unsigned char> d_active_;   // packed jobs: per molecule build flag
    bool packed_ = false;              // built by the packed (several-molecule) constructor
    hfx_launch_shape shape_{256, 4096, 8, kDefaultLaneMinNpp, {0, 0, 0, 0}};

    // super pairs (hfx_team.hpp): host image without the pools, device tables
    SuperData sup_;
    std::vector<double> qsup_;      // per super pair: largest bound of its members
    DevBuf<SuperPair> d_super_;
    DevBuf<double> d_shdr_, d_scoef_, d_smq_;
    DevBuf<int> d_stab_, d_stypes_;
    DevBuf<short> d_scode_;
    DevBuf<unsigned> d_sridx_;
    std::shared_ptr<DevBuf<double>> team_boys_;
    DevBuf<double> d_tdsh_;         // per super pair max |D| (density screening)

    std::vector<HostPair> hpairs_;
    GroupSet gs_fp64_, gs_mixed_;
    DevBuf<int> d_counters_;
    DevBuf<double> d_dsh_;
    DevBuf<float> d_d32_;           // float copies of the build's densities (FP32 groups)
    std::vector<DPair> dpairs_host_;
    DevBuf<float> d_rec32_;
    DevBuf<float> d_boys32_;
    DevBuf<PairClassTab> d_pct_;
    DevBuf<int> d_abs_;
    DevBuf<short> d_kh_, d_kl_;
    std::vector<cudaStream_t> aux_;
    std::vector<cudaEvent_t> aux_ev_;
    cudaEvent_t fork_ev_ = nullptr;
    std::vector<double> qsh_;     // per pair
    std::vector<double> qbf_;     // per BF pair
    DevBuf<DPair> d_pairs_;
    DevBuf<double> d_qbf_;
    DevBuf<float> d_qbf32_;         // float copy of d_qbf_ (the FP32 kernels' screen)
    DevBuf<double> d_D_, d_D2_, d_Dj_, d_J_, d_K_, d_K2_, d_out1_, d_out2_, d_out3_;
};

}  // namespace hfx
