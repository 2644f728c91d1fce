// Multifrontal engine: device storage of the fronts, the static launch
// schedule of the factorisation and of the solves, and their execution.
#pragma once
#include "internal.h"
#include "sub_kernels.cuh"
#include "devvec.cuh"
#include "tc_gemm.h"
#include <type_traits>
#include <cstdlib>
#include <functional>
#include <map>
#include <memory>
#include <mutex>

namespace wt3d {

using Launch = std::function<void(cudaStream_t)>;

// Launch kinds, for the per-kernel profile.
enum LaunchKind { LK_MEMSET = 0, LK_SCATTER, LK_EXTEND_ADD, LK_PANEL, LK_TRSM, LK_GEMM, LK_SUBSTEP, LK_SPLIT,
                  LK_TCGEMM, LK_NKINDS };

struct LaunchRec {
    Launch fn;
    int kind;
    double flops;        // real-flop count of a GEMM launch (sum of 8 M N K)
    double bytes = 0;    // operand bytes of a GEMM launch (A, B read; C read and written)
    bool side = false;   // off the factorisation's chain: nothing of the factorisation reads its results
};

// A list of launches plus the task arrays they read.
template <class T>
struct Schedule {
    std::vector<LaunchRec> launches;
    int kernels() const
    {
        int c = 0;
        for (auto &l : launches) c += l.kind != LK_MEMSET;
        return c;
    }
    DevVec<PanelTask> panel;
    DevVec<BandTask> band;
    DevVec<GemmTask<T>> gemm;
    DevVec<GemmUnit> unit;                                    // their tiles
    std::vector<GemmTask<T>> hgemm;                           // host copies while the schedule is built
    std::vector<GemmUnit> hunit;
    DevVec<EATask> ea;
    DevVec<EAUnit> eau;
    DevVec<InvTask> inv;                                      // block-inverse columns
    DevVec<SkUnit> sk;                                        // units of the substitution products
    std::vector<std::vector<GemmTask<float>>> tc_pending;   // tensor-core task lists, built after allocation
    std::vector<std::unique_ptr<TcLaunch>> tc;
    cudaGraphExec_t graph = nullptr;
    ~Schedule()
    {
        if (graph) cudaGraphExecDestroy(graph);
    }
};

// Buffers a factorisation needs only while it runs: the two level-parity
// update buffers and the tensor-core split-operand workspace.  Handles of the
// same grid and precision share one; `mu` serialises their factorisations.
template <class T>
struct FactorWorkspace {
    DevVec<cx<T>> upd0, upd1;
    DevVec<float> tcws;
    std::mutex mu;
    size_t bytes() const { return (upd0.n + upd1.n) * sizeof(cx<T>) + tcws.n * sizeof(float); }
};

template <class T>
class Engine {
public:
    const Symbolic *S = nullptr;
    DevVec<cx<T>> fac, binv;      // factors; inverses of the diagonal blocks (see k_tile_inverse)
    // right-hand sides of a pass, [row][sk_columns(m)] in the new ordering: X the
    // sources (then the forward sweep's partial sums), Z the forward sweep's
    // solution (then the backward sweep's partial sums), Y the solution.  Z and
    // Y are zero when a pass starts (k_gather_new).
    DevVec<cx<T>> X, Z, Y;
    std::shared_ptr<FactorWorkspace<T>> ws;
    DevVec<int> ipiv, border;
    DevVec<int> gord;   // per pivot position (new ordering): the row that the interchanges leave there
    DevVec<int> eapos;   // per child: border index of every row of the parent front, -1 for none (k_extend_add)
    DevVec<FrontDev> fr;
    std::vector<FrontDev> hfr;
    DevVec<long long> map;
    DevVec<int> npert;
    DevVec<unsigned long long> maxabs;
    std::unique_ptr<Schedule<T>> fsched;
    std::map<int, std::unique_ptr<Schedule<T>>> ssched[2];   // [adjoint][m]
    // vectors of a band launch from which four threads take two
    static constexpr long long BAND_TWO = 152 * 4 * 32;
    // flops from which a factorisation's update goes to the tensor-core kernel
    static constexpr double TC_MIN_FLOPS = 1e9;
    static constexpr int SBW = SB<T>;   // columns per diagonal block of the substitutions
    // units a launch of k_skinny is cut into, and the shortest K of a unit
    static constexpr int SK_SLOTS = 152 * 8, SK_KMIN = 64;
    // complex64 factor entries from which the products of a pass over one column are
    // k_gemv's (all of A^H are).  One kernel for a whole pass: launches of two that need different splits
    // of L1 and shared memory wait for each other's SMs, and choosing by launch lost 10 %.
    // Milliseconds per pass, k_skinny and k_gemv: 14x12x13 0.158 and 0.169, 20^3 0.268 and
    // 0.279, 29x27x25 (1.2e8 entries) 0.50 and 0.47, 40^3 1.54 and 1.29, 64x64x48 5.4 and
    // 4.2; A^H: 14x12x13 0.111 and 0.109, 20^3 0.27 and 0.20, 64x64x48 5.7 and 4.0.
    // complex128 (calls of one pass): 14x12x13 0.35 and 0.37, 24x22x20 1.31 and 1.43,
    // 40^3 6.57 and 6.71, so none forward; A^H 0.37 and 0.34, 1.27 and 1.28, 6.42 and 6.10.
    static constexpr double GEMV_MIN_ENTRIES = 8e7;
    // outer block width of the two-level LU (WT3D_WB: a multiple of KB, 512 by default)
    const int WB = [] {
        const char *e = getenv("WT3D_WB");
        const int v = e ? atoi(e) : 512;
        return (v >= KB && v % KB == 0) ? v : 512;
    }();
    cudaStream_t side = nullptr;     // branch of the factorisation's graph for the launches off its chain
    cudaEvent_t side_ev = nullptr;
    // pivots below pivot_rel times the largest entry are perturbed: only
    // (near-)zero ones, since Dirichlet rows carry unit pivots next to O(1e8)
    // stiffness entries
    double pivot_rel = 1e-20;
    // tcgen05 path for complex64 front updates (WT3D_TC=0 selects the SIMT kernel)
    bool use_tc = std::is_same<T, float>::value && !(getenv("WT3D_TC") && getenv("WT3D_TC")[0] == '0');
    // tensor cores for the products of complex64 substitution passes (WT3D_TS=0: FP32 pipe)
    bool use_ts = std::is_same<T, float>::value && !(getenv("WT3D_TS") && getenv("WT3D_TS")[0] == '0');
    DevVec<float> own_tcws;   // private split workspace, only if the shared one is too small
    DevVec<int> tc_err;                                 // barrier-timeout flag of the tensor-core kernel
    std::vector<Schedule<T> *> built_tc;   // schedules whose tensor maps point into the split workspace
    // launch schedules as captured CUDA graphs (WT3D_GRAPHS=0: direct launches, for profilers)
    bool use_graphs = !(getenv("WT3D_GRAPHS") && getenv("WT3D_GRAPHS")[0] == '0');

    // device bytes this engine holds on its own (the shared workspace excluded)
    size_t device_bytes() const
    {
        return (fac.n + X.n + Z.n + Y.n + binv.n) * sizeof(cx<T>) + (ipiv.n + border.n + eapos.n + gord.n) * 4 +
               fr.n * sizeof(FrontDev) +
               map.n * 8 + scale.n * 8 + own_tcws.n * sizeof(float);
    }

    // Reads (and clears) the barrier-timeout flag of the tensor-core kernels;
    // call after the stream that ran them is synchronised.
    int check_tc_err()
    {
        int e = 0;
        WT_CUDA(cudaMemcpy(&e, tc_err.p, sizeof(int), cudaMemcpyDeviceToHost));
        if (!e) return WT3D_OK;
        WT_CUDA(cudaMemset(tc_err.p, 0, sizeof(int)));
        set_error("tensor-core kernel: mbarrier wait expired (code " + std::to_string(e) + ")");
        return WT3D_ERR_CUDA;
    }
    size_t workspace_bytes() const { return ws ? ws->bytes() : 0; }
    // split workspace of the tensor-core launches: private if allocated, else the shared one
    float *tcws_base() const { return own_tcws.p ? own_tcws.p : ws->tcws.p; }
    size_t tcws_size() const { return own_tcws.p ? own_tcws.n : ws->tcws.n; }

    const int *d_irptr = nullptr, *d_jcptr = nullptr;   // natural 0-based CSR of the operator
    DevVec<double> scale;                              // Jacobi scaling 1/sqrt|a_ii|, natural ordering

    int init(const Symbolic &sym, const std::vector<long long> &hmap, const int *irp, const int *jcp,
             std::shared_ptr<FactorWorkspace<T>> w)
    {
        S = &sym;
        d_irptr = irp;
        d_jcptr = jcp;
        ws = w ? w : std::make_shared<FactorWorkspace<T>>();
        int rc;
        if ((rc = fac.alloc(sym.fac_total))) return rc;
        {
            std::lock_guard<std::mutex> lk(ws->mu);
            const size_t n0 = std::max<long long>(sym.upd_size[0], 1), n1 = std::max<long long>(sym.upd_size[1], 1);
            if (ws->upd0.n < n0 && (rc = ws->upd0.alloc(n0))) return rc;
            if (ws->upd1.n < n1 && (rc = ws->upd1.alloc(n1))) return rc;
        }
        const size_t nx = (size_t)sym.n * MAXRHS;
        if ((rc = X.alloc(nx)) || (rc = Z.alloc(nx)) || (rc = Y.alloc(nx))) return rc;
        if ((rc = ipiv.alloc(sym.n))) return rc;
        if ((rc = border.upload(sym.border))) return rc;
        if ((rc = map.upload(hmap))) return rc;
        if ((rc = npert.alloc(1))) return rc;
        if ((rc = maxabs.alloc(1))) return rc;
        if ((rc = scale.alloc(sym.n))) return rc;
        if ((rc = tc_err.alloc(1))) return rc;
        WT_CUDA(cudaMemset(tc_err.p, 0, sizeof(int)));
        if (use_tc && (rc = tc_init())) return rc;
        std::vector<FrontDev> h(sym.fronts.size());
        long long ninv = 0;
        for (size_t f = 0; f < h.size(); f++) {
            const Front &F = sym.fronts[f];
            h[f].inv = ninv;
            ninv += inv_entries<T>(F.p);
            h[f].fac = F.fac_off;
            h[f].upd = F.upd_off;
            h[f].border = F.border_off;
            h[f].p = F.p;
            h[f].b = F.b;
            h[f].first = F.first;
            h[f].parity = F.level & 1;
        }
        if ((rc = fr.upload(h))) return rc;
        hfr = h;
        if ((rc = binv.alloc((size_t)ninv))) return rc;
        if ((rc = gord.alloc((size_t)sym.n))) return rc;
        WT_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        WT_CUDA(cudaEventCreateWithFlags(&side_ev, cudaEventDisableTiming));
        // kernel attributes are per device: once for each device this process uses
        static std::once_flag attr_once[64];
        int dev = 0;
        cudaGetDevice(&dev);
        std::call_once(attr_once[dev & 63], [] {
            cudaFuncSetAttribute(k_tile_inverse<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)BandCfg<T, 1>::smem);
            cudaFuncSetAttribute(k_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)panel_smem<T>());
            cudaFuncSetAttribute(k_bands<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)BandCfg<T, 1>::smem);
            cudaFuncSetAttribute(k_bands<T, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)BandCfg<T, 2>::smem);
            sk_attributes();
        });
        return build_factor_schedule();
    }
    Engine() = default;
    Engine(const Engine &) = delete;
    Engine &operator=(const Engine &) = delete;
    ~Engine()
    {
        if (side_ev) cudaEventDestroy(side_ev);
        if (side) cudaStreamDestroy(side);
    }

    static void sk_attributes()
    {
        sk_attr<1>();
        sk_attr<4>();
        sk_attr<8>();
        sk_attr<16>();
        sk_attr<32>();
    }
    template <int NC>
    static void sk_attr()
    {
        cudaFuncSetAttribute(k_skinny<T, NC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)SkCfg<T, NC>::smem(false));
        cudaFuncSetAttribute(k_skinny<T, NC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)SkCfg<T, NC>::smem(true));
    }

    // a launch as programmatic dependent of the product before it
    template <class Kernel>
    static void sk_chain(Kernel k, size_t smem, const SkUnit *u, int n, const cx<T> *in, cx<T> *out, cudaStream_t st)
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)n);
        cfg.blockDim = dim3(SK_TH);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k, u, in, out);
    }
    template <int NC>
    static void sk_launch_n(bool herm, const SkUnit *u, int n, const cx<T> *in, cx<T> *out, cudaStream_t st)
    {
        if (herm) sk_chain(k_skinny<T, NC, true>, SkCfg<T, NC>::smem(true), u, n, in, out, st);
        else sk_chain(k_skinny<T, NC, false>, SkCfg<T, NC>::smem(false), u, n, in, out, st);
    }
    static void sk_launch(int nc, bool gemv, bool herm, const SkUnit *u, int n, const cx<T> *in, cx<T> *out,
                          cudaStream_t st)
    {
        if (gemv) {   // complex128: A^H only
            if (herm) sk_chain(k_gemv<T, true>, 0, u, n, in, out, st);
            else if constexpr (sizeof(T) == 4) sk_chain(k_gemv<T, false>, 0, u, n, in, out, st);
            return;
        }
        if (nc == 1) sk_launch_n<1>(herm, u, n, in, out, st);
        else if (nc == 4) sk_launch_n<4>(herm, u, n, in, out, st);
        else if (nc == 8) sk_launch_n<8>(herm, u, n, in, out, st);
        else if (nc == 16) sk_launch_n<16>(herm, u, n, in, out, st);
        else sk_launch_n<32>(herm, u, n, in, out, st);
    }

    // ---------------------------------------------------------------------
    static void add_gemm(std::vector<GemmTask<T>> &v, const cx<T> *A, int lda, const cx<T> *B, int ldb, cx<T> *C,
                         int ldc, int M, int N, int K)
    {
        if (M <= 0 || N <= 0 || K <= 0) return;
        GemmTask<T> g{};
        g.A = A; g.B = B; g.C = C;
        g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.M = M; g.N = N; g.K = K;
        v.push_back(g);
    }

    static double gemm_bytes(const GemmTask<T> &g)
    {
        return ((double)g.M * g.K + (double)g.K * g.N + 2.0 * g.M * g.N) * sizeof(cx<T>);
    }

    // Appends the launches of the GEMM tasks v (and empties it): tasks the
    // tensor-core kernel takes (complex64) go to a tcgen05 launch, the rest to the
    // SIMT kernel.  A tensor-core launch comes with two operand-split launches
    // before it, 45 us for the three at the least; below TC_MIN_FLOPS the SIMT
    // kernel is done sooner.
    void push_gemm_launch(Schedule<T> &sc, std::vector<GemmTask<T>> &v)
    {
        std::vector<GemmTask<T>> simt;
        Schedule<T> *psc = &sc;
        if constexpr (std::is_same<T, float>::value) {
            std::vector<GemmTask<float>> tcv;
            double fl = 0, by = 0;
            for (const auto &g : v) {
                if (use_tc && tc_eligible(g)) {
                    tcv.push_back(g);
                    fl += 8.0 * g.M * (double)g.N * g.K;
                    by += gemm_bytes(g);
                } else {
                    simt.push_back(g);
                }
            }
            if (fl < TC_MIN_FLOPS) {
                simt = v;
            } else {
                const int idx = (int)sc.tc_pending.size();
                sc.tc_pending.push_back(std::move(tcv));
                sc.launches.push_back({[psc, idx](cudaStream_t st) { tc_split(*psc->tc[idx], st); }, LK_SPLIT, 0});
                sc.launches.push_back({[psc, idx, this](cudaStream_t st) { tc_mma(*psc->tc[idx], tc_err.p, st); },
                                       LK_TCGEMM, fl, by});
            }
        } else {
            simt = v;
        }
        v.clear();
        if (simt.empty()) return;
        double fl = 0, by = 0;
        for (const auto &g : simt) {
            fl += 8.0 * g.M * (double)g.N * g.K;
            by += gemm_bytes(g);
        }
        const size_t u0 = sc.hunit.size();
        gemm_units(simt, (int)sc.hgemm.size(), sc.hunit);
        sc.hgemm.insert(sc.hgemm.end(), simt.begin(), simt.end());
        const unsigned nu = (unsigned)(sc.hunit.size() - u0);
        sc.launches.push_back({[psc, u0, nu](cudaStream_t st) {
            k_gemm<T><<<nu, GemmCfg<T>::TH, 0, st>>>(psc->gemm.p, psc->unit.p + u0);
        }, LK_GEMM, fl, by});
    }

    // Allocates the shared tensor-core workspace and builds the tensor maps of
    // every pending tensor-core launch of a schedule.
    int finish_tc(Schedule<T> &sc)
    {
        if constexpr (std::is_same<T, float>::value) {
            long long need = 0;
            for (auto &v : sc.tc_pending) need = std::max(need, tc_workspace_floats(v.data(), (int)v.size()));
            if (need > 0 && tcws_base() == nullptr) {
                // first user of the shared workspace sizes it
                std::lock_guard<std::mutex> lk(ws->mu);
                if (ws->tcws.n == 0) {
                    int rc = ws->tcws.alloc(need);
                    if (rc) return rc;
                }
            }
            if (need > (long long)tcws_size()) {
                int rc = own_tcws.alloc(need);
                if (rc) return rc;
                // schedules built earlier point into the old workspace: rebuild their maps
                for (auto *o : built_tc) {
                    for (size_t i = 0; i < o->tc_pending.size(); i++) {
                        o->tc[i].reset(new TcLaunch());
                        if ((rc = tc_build_launch(*o->tc[i], o->tc_pending[i].data(), (int)o->tc_pending[i].size(),
                                                  tcws_base())))
                            return rc;
                    }
                    if (o->graph) { cudaGraphExecDestroy(o->graph); o->graph = nullptr; }
                }
            }
            sc.tc.clear();
            for (auto &v : sc.tc_pending) {
                sc.tc.emplace_back(new TcLaunch());
                int rc = tc_build_launch(*sc.tc.back(), v.data(), (int)v.size(), tcws_base());
                if (rc) return rc;
            }
            built_tc.push_back(&sc);
        }
        return WT3D_OK;
    }

    // The inverses of the diagonal blocks that end in [k0, k1) of the fronts fl,
    // once the panels [p0, end) of hp are factored.  Off the factorisation's
    // chain (only the substitutions read them): a branch of its graph.
    void push_inverses(Schedule<T> &sc, const std::vector<int> &fl, const std::vector<PanelTask> &hp, size_t p0,
                       std::vector<InvTask> &hi, int k0, int k1)
    {
        Schedule<T> *psc = &sc;
        const int np = (int)(hp.size() - p0);
        if (np) {
            sc.launches.push_back({[psc, this, p0, np](cudaStream_t st) {
                k_tile_inverse<T><<<4 * np, BD_TH, BandCfg<T, 1>::smem, st>>>(psc->panel.p + p0, fr.p, fac.p, gord.p, ipiv.p, binv.p);
            }, LK_PANEL, 0});
            sc.launches.back().side = true;
        }
        const size_t i0 = hi.size();
        for (int f : fl) {
            const int p = S->fronts[f].p;
            for (int c0 = 0; c0 < p; c0 += SBW) {
                const int end = std::min(c0 + SBW, p), w = end - c0, nt = (w + KB - 1) / KB;
                if (end - 1 < k0 || end - 1 >= k1) continue;
                for (int up = 0; up < 2; up++)
                    for (int t = 0; t < nt; t++) {
                        if (up ? t == 0 : t == nt - 1) continue;
                        for (int h = 0; h < 2; h++)
                            if (KB * t + IV_N * h < w) hi.push_back(InvTask{f, c0, t, h, up});
                    }
            }
        }
        // longest chains first
        std::stable_sort(hi.begin() + i0, hi.end(), [this](const InvTask &a, const InvTask &b) {
            auto len = [this](const InvTask &x) {
                return x.upper ? x.t : (std::min(SBW, S->fronts[x.f].p - x.c0) + KB - 1) / KB - 1 - x.t;
            };
            return len(a) > len(b);
        });
        const int ni = (int)(hi.size() - i0);
        if (ni) {
            sc.launches.push_back({[psc, this, i0, ni](cudaStream_t st) {
                k_block_inverse<T><<<ni, IV_TH, 0, st>>>(psc->inv.p + i0, fr.p, fac.p, gord.p, binv.p);
            }, LK_PANEL, 0});
            sc.launches.back().side = true;
        }
    }

    int build_factor_schedule()
    {
        auto sc = std::make_unique<Schedule<T>>();
        std::vector<PanelTask> hp;
        std::vector<BandTask> hb;
        std::vector<GemmTask<T>> hg;
        std::vector<EATask> he;
        std::vector<EAUnit> heu;
        std::vector<int> hpos;
        std::vector<InvTask> hi;
        Schedule<T> *psc = sc.get();
        const Symbolic &sym = *S;
        cx<T> *F = fac.p;
        cx<T> *U[2] = {ws->upd0.p, ws->upd1.p};
        // zero the factor pool, scale and scatter the operator
        {
            cx<T> *fp = F; size_t bytes = fac.n * sizeof(cx<T>);
            long long *mp = map.p;
            Engine<T> *self = this;
            const long long n = sym.n;
            sc->launches.push_back({[fp, bytes](cudaStream_t st) { cudaMemsetAsync(fp, 0, bytes, st); }, LK_MEMSET, 0});
            sc->launches.push_back({[self, n](cudaStream_t st) {
                k_jacobi_scale<<<ceil_div(n, 256), 256, 0, st>>>(n, self->d_irptr, self->d_jcptr, self->a_dev,
                                                                 self->scale.p);
            }, LK_SCATTER, 0});
            sc->launches.push_back({[self, mp, n, fp](cudaStream_t st) {
                k_scatter<T><<<ceil_div(n, 256), 256, 0, st>>>(n, self->d_irptr, self->d_jcptr, mp, self->a_dev,
                                                               self->scale.p, fp);
            }, LK_SCATTER, 0});
        }
        const int nlev = (int)sym.levels.size();
        for (int L = nlev - 1; L >= 0; L--) {
            const std::vector<int> &fl = sym.levels[L];
            // what the children left, into the factor pool and this level's update
            // region (all of it: zeros where no child contributes)
            {
                const size_t u0 = heu.size();
                for (int f : fl) {
                    const Front &P = sym.fronts[f];
                    EATask t{f, -1, -1, 0, 0};
                    for (int s = 0; s < P.nchild; s++) {
                        const Front &C = sym.fronts[P.child[s]];
                        if (C.b == 0) continue;
                        const size_t o = hpos.size();
                        hpos.resize(o + P.nf(), -1);
                        for (int i = 0; i < C.b; i++) hpos[o + sym.rel[C.border_off + i]] = i;
                        (t.child0 < 0 ? t.child0 : t.child1) = P.child[s];
                        (t.child1 < 0 ? t.pos0 : t.pos1) = (long long)o;
                    }
                    const int first = t.child0 < 0 ? P.p : 0;   // a leaf only has zeros to write
                    for (int r = first; r < P.nf(); r += EA_ROWS) heu.push_back(EAUnit{(int)he.size(), r});
                    he.push_back(t);
                }
                const unsigned nu = (unsigned)(heu.size() - u0);
                if (nu)
                    sc->launches.push_back({[psc, this, u0, nu](cudaStream_t st) {
                        k_extend_add<T><<<nu, 32 * EA_ROWS, 0, st>>>(psc->ea.p, psc->eau.p + u0, fr.p, eapos.p, fac.p,
                                                                     ws->upd0.p, ws->upd1.p);
                    }, LK_EXTEND_ADD, 0});
            }
            // Two-level blocked partial LU, level-synchronous over fronts.
            // Inner KB-wide panels: panel LU, row band (all columns right of
            // the panel), column band (all rows below), and updates confined to
            // the rows or the columns of the current WB-wide outer block, by
            // recursive halving: after 1, 2, 4 .. panels the rows and columns of
            // as many next panels receive one update of rank 64, 128, 256 ..
            // (a rank-64 update of the whole rest after every panel moves the
            // outer block's rows and columns 28 times instead of 12).  Once an
            // outer block is done, the rows and columns below and right of it
            // receive one rank-WB update, so most of the elimination runs as
            // K = WB GEMMs on the tensor cores.
            int maxp = 0;
            for (int f : fl) maxp = std::max(maxp, sym.fronts[f].p);
            for (int c0 = 0; c0 < maxp; c0 += WB) {
                const size_t pblk = hp.size();   // first panel of this outer block
                for (int k = c0; k < std::min(c0 + WB, maxp); k += KB) {
                    const size_t p0 = hp.size(), b0 = hb.size();
                    // panels the next update covers: the largest power of two that
                    // divides the number of panels done in this outer block
                    const int done = (k - c0) / KB + 1, s = done & -done;
                    // band vectors of the step: two per four threads if they fill the chip
                    long long nvec = 0;
                    for (int f : fl)
                        if (sym.fronts[f].p > k)
                            nvec += 2LL * std::max(0, sym.fronts[f].p - k - KB) + 2LL * sym.fronts[f].b;
                    const bool two = nvec >= BAND_TWO;
                    const int bv = two ? BandCfg<T, 2>::V : BandCfg<T, 1>::V;
                    for (int f : fl) {
                        const Front &Fr = sym.fronts[f];
                        if (Fr.p <= k) continue;
                        const int nf = Fr.nf(), kb = std::min(KB, Fr.p - k), k2 = k + kb;
                        const int cend = std::min(c0 + WB, Fr.p);
                        hp.push_back(PanelTask{f, k});
                        for (int c = k2; c < nf; c += bv) hb.push_back(BandTask{f, k, c, 0});
                        for (int r = k2; r < Fr.p; r += bv) hb.push_back(BandTask{f, k, r, 1});
                        for (int r = 0; r < Fr.b; r += bv) hb.push_back(BandTask{f, k, r, 2});
                        if (k2 >= cend) continue;
                        cx<T> *Pb = F + Fr.fac_off;
                        cx<T> *Lo = Pb + (long long)Fr.p * nf;
                        const int ks = k2 - s * KB, t1 = std::min(k2 + s * KB, cend), w = k2 - ks;
                        // the rows of the next s panels, every column right of them
                        add_gemm(hg, Pb + (long long)k2 * nf + ks, nf, Pb + (long long)ks * nf + k2, nf,
                                 Pb + (long long)k2 * nf + k2, nf, t1 - k2, nf - k2, w);
                        // their columns, the rows below
                        add_gemm(hg, Pb + (long long)t1 * nf + ks, nf, Pb + (long long)ks * nf + k2, nf,
                                 Pb + (long long)t1 * nf + k2, nf, Fr.p - t1, t1 - k2, w);
                        add_gemm(hg, Lo + ks, Fr.p, Pb + (long long)ks * nf + k2, nf, Lo + k2, Fr.p, Fr.b, t1 - k2, w);
                    }
                    const int np = (int)(hp.size() - p0), nbd = (int)(hb.size() - b0);
                    sc->launches.push_back({[psc, this, p0, np](cudaStream_t st) {
                        k_panel<T><<<np, 256, panel_smem<T>(), st>>>(psc->panel.p + p0, fr.p, fac.p, maxabs.p, pivot_rel, npert.p, gord.p);
                    }, LK_PANEL, 0});
                    if (nbd)
                        sc->launches.push_back({[psc, this, b0, nbd, two](cudaStream_t st) {
                            if (two)
                                k_bands<T, 2><<<nbd, BD_TH, BandCfg<T, 2>::smem, st>>>(psc->band.p + b0, fr.p, fac.p,
                                                                                       gord.p);
                            else
                                k_bands<T, 1><<<nbd, BD_TH, BandCfg<T, 1>::smem, st>>>(psc->band.p + b0, fr.p, fac.p,
                                                                                       gord.p);
                        }, LK_TRSM, 0});
                    push_gemm_launch(*sc, hg);
                }
                push_inverses(*sc, fl, hp, pblk, hi, c0, std::min(c0 + WB, maxp));
                // rank-WB update of everything below and right of the outer block
                for (int f : fl) {
                    const Front &Fr = sym.fronts[f];
                    if (Fr.p <= c0) continue;
                    const int nf = Fr.nf(), cend = std::min(c0 + WB, Fr.p), w = cend - c0;
                    cx<T> *Pb = F + Fr.fac_off;
                    cx<T> *Lo = Pb + (long long)Fr.p * nf;
                    add_gemm(hg, Pb + (long long)cend * nf + c0, nf, Pb + (long long)c0 * nf + cend, nf,
                             Pb + (long long)cend * nf + cend, nf, Fr.p - cend, nf - cend, w);
                    add_gemm(hg, Lo + c0, Fr.p, Pb + (long long)c0 * nf + cend, nf, Lo + cend, Fr.p, Fr.b,
                             Fr.p - cend, w);
                }
                push_gemm_launch(*sc, hg);
            }
            // Schur complement F22 -= L21 U12 (K = p)
            {
                for (int f : fl) {
                    const Front &Fr = sym.fronts[f];
                    if (Fr.b == 0) continue;
                    const int nf = Fr.nf();
                    cx<T> *Pb = F + Fr.fac_off;
                    cx<T> *Lo = Pb + (long long)Fr.p * nf;
                    add_gemm(hg, Lo, Fr.p, Pb + Fr.p, nf, U[L & 1] + Fr.upd_off, Fr.b, Fr.b, Fr.b, Fr.p);
                }
                push_gemm_launch(*sc, hg);
            }
        }
        int rc;
        if ((rc = sc->panel.upload(hp))) return rc;
        if ((rc = sc->band.upload(hb))) return rc;
        if ((rc = sc->gemm.upload(sc->hgemm)) || (rc = sc->unit.upload(sc->hunit))) return rc;
        sc->hgemm.clear();
        sc->hunit.clear();
        if ((rc = sc->ea.upload(he)) || (rc = sc->eau.upload(heu)) || (rc = eapos.upload(hpos))) return rc;
        if ((rc = sc->inv.upload(hi))) return rc;
        if ((rc = finish_tc(*sc))) return rc;
        fsched = std::move(sc);
        return WT3D_OK;
    }

    // One product of a substitution pass: out (=, -=) op(A) in, A a factor block
    // or (flags SK_LOWER / SK_UPPER) a packed block inverse.
    struct Product {
        const cx<T> *A;
        int lda, M, K;
        const int *bmap;   // input rows bmap[k], or b0 + k
        int b0;
        const int *cmap;   // output rows cmap[i], or c0 + i
        int c0;
        int flags;
    };

    // Appends the launches of the products of one step.
    void push_products(Schedule<T> &sc, std::vector<SkUnit> &hu, std::vector<Product> v, bool herm, const cx<T> *in,
                       cx<T> *out, int m)
    {
        const int nc = sk_columns(m);
        Schedule<T> *psc = &sc;
        if (v.empty()) return;
        // K range of the 64 rows from r0: all of it, or the triangle's part
        auto range = [&](const Product &q, int r0, int &k0, int &k1) {
            k0 = 0;
            k1 = q.K;
            if (!(q.flags & (SK_LOWER | SK_UPPER))) return;
            if (((q.flags & SK_LOWER) != 0) != herm) k1 = std::min(q.K, r0 + SK_M);
            else k0 = r0;
        };
        double work = 0, fl = 0;
        for (const Product &q : v)
            for (int r0 = 0; r0 < q.M; r0 += SK_M) {
                int k0, k1;
                range(q, r0, k0, k1);
                work += k1 - k0;
                fl += 8.0 * std::min(SK_M, q.M - r0) * (double)(k1 - k0) * m;
            }
        // K chunk for about SK_SLOTS units
        const int chunk = std::min<long long>(SK_KMAX, std::max<long long>(SK_KMIN, (long long)(work / SK_SLOTS / 64 + 1) * 64));
        const size_t u0 = hu.size();
        for (const Product &q : v)
            for (int r0 = 0; r0 < q.M; r0 += SK_M) {
                int k0, k1;
                range(q, r0, k0, k1);
                const int n = std::max(1, (k1 - k0 + chunk / 2) / chunk);   // chunks of about the same length
                const int len = std::min<int>(SK_KMAX, ((k1 - k0 + n - 1) / n + 31) / 32 * 32);
                for (int k = k0; k < k1; k += len) {
                    SkUnit u{};
                    u.A = herm ? q.A + (long long)k * q.lda + r0 : q.A + (long long)r0 * q.lda + k;
                    u.bmap = q.bmap ? q.bmap + k : nullptr;
                    u.b0 = q.b0 + k;
                    u.cmap = q.cmap ? q.cmap + r0 : nullptr;
                    u.c0 = q.c0 + r0;
                    u.lda = q.lda;
                    u.M = std::min(SK_M, q.M - r0);
                    u.K = std::min(len, k1 - k);
                    u.flags = q.flags | (k1 - k0 > len ? SK_ATOM : 0);
                    u.d = k - r0;
                    hu.push_back(u);
                }
            }
        const int nu = (int)(hu.size() - u0);
        const bool tri = (v[0].flags & (SK_LOWER | SK_UPPER)) != 0;
        const double by = fl / m * sizeof(cx<T>) / 8;
        if constexpr (std::is_same<T, float>::value)
            if (use_ts && sk_tensor(nc, chunk)) {
                sc.launches.push_back({[psc, u0, nu, nc, herm, in, out](cudaStream_t st) {
                    sk_tensor_launch(nc, herm, psc->sk.p + u0, nu, in, out, st);
                }, tri ? LK_SUBSTEP : LK_TCGEMM, fl, by});
                return;
            }
        const bool gemv = nc == 1 && (herm || (sizeof(T) == 4 && (double)fac.n >= GEMV_MIN_ENTRIES));
        sc.launches.push_back({[psc, u0, nu, nc, gemv, herm, in, out](cudaStream_t st) {
            sk_launch(nc, gemv, herm, psc->sk.p + u0, nu, in, out, st);
        }, tri ? LK_SUBSTEP : LK_GEMM, fl, by});
    }

    // Solve schedule for m right-hand sides: X (sources, new ordering) to Y.
    // Every level of a sweep walks the SBW-wide diagonal blocks of its fronts: the
    // block inverse gives the block's unknowns, then the rows outside the block
    // are updated with them.
    Schedule<T> *solve_schedule(int m, bool adjoint)
    {
        auto it = ssched[adjoint].find(m);
        if (it != ssched[adjoint].end()) return it->second.get();
        auto sc = std::make_unique<Schedule<T>>();
        std::vector<SkUnit> hu;
        const Symbolic &sym = *S;
        const int nlev = (int)sym.levels.size();
        auto block = [&](int f, int c0) {   // the packed inverse of block c0
            return binv.p + hfr[f].inv + (long long)(c0 / SBW) * SBW * SBW;
        };
        // ---- forward sweep: leaves to root ----
        for (int L = nlev - 1; L >= 0; L--) {
            const std::vector<int> &fl = sym.levels[L];
            int maxp = 0;
            for (int f : fl) maxp = std::max(maxp, sym.fronts[f].p);
            for (int c0 = 0; c0 < maxp; c0 += SBW) {
                std::vector<Product> ap, up;
                for (int f : fl) {
                    const Front &Fr = sym.fronts[f];
                    if (Fr.p <= c0) continue;
                    const int nf = Fr.nf(), cend = std::min(c0 + SBW, Fr.p), w = cend - c0, r = Fr.first + c0;
                    const cx<T> *Pb = fac.p + Fr.fac_off;
                    const cx<T> *W = block(f, c0);
                    if (!adjoint) ap.push_back({W, inv_ld(w), w, w, gord.p + r, 0, nullptr, r, SK_LOWER});
                    else ap.push_back({W, inv_ld(w), w, w, nullptr, r, nullptr, r, SK_UPPER});
                    if (cend == Fr.p) continue;
                    if (!adjoint)   // x[cend:p] -= L[cend:p, c0:cend] z[c0:cend]
                        up.push_back({Pb + (long long)cend * nf + c0, nf, Fr.p - cend, w, nullptr, r, nullptr,
                                      Fr.first + cend, SK_SUB});
                    else            // x[cend:p] -= U[c0:cend, cend:p]^H z[c0:cend]
                        up.push_back({Pb + (long long)c0 * nf + cend, nf, Fr.p - cend, w, nullptr, r, nullptr,
                                      Fr.first + cend, SK_SUB});
                }
                push_products(*sc, hu, std::move(ap), adjoint, X.p, Z.p, m);
                push_products(*sc, hu, std::move(up), adjoint, Z.p, X.p, m);
            }
            // x[border] -= L21 z   (adjoint: U12^H z); siblings share border rows
            std::vector<Product> bo;
            for (int f : fl) {
                const Front &Fr = sym.fronts[f];
                if (Fr.b == 0) continue;
                const cx<T> *Pb = fac.p + Fr.fac_off, *Lo = Pb + (long long)Fr.p * Fr.nf();
                bo.push_back({adjoint ? Pb + Fr.p : Lo, adjoint ? Fr.nf() : Fr.p, Fr.b, Fr.p, nullptr, Fr.first,
                              border.p + Fr.border_off, 0, SK_SUB | SK_ATOM});
            }
            push_products(*sc, hu, std::move(bo), adjoint, Z.p, X.p, m);
        }
        // ---- backward sweep: root to leaves ----
        for (int L = 0; L < nlev; L++) {
            const std::vector<int> &fl = sym.levels[L];
            int maxp = 0;
            std::vector<Product> bo;
            for (int f : fl) {
                const Front &Fr = sym.fronts[f];
                maxp = std::max(maxp, Fr.p);
                if (Fr.b == 0) continue;
                const cx<T> *Pb = fac.p + Fr.fac_off, *Lo = Pb + (long long)Fr.p * Fr.nf();
                // z -= U12 y[border]   (adjoint: L21^H y[border])
                bo.push_back({adjoint ? Lo : Pb + Fr.p, adjoint ? Fr.p : Fr.nf(), Fr.p, Fr.b,
                              border.p + Fr.border_off, 0, nullptr, Fr.first, SK_SUB});
            }
            push_products(*sc, hu, std::move(bo), adjoint, Y.p, Z.p, m);
            for (int c0 = (maxp - 1) / SBW * SBW; c0 >= 0; c0 -= SBW) {
                std::vector<Product> ap, up;
                for (int f : fl) {
                    const Front &Fr = sym.fronts[f];
                    if (Fr.p <= c0) continue;
                    const int nf = Fr.nf(), w = std::min(c0 + SBW, Fr.p) - c0, r = Fr.first + c0;
                    const cx<T> *Pb = fac.p + Fr.fac_off;
                    const cx<T> *W = block(f, c0);
                    if (!adjoint) ap.push_back({W, inv_ld(w), w, w, nullptr, r, nullptr, r, SK_UPPER});
                    else ap.push_back({W, inv_ld(w), w, w, nullptr, r, gord.p + r, 0, SK_LOWER});
                    if (c0 == 0) continue;
                    // z[0:c0] -= U[0:c0, c0:cend] y[c0:cend]   (adjoint: L[c0:cend, 0:c0]^H)
                    up.push_back({adjoint ? Pb + (long long)c0 * nf : Pb + c0, nf, c0, w, nullptr, r, nullptr,
                                  Fr.first, SK_SUB});
                }
                push_products(*sc, hu, std::move(ap), adjoint, Z.p, Y.p, m);
                push_products(*sc, hu, std::move(up), adjoint, Y.p, Z.p, m);
            }
        }
        if (sc->sk.upload(hu)) return nullptr;
        Schedule<T> *ret = sc.get();
        ssched[adjoint][m] = std::move(sc);
        return ret;
    }

    const double2 *a_dev = nullptr;   // complex128 operator values (set before factor)

    int run(Schedule<T> &sc, cudaStream_t st)
    {
        if (use_graphs) {
            if (!sc.graph) {
                cudaGraph_t g;
                WT_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                bool forked = false, behind = true;   // behind: the main branch has moved on since the last fork
                for (auto &l : sc.launches) {
                    if (l.side && behind) {
                        cudaEventRecord(side_ev, st);
                        cudaStreamWaitEvent(side, side_ev, 0);
                        forked = true;
                        behind = false;
                    }
                    l.fn(l.side ? side : st);
                    if (!l.side) behind = true;
                }
                if (forked) {
                    cudaEventRecord(side_ev, side);
                    cudaStreamWaitEvent(st, side_ev, 0);
                }
                WT_CUDA(cudaStreamEndCapture(st, &g));
                cudaError_t e = cudaGraphInstantiate(&sc.graph, g, 0);
                cudaGraphDestroy(g);
                if (e != cudaSuccess) {
                    set_error(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
                    sc.graph = nullptr;
                    return WT3D_ERR_CUDA;
                }
            }
            WT_CUDA(cudaGraphLaunch(sc.graph, st));
        } else {
            for (auto &l : sc.launches) l.fn(st);
        }
        WT_CUDA(cudaGetLastError());
        return WT3D_OK;
    }

    // Factorisation with one event pair around every launch (no graph):
    // out[k] = milliseconds spent in launches of kind k, out[LK_NKINDS] =
    // GEMM real flops, out[LK_NKINDS+1] = GEMM launches.
    // Runs a schedule once with an event pair around every launch; ms[i] per launch.
    int profile_each(Schedule<T> &sc, cudaStream_t st, std::vector<float> &ms)
    {
        const size_t nl = sc.launches.size();
        std::vector<cudaEvent_t> ev(2 * nl);
        for (auto &e : ev) WT_CUDA(cudaEventCreate(&e));
        for (size_t i = 0; i < nl; i++) {
            WT_CUDA(cudaEventRecord(ev[2 * i], st));
            sc.launches[i].fn(st);
            WT_CUDA(cudaEventRecord(ev[2 * i + 1], st));
        }
        WT_CUDA(cudaStreamSynchronize(st));
        ms.assign(nl, 0.f);
        for (size_t i = 0; i < nl; i++) cudaEventElapsedTime(&ms[i], ev[2 * i], ev[2 * i + 1]);
        for (auto &e : ev) cudaEventDestroy(e);
        WT_CUDA(cudaGetLastError());
        return WT3D_OK;
    }

    // The factor schedule under profile_each (the factorisation is complete afterwards).
    int profile_factor_each(const double2 *d_a, long long nnz, cudaStream_t st, std::vector<float> &ms)
    {
        a_dev = d_a;
        WT_CUDA(cudaMemsetAsync(maxabs.p, 0, sizeof(unsigned long long), st));
        k_maxabs<<<1216, 256, 0, st>>>(nnz, d_a, maxabs.p);
        return profile_each(*fsched, st, ms);
    }

    int profile_factor(const double2 *d_a, long long nnz, cudaStream_t st, double *out)
    {
        a_dev = d_a;
        WT_CUDA(cudaMemsetAsync(maxabs.p, 0, sizeof(unsigned long long), st));
        k_maxabs<<<1216, 256, 0, st>>>(nnz, d_a, maxabs.p);
        const size_t nl = fsched->launches.size();
        std::vector<cudaEvent_t> ev(2 * nl);
        for (auto &e : ev) WT_CUDA(cudaEventCreate(&e));
        for (size_t i = 0; i < nl; i++) {
            WT_CUDA(cudaEventRecord(ev[2 * i], st));
            fsched->launches[i].fn(st);
            WT_CUDA(cudaEventRecord(ev[2 * i + 1], st));
        }
        WT_CUDA(cudaStreamSynchronize(st));
        for (int k = 0; k < LK_NKINDS + 2; k++) out[k] = 0;
        for (size_t i = 0; i < nl; i++) {
            float ms = 0;
            cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]);
            out[fsched->launches[i].kind] += ms;
            if (fsched->launches[i].kind == LK_GEMM || fsched->launches[i].kind == LK_TCGEMM) {
                out[LK_NKINDS] += fsched->launches[i].flops;
                out[LK_NKINDS + 1] += 1;
            }
        }
        for (auto &e : ev) cudaEventDestroy(e);
        WT_CUDA(cudaGetLastError());
        return WT3D_OK;
    }

    // One pass of a solve schedule with an event pair per launch: out[k] = ms of kind k.
    int profile_schedule(Schedule<T> &sc, cudaStream_t st, double *out)
    {
        const size_t nl = sc.launches.size();
        std::vector<cudaEvent_t> ev(2 * nl);
        for (auto &e : ev) WT_CUDA(cudaEventCreate(&e));
        for (size_t i = 0; i < nl; i++) {
            WT_CUDA(cudaEventRecord(ev[2 * i], st));
            sc.launches[i].fn(st);
            WT_CUDA(cudaEventRecord(ev[2 * i + 1], st));
        }
        WT_CUDA(cudaStreamSynchronize(st));
        for (int k = 0; k < LK_NKINDS + 2; k++) out[k] = 0;
        for (size_t i = 0; i < nl; i++) {
            float ms = 0;
            cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]);
            out[sc.launches[i].kind] += ms;
            if (sc.launches[i].kind == LK_GEMM || sc.launches[i].kind == LK_TCGEMM) {
                out[LK_NKINDS] += sc.launches[i].flops;
                out[LK_NKINDS + 1] += 1;
            }
        }
        for (auto &e : ev) cudaEventDestroy(e);
        return WT3D_OK;
    }

    int factor(const double2 *d_a, long long nnz, cudaStream_t st, int *h_npert)
    {
        if (d_a != a_dev && fsched->graph) { cudaGraphExecDestroy(fsched->graph); fsched->graph = nullptr; }
        a_dev = d_a;
        WT_CUDA(cudaMemsetAsync(maxabs.p, 0, sizeof(unsigned long long), st));
        k_maxabs<<<1216, 256, 0, st>>>(nnz, d_a, maxabs.p);
        WT_CUDA(cudaMemsetAsync(npert.p, 0, sizeof(int), st));
        int rc = run(*fsched, st);
        if (rc) return rc;
        if (h_npert) {
            WT_CUDA(cudaMemcpyAsync(h_npert, npert.p, sizeof(int), cudaMemcpyDeviceToHost, st));
        }
        return WT3D_OK;
    }

};

}  // namespace wt3d
