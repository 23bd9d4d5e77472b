// Batches of independent VMC problems advanced together (nqs_gpu_batch_*).
//
// Every instance has its own Hamiltonian, lattice, ansatz, sampler and
// workspaces; a batch step runs, for each instance, the derived-table rebuild,
// the Philox chains, the FP32 estimator (local energies + Jacobian), the energy
// statistics and ESS, the column means, the centring / TF32 split and the
// tensor-core Gram, then ONE cooperative launch that factors, inverts and
// refines the systems of all instances (each instance owns a range of CTAs with
// its own grid barrier), then per instance delta = O_c^T y / N_s (sample space)
// and the update.  The first step runs uncaptured and autotunes the split of
// the cooperative launch's CTAs between the instances (balanced by the systems'
// solve times measured on the Grams of that step); from the second step the whole
// sequence is one CUDA graph replayed per step, the samplers' move counters
// living in device memory so that each replay draws new random numbers.
#include <algorithm>
#include <math.h>
#include <stdlib.h>

#include "nqs_amp.cuh"

namespace nqs {

struct Sampler;
bool sampler_produce_dev(Sampler *sm, int n, uint64_t **d_out, unsigned long long *move_dev);
void sampler_host_advance(Sampler *sm, int n);
uint64_t sampler_move_counter(const Sampler *sm);
int sampler_chains(const Sampler *sm);
const unsigned long long *sampler_counts(const Sampler *sm);
bool sampler_fp32(const Sampler *sm);

// A step's words of one instance in pinned memory, written by its update kernel (five copies of a few
// bytes per instance were five nodes of the batch's graph).
struct BatchWords {
    double scal[16], nrm[2];
    unsigned long long counts[2];        // sampler: accepted, proposed
    int status, err;                     // of the mixed solve
};

struct BatchInst {
    nqs_config_t cfg{};
    int sx = 0, sy = 0;
    Ansatz *a = nullptr;
    Sampler *s = nullptr;
    nqs_log_amp_fn_t fn = nullptr;
    void *user = nullptr;
    DevAmp A{};
    DevHam H{};
    int Ns = 0, C = 0;
    long P = 0;
    DevBuf<double> E, Ei, eps, O, gm, scal, delta, y, part, es;
    DevBuf<unsigned long long> move;
    MixedSys *mx = nullptr;
    BatchWords *h = nullptr;  // pinned: the step's words
    int fp64_fallback = 0, fp64_conv = 0;   // last step solved in FP64 after an FP32 breakdown
    ~BatchInst() {
        if (mx) mixed_sys_free(mx);
        if (h) cudaFreeHost(h);
    }
};

struct Batch {
    std::vector<BatchInst *> inst;
    MixedBatch *mb = nullptr;
    std::vector<int> ctas;
    int bd_from = 0;                     // systems of order >= bd_from use 128-wide diagonal blocks
    std::vector<double> tune_ms;
    cudaGraphExec_t exec = nullptr;
    long graph_kernels = 0;
    int steps = 0;
    long fallbacks = 0;                  // instance steps re-solved in FP64
    int sweeps = 5, passes = 3, space = 0;
    std::vector<cudaStream_t> side;      // instances' work forks onto these and joins the main stream
    std::vector<cudaEvent_t> join;
    cudaEvent_t fork = nullptr;
    ~Batch() {
        if (exec) cudaGraphExecDestroy(exec);
        for (cudaStream_t s : side) cudaStreamDestroy(s);
        for (cudaEvent_t e : join) cudaEventDestroy(e);
        if (fork) cudaEventDestroy(fork);
        if (mb) mixed_batch_free(mb);
        for (BatchInst *b : inst) delete b;
    }
};

// True when the mixed solve of an instance broke down: a non-positive FP32
// pivot, or a CG residual above the bound (nrm = |r|^2, |rhs|^2).
__host__ __device__ inline bool mixed_broken(int status, const double *nrm) {
    const double rel = nrm[1] > 0.0 ? sqrt(nrm[0] / nrm[1]) : 0.0;
    return status >= 0 || !(rel <= MIXED_RESID_MAX);
}

// theta -= lr delta and ||delta||^2, with delta = 0 when the instance's mixed
// solve broke down or its kernels reported an error (decided by one thread: the
// test's FP64 division and square root cost 16 cycles per warp instruction on this
// GPU's FP64 pipe).
// host, when given, receives the step's words.
__global__ void k_batch_apply(double *params, const double *__restrict__ delta, long P, double lr, double *scal,
                              const int *mstatus, const int *merr, const double *mnrm, int unconditional,
                              BatchWords *host, const unsigned long long *counts) {
    __shared__ double red[1024];
    __shared__ bool zero_s;
    if (threadIdx.x == 0) zero_s = !unconditional && (mixed_broken(mstatus[0], mnrm) || merr[0] != 0);
    __syncthreads();
    const bool zero = zero_s;
    double s = 0.0;
    for (long k = threadIdx.x; k < P; k += blockDim.x) {
        const double d = zero ? 0.0 : delta[k];
        params[k] += -lr * d;
        s += d * d;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) scal[S_NORM2] = red[0];
    if (!host) return;
    if (threadIdx.x < 16) host->scal[threadIdx.x] = threadIdx.x == S_NORM2 ? red[0] : scal[threadIdx.x];
    if (threadIdx.x < 2) {
        host->nrm[threadIdx.x] = mnrm[threadIdx.x];
        host->counts[threadIdx.x] = counts[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        host->status = mstatus[0];
        host->err = merr[0];
    }
}

bool enqueue_gated_apply(double *params, const double *delta, long P, double lr, double *scal, const int *mstatus,
                         const int *merr, const double *mnrm) {
    NQS_LAUNCH("apply_update");
    k_batch_apply<<<1, 1024, 0, ctx().stream>>>(params, delta, P, lr, scal, mstatus, merr, mnrm, 0, nullptr, nullptr);
    return NQS_CUDA(cudaGetLastError());
}

static bool enqueue_front(BatchInst &b, cudaStream_t st) {
    uint64_t *bits = nullptr;
    if (!ansatz_refresh_derived(b.a) || !sampler_produce_dev(b.s, b.Ns, &bits, b.move.p) ||
        !launch_local_estimator(b.A, b.H, bits, b.Ns, b.E.p, b.Ei.p, b.O.p, nullptr, 1, true) ||
        !enqueue_energy_stats(b.E.p, b.Ns, b.C, b.scal.p, b.eps.p, b.es.p, ctx().stream) ||
        !enqueue_col_means(b.O.p, b.Ns, b.P, b.scal.p, b.gm.p, b.part.p))
        return false;
    mixed_sys_front(b.mx, st, true);
    return NQS_CUDA(cudaGetLastError());
}

static bool enqueue_back(BatchInst &b, cudaStream_t st) {
    if (!mixed_sys_param_space(b.mx) && !enqueue_col_dot(b.O.p, b.Ns, b.P, b.y.p, 1.0 / (double)b.Ns, b.delta.p))
        return false;
    {
        NQS_LAUNCH("apply_update");
        k_batch_apply<<<1, 1024, 0, st>>>(b.a->d_params.p, b.delta.p, b.P, b.cfg.learning_rate, b.scal.p,
                                          mixed_sys_status(b.mx), mixed_sys_err(b.mx), mixed_sys_nrm(b.mx), 0, b.h,
                                          sampler_counts(b.s));
    }
    return NQS_CUDA(cudaGetLastError()) && NQS_CUDA(cudaMemcpyAsync(b.a->h_params, b.a->d_params.p, sizeof(double) * b.P,
                                                                   cudaMemcpyDeviceToHost, st));
}

// Run `work(instance)` for every instance on the side streams (instance i on
// stream i mod S, the library's launches redirected there), forked from and
// joined back into the main stream: independent instances overlap, and in a
// captured sequence they become parallel branches of the graph.
template <typename F>
static bool fork_join(Batch &B, cudaStream_t main, F work) {
    Context &c = ctx();
    if (!NQS_CUDA(cudaEventRecord(B.fork, main))) return false;
    for (cudaStream_t s : B.side)
        if (!NQS_CUDA(cudaStreamWaitEvent(s, B.fork, 0))) return false;
    bool ok = true;
    for (size_t i = 0; i < B.inst.size() && ok; i++) {
        c.stream = B.side[i % B.side.size()];
        ok = work(*B.inst[i], c.stream);
    }
    c.stream = main;
    for (size_t k = 0; k < B.side.size(); k++)
        ok = ok && NQS_CUDA(cudaEventRecord(B.join[k], B.side[k])) &&
             NQS_CUDA(cudaStreamWaitEvent(main, B.join[k], 0));
    return ok;
}

// Splits of the cooperative launch's CTAs between the instances to start from: the largest equal
// counts (a power of two) and counts proportional to the order n_i of instance i's system, within
// the co-resident limit.
static std::vector<std::vector<int>> cta_starts(const Batch &B, int cap) {
    const int K = (int)B.inst.size();
    std::vector<std::vector<int>> c;
    int u = 1;
    while (2 * u * K <= cap && u < 32) u *= 2;
    c.push_back(std::vector<int>((size_t)K, u));
    double tot = 0.0;
    for (BatchInst *b : B.inst) tot += (double)mixed_sys_order(b->mx);
    std::vector<int> prop((size_t)K);
    for (int i = 0; i < K; i++)
        prop[i] = (int)floor((double)mixed_sys_order(B.inst[i]->mx) / tot * (double)(cap - K)) + 1;
    c.push_back(prop);
    return c;
}

// One system's solve times by CTA count, t = c + w / g through the two counts nearest to g.
struct SolveTimes {
    std::map<int, double> at;
    void line(int g, double &c, double &w) const {
        int g1 = -1, g2 = -1;
        for (const auto &e : at) {
            if (g1 < 0 || abs(e.first - g) < abs(g1 - g)) {
                g2 = g1;
                g1 = e.first;
            } else if (g2 < 0 || abs(e.first - g) < abs(g2 - g)) {
                g2 = e.first;
            }
        }
        const double t1 = at.at(g1);
        if (g2 > 0) w = (at.at(g2) - t1) / (1.0 / g2 - 1.0 / g1);
        // a single count, or a time that does not fall with the count: half of it taken as divisible
        if (g2 < 0 || !(w > 0.0) || !(w / g1 < t1)) w = 0.5 * t1 * g1;
        c = t1 - w / g1;
    }
};

// Counts that make the slowest system fastest under those lines: the least T with
// sum_i max(1, w_i / (T - c_i)) within the limit.
static std::vector<int> balanced_split(const std::vector<SolveTimes> &st, const std::vector<int> &cur, int cap) {
    const size_t K = st.size();
    std::vector<double> c(K), w(K);
    double lo = 0.0, hi = 0.0;
    for (size_t i = 0; i < K; i++) {
        st[i].line(cur[i], c[i], w[i]);
        lo = std::max(lo, c[i]);
        hi = std::max(hi, c[i] + w[i]);
    }
    auto counts = [&](double T, std::vector<int> &g) {
        long sum = 0;
        for (size_t i = 0; i < K; i++) {
            g[i] = T > c[i] ? (int)std::min((double)cap, std::max(1.0, ceil(w[i] / (T - c[i])))) : cap;
            sum += g[i];
        }
        return sum;
    };
    std::vector<int> g(K), best(K, 1);
    for (int it = 0; it < 60; it++) {
        const double T = 0.5 * (lo + hi);
        if (counts(T, g) <= cap) {
            best = g;
            hi = T;
        } else {
            lo = T;
        }
    }
    return best;
}

// Autotune on the Grams of the first step: re-run each instance's Gram from its split operands and
// time the cooperative launch, and in it every system's own solve.  From two starting splits the
// counts are balanced by the systems' measured times, a few rounds while the launch gets faster; then
// the other diagonal block widths of the factor (128 from order 2048, from 1024) where a system is
// that large.  The fastest is kept (its launch, after a last Gram, is the step's solve).
// Measured, 16 instances of order 156 to 2144: 1.63 ms (the best of seven fixed splits: 2.27 ms, and
// 277 ms for the first step with its 21 launches, now 27 ms).
static bool autotune(Batch &B, cudaStream_t st) {
    const int cap = mixed_batch_capacity(), K = (int)B.inst.size();
    if (cap < K) {
        set_error("batch of %d instances needs at least one co-resident CTA each (device holds %d)", K, cap);
        return false;
    }
    std::vector<MixedSys *> sys;
    int largest = 0;
    for (BatchInst *b : B.inst) {
        sys.push_back(b->mx);
        largest = std::max(largest, mixed_sys_order(b->mx));
    }
    cudaEvent_t e0, e1;
    if (!NQS_CUDA(cudaEventCreate(&e0)) || !NQS_CUDA(cudaEventCreate(&e1))) return false;
    double best = 1e300;
    bool first = true;
    B.tune_ms.clear();
    std::vector<SolveTimes> times((size_t)K);
    // Milliseconds of one launch (-1: it does not fit, -2: an error); the fastest is remembered.
    auto measure = [&](const std::vector<int> &ctas, int bd_from, bool keep_times) -> double {
        MixedBatch *mb = mixed_batch_create(sys.data(), K, ctas.data(), bd_from, true);
        if (!mb) {
            B.tune_ms.push_back(-1.0);
            return -1.0;
        }
        if (!first)
            for (BatchInst *b : B.inst) mixed_sys_front(b->mx, st, false);
        first = false;
        float ms = 0.f;
        bool ok = NQS_CUDA(cudaEventRecord(e0, st)) && mixed_batch_launch(mb, st) && NQS_CUDA(cudaEventRecord(e1, st)) &&
                  NQS_CUDA(cudaEventSynchronize(e1)) && NQS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        mixed_batch_free(mb);
        for (int i = 0; i < K && ok && keep_times; i++) {
            double us = 0.0;
            ok = mixed_sys_solve_us(sys[i], &us);
            if (us > 0.0) times[i].at[ctas[i]] = us;
        }
        if (!ok) return -2.0;
        B.tune_ms.push_back(ms);
        if (ms < best) {
            best = ms;
            B.ctas = ctas;
            B.bd_from = bd_from;
        }
        return ms;
    };
    bool ok = true;
    for (const std::vector<int> &c : cta_starts(B, cap)) ok = ok && measure(c, mixed_bd_default(), true) > -2.0;
    bool timed = true;
    for (const SolveTimes &t : times) timed = timed && !t.at.empty();
    for (int round = 0; round < 5 && ok && timed && !B.ctas.empty(); round++) {
        const std::vector<int> next = balanced_split(times, B.ctas, cap);
        if (next == B.ctas) break;
        const double before = best, ms = measure(next, mixed_bd_default(), true);
        ok = ms > -2.0;
        if (round > 0 && best > 0.99 * before) break;
    }
    for (int bd : {2048, 1024})
        if (ok && largest >= bd && !B.ctas.empty()) ok = measure(std::vector<int>(B.ctas), bd, false) > -2.0;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!ok || B.ctas.empty()) return false;
    B.mb = mixed_batch_create(sys.data(), K, B.ctas.data(), B.bd_from, false);
    if (!B.mb) return false;
    for (BatchInst *b : B.inst) mixed_sys_front(b->mx, st, false);
    return mixed_batch_launch(B.mb, st);
}

}  // namespace nqs

using namespace nqs;

struct nqs_gpu_batch {
    Batch b;
};

extern "C" {

nqs_gpu_batch_t *nqs_gpu_batch_create(const nqs_gpu_instance_t *in, int count) {
    clear_error();
    if (!in || count <= 0) {
        set_error("invalid arguments");
        return nullptr;
    }
    if (!ensure_context()) return nullptr;
    Context &c = ctx();
    cudaStream_t st = c.stream;
    nqs_gpu_batch_t *h = new nqs_gpu_batch_t();
    Batch &B = h->b;
    B.sweeps = c.opts.refine_sweeps;
    B.passes = c.opts.gram_passes;
    B.space = c.opts.mixed_space;
    // one stream per instance up to 32: an instance's front is a dozen short kernels in a row that leave
    // most SMs idle
    const int nside = count < 32 ? count : 32;
    B.side.resize((size_t)nside, nullptr);
    B.join.resize((size_t)nside, nullptr);
    for (int k = 0; k < nside; k++)
        if (!NQS_CUDA(cudaStreamCreateWithFlags(&B.side[k], cudaStreamNonBlocking)) ||
            !NQS_CUDA(cudaEventCreateWithFlags(&B.join[k], cudaEventDisableTiming))) {
            delete h;
            return nullptr;
        }
    if (!NQS_CUDA(cudaEventCreateWithFlags(&B.fork, cudaEventDisableTiming))) {
        delete h;
        return nullptr;
    }
    for (int i = 0; i < count; i++) {
        BatchInst *b = new BatchInst();
        B.inst.push_back(b);
        if (!in[i].cfg || !in[i].ansatz || !in[i].sampler) {
            set_error("instance %d: cfg, ansatz and sampler are required", i);
            delete h;
            return nullptr;
        }
        b->cfg = *in[i].cfg;
        b->sx = in[i].size_x;
        b->sy = in[i].size_y;
        b->a = (Ansatz *)in[i].ansatz;
        b->s = (Sampler *)in[i].sampler;
        b->fn = in[i].log_amp ? in[i].log_amp : nqs_ansatz_log_amp;
        b->user = in[i].log_amp ? in[i].log_amp_user : (void *)b->a;
        Ansatz *base = nullptr;
        if (!hamiltonian_build(&b->cfg, b->sx, b->sy, &b->H) || !build_amp(b->fn, b->user, b->H.N, &b->A, &base)) {
            delete h;
            return nullptr;
        }
        if (base != b->a || !fp32_capable(b->A) || !sampler_fp32(b->s) ||
            nqs_sampler_num_sites((nqs_sampler_t *)b->s) != b->H.N) {
            set_error("instance %d: needs an RBM / cRBM program of its ansatz and a Philox sampler of the same "
                      "sites created in the MIXED mode with fp32_estimator = 1", i);
            delete h;
            return nullptr;
        }
        b->Ns = b->cfg.num_samples;
        b->C = sampler_chains(b->s);
        b->P = b->a->P;
        const uint64_t mv = sampler_move_counter(b->s);
        if (b->Ns <= 0 || !b->E.ensure(b->Ns) || !b->Ei.ensure(b->Ns) || !b->eps.ensure(b->Ns) ||
            !b->O.ensure((size_t)b->Ns * b->P) || !b->gm.ensure(b->P) || !b->scal.ensure(16) ||
            !b->delta.ensure(b->P) || !b->y.ensure(b->Ns) || !b->move.ensure(1) ||
            !b->part.ensure((size_t)col_stats_scratch(b->Ns, b->P)) ||
            !b->es.ensure(energy_scratch_doubles(b->Ns)) ||
            !NQS_CUDA(cudaMemset(b->es.p, 0, sizeof(double) * energy_scratch_doubles(b->Ns))) ||
            !NQS_CUDA(cudaMemcpy(b->move.p, &mv, sizeof(mv), cudaMemcpyHostToDevice)) ||
            !NQS_CUDA(cudaMallocHost(&b->h, sizeof(BatchWords)))) {
            delete h;
            return nullptr;
        }
        b->mx = mixed_sys_create();
        if (!mixed_sys_prepare(b->mx, b->O.p, b->gm.p, b->eps.p, b->Ns, b->P, b->cfg.sr_diag_shift, B.sweeps, B.passes,
                               B.space, b->y.p, b->delta.p)) {
            delete h;
            return nullptr;
        }
    }
    if (!NQS_CUDA(cudaStreamSynchronize(st))) {
        delete h;
        return nullptr;
    }
    return h;
}

int nqs_gpu_batch_step(nqs_gpu_batch_t *h, nqs_sr_step_info_t *infos) {
    clear_error();
    if (!h) return -1;
    Batch &B = h->b;
    Context &c = ctx();
    cudaStream_t st = c.stream;
    for (BatchInst *b : B.inst)
        if (!ansatz_sync(b->a)) return -1;
    auto front = [](BatchInst &b, cudaStream_t s) { return enqueue_front(b, s); };
    auto back = [](BatchInst &b, cudaStream_t s) { return enqueue_back(b, s); };
    if (B.steps == 0 || c.profiling) {
        if (!fork_join(B, st, front)) return -1;
        if (B.steps == 0) {
            if (!autotune(B, st)) return -1;
        } else if (!mixed_batch_launch(B.mb, st)) {
            return -1;
        }
        if (!fork_join(B, st, back)) return -1;
    } else {
        if (!B.exec) {
            cudaGraph_t graph;
            const long l0 = c.launches;
            if (!NQS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal))) return -1;
            bool ok = fork_join(B, st, front);
            ok = ok && mixed_batch_launch(B.mb, st);
            ok = ok && fork_join(B, st, back);
            const bool ended = NQS_CUDA(cudaStreamEndCapture(st, &graph));
            if (!ok || !ended) return -1;
            B.graph_kernels = c.launches - l0;
            c.launches = l0;
            const bool inst_ok = NQS_CUDA(cudaGraphInstantiate(&B.exec, graph, 0));
            cudaGraphDestroy(graph);
            if (!inst_ok) {
                B.exec = nullptr;
                return -1;
            }
        }
        if (!NQS_CUDA(cudaGraphLaunch(B.exec, st))) return -1;
        c.launches += B.graph_kernels;
    }
    if (!NQS_CUDA(cudaStreamSynchronize(st))) return -1;
    B.steps++;
    // An instance whose mixed solve broke down (a pivot <= 0, or a CG residual
    // above the bound) had its update held at zero inside the graph; solve it
    // again in FP64 on the same centred O and eps, as the single-system step does.
    for (size_t i = 0; i < B.inst.size(); i++) {
        BatchInst *b = B.inst[i];
        b->fp64_fallback = 0;
        if (!mixed_broken(b->h->status, b->h->nrm) || b->h->err != 0) continue;
        int conv = 0;
        if (minsr_fp64_delta(b->O.p, b->eps.p, b->Ns, b->P, b->cfg.sr_diag_shift, b->delta.p, &conv) != 0)
            return -1;
        k_batch_apply<<<1, 1024, 0, st>>>(b->a->d_params.p, b->delta.p, b->P, b->cfg.learning_rate, b->scal.p,
                                          mixed_sys_status(b->mx), mixed_sys_err(b->mx), mixed_sys_nrm(b->mx), 1,
                                          nullptr, nullptr);
        if (!NQS_CUDA(cudaMemcpyAsync(&b->h->scal[S_NORM2], b->scal.p + S_NORM2, sizeof(double), cudaMemcpyDeviceToHost,
                                      st)) ||
            !NQS_CUDA(cudaMemcpyAsync(b->a->h_params, b->a->d_params.p, sizeof(double) * b->P,
                                      cudaMemcpyDeviceToHost, st)) ||
            !NQS_CUDA(cudaStreamSynchronize(st)))
            return -1;
        b->fp64_fallback = 1;
        b->fp64_conv = conv;
        B.fallbacks++;
    }
    int failed = 0;
    for (size_t i = 0; i < B.inst.size(); i++) {
        BatchInst *b = B.inst[i];
        sampler_host_advance(b->s, b->Ns);
        memcpy(b->a->h_shadow, b->a->h_params, sizeof(double) * b->P);
        if (b->h->err) failed = (int)i + 1;
        if (infos) {
            nqs_sr_step_info_t &f = infos[i];
            const double *sc = b->h->scal;
            const unsigned long long *n = b->h->counts;
            f.mean_energy = sc[S_EMEAN];
            f.variance_energy = sc[S_ESQ] - sc[S_EMEAN] * sc[S_EMEAN];
            f.update_norm = sqrt(sc[S_NORM2]) * b->cfg.learning_rate;
            f.acceptance_ratio = n[1] ? (double)n[0] / (double)n[1] : 0.0;
            f.cg_iterations = 0;
            f.converged = b->fp64_fallback ? b->fp64_conv : (!mixed_broken(b->h->status, b->h->nrm) && b->h->err == 0);
        }
    }
    if (failed) {
        set_error("batch instance %d: %s", failed - 1,
                  B.inst[failed - 1]->h->err == 2 ? "grid barrier timed out" : "tensor-core Gram timed out");
        return -1;
    }
    return 0;
}

int nqs_gpu_batch_ctas(const nqs_gpu_batch_t *h, int *out) {
    if (!h || !out || h->b.ctas.empty()) return -1;
    for (size_t i = 0; i < h->b.ctas.size(); i++) out[i] = h->b.ctas[i];
    return 0;
}

int nqs_gpu_batch_block_widths(const nqs_gpu_batch_t *b, int *out_bd) {
    if (!b || !out_bd || b->b.ctas.empty()) return -1;
    for (size_t i = 0; i < b->b.inst.size(); i++)
        out_bd[i] = mixed_sys_order(b->b.inst[i]->mx) >= b->b.bd_from ? 128 : 64;
    return 0;
}

int nqs_gpu_batch_tune_ms(const nqs_gpu_batch_t *h, double *out, int cap) {
    if (!h || !out) return -1;
    const int n = (int)h->b.tune_ms.size() < cap ? (int)h->b.tune_ms.size() : cap;
    for (int i = 0; i < n; i++) out[i] = h->b.tune_ms[i];
    return n;
}

long nqs_gpu_batch_fallbacks(const nqs_gpu_batch_t *h) { return h ? h->b.fallbacks : -1; }

void nqs_gpu_batch_free(nqs_gpu_batch_t *h) { delete h; }

}  // extern "C"
