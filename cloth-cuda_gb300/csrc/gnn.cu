// Learned warm start: host side and C ABI (no counterpart in the reference).
// The kernels live in gnn_kernels.cuh; this file owns the parameters, the
// activation buffers, the training step and the binding to a solver.
#include "gnn_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

using namespace pdg;
using namespace pdg::gnn;

#define GK(call)                                                                                \
    do {                                                                                        \
        const cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                                  \
            return set_error(e_ == cudaErrorMemoryAllocation ? PDG_ERR_ALLOC : PDG_ERR_CUDA,    \
                             "warm start: %s: %s", #call, cudaGetErrorString(e_));              \
    } while (0)

struct pdg_warmstart {
    Layout lay;
    long long t = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    DevBuf<float> p, g, m, v, bdp;
    DevBuf<float> part;   // per-block partial weight gradients (summed in a fixed order), from the first backward pass on
    DevBuf<bf16> wbuf;
    Bf16Weights W{};
    // graph and activations
    int N = 0, E = 0;
    DevBuf<int> ptr, adj, rev;
    DevBuf<float> rest, deg_inv;
    DevBuf<float4> ef, stat, Xn, Vn, Dn;
    DevBuf<float4> Xd;    // the deep solve's x* in the trajectory's vertex order
    DevBuf<float> ew;     // per directed edge: weight of the energy-norm term of the loss
    DevBuf<uint2> mask[L];   // per edge: signs of the message's channels
    DevBuf<bf16> xin, cat[L], pq[L], uo[L], hfin;
    DevBuf<float> out, target, freew, dout, dh, dtmp, da, dpq;
    DevBuf<double> loss;
    DevBuf<int> bad;      // the graph failed its checks
    float smooth = 0.f;   // weight of the neighbour-difference term of the loss
    int energy = 0;       // 1: that term weighted by the PD system's stiffness per edge
    // sweeps each start runs before the judge compares them; 1: the starts'
    // own residuals, which each chain's first sweep evaluates
    int judge = 1;
    pdg_solver* solver = nullptr;
    ~pdg_warmstart()
    {
        if (own_stream && stream) cudaStreamDestroy(stream);
    }
};

namespace {

inline int nb(long long n, int b) { return (int)((n + b - 1) / b); }

constexpr int kWgradBlocks = 304;        // at most, blocks of a weight-gradient reduction
constexpr int kMsgBwdBlocks = 3 * 152;   // at most, blocks of the message backward (those resident at once)

int refresh_bf16(pdg_warmstart* w, cudaStream_t st)
{
    k_copies<<<nb(w->lay.total, 256), 256, 0, st>>>(w->lay.total, w->p.p, w->lay, w->W, w->bdp.p);
    GK(cudaGetLastError());
    return PDG_OK;
}

int alloc_params(pdg_warmstart* w)
{
    const int n = w->lay.total;
    GK(w->p.alloc(n)); GK(w->g.alloc(n)); GK(w->m.alloc(n)); GK(w->v.alloc(n)); GK(w->bdp.alloc(16));
    // bf16 copies: We 64x16, per layer AB 128x64, ABt 64x128, U 64x128, Ut 128x64, Wd 16x64, Wdt 64x16
    const size_t sizes[] = {(size_t)H * NFP, 2u * H * H, 2u * H * H, 2u * H * H, 2u * H * H, 16u * H, (size_t)H * 16};
    size_t total = sizes[0] + L * (sizes[1] + sizes[2] + sizes[3] + sizes[4]) + sizes[5] + sizes[6];
    GK(w->wbuf.alloc(total));
    GK(cudaMemsetAsync(w->wbuf.p, 0, sizeof(bf16) * total, w->stream));
    GK(cudaMemsetAsync(w->bdp.p, 0, sizeof(float) * 16, w->stream));
    bf16* q = w->wbuf.p;
    w->W.We = q; q += sizes[0];
    for (int l = 0; l < L; ++l) {
        w->W.AB[l] = q; q += sizes[1];
        w->W.ABt[l] = q; q += sizes[2];
        w->W.U[l] = q; q += sizes[3];
        w->W.Ut[l] = q; q += sizes[4];
    }
    w->W.Wd = q; q += sizes[5];
    w->W.Wdt = q;
    GK(cudaMemsetAsync(w->g.p, 0, sizeof(float) * n, w->stream));
    GK(cudaMemsetAsync(w->m.p, 0, sizeof(float) * n, w->stream));
    GK(cudaMemsetAsync(w->v.p, 0, sizeof(float) * n, w->stream));
    return PDG_OK;
}

// Buffers for N nodes and E directed edges.  They are kept for the network's
// lifetime and only grow: a call of pdg_warmstart_eval allocated and freed
// about 35 of them, more than half of its time on a 97x97 graph.
int alloc_graph(pdg_warmstart* w, int N, int E)
{
    w->N = N; w->E = E;
    GK(w->ptr.reserve(N + 1)); GK(w->adj.reserve(E)); GK(w->rev.reserve(E));
    GK(w->rest.reserve(E)); GK(w->deg_inv.reserve(N)); GK(w->ef.reserve(E)); GK(w->stat.reserve(N));
    GK(w->Xn.reserve(N)); GK(w->Vn.reserve(N)); GK(w->Dn.reserve(N)); GK(w->ew.reserve(E));
    GK(w->xin.reserve((size_t)N * NFP));
    for (int l = 0; l < L; ++l) {
        GK(w->cat[l].reserve((size_t)N * 2 * H)); GK(w->pq[l].reserve((size_t)N * 2 * H)); GK(w->uo[l].reserve((size_t)N * H));
        GK(w->mask[l].reserve(E));
    }
    GK(w->hfin.reserve((size_t)N * H));
    GK(w->out.reserve((size_t)N * 16)); GK(w->target.reserve((size_t)N * 3)); GK(w->freew.reserve(N));
    GK(w->dout.reserve((size_t)N * 16)); GK(w->dh.reserve((size_t)N * H)); GK(w->dtmp.reserve((size_t)N * H));
    GK(w->da.reserve((size_t)N * H)); GK(w->dpq.reserve((size_t)N * 2 * H)); GK(w->loss.reserve(1)); GK(w->bad.reserve(1));
    return PDG_OK;
}

// The network on the current features for training: every activation the
// backward pass needs is kept (h and a per layer, P and Q, the update's ReLU
// output, the last h and the decoder output).  Inference runs the fused
// kernels instead (warm_infer_enqueue), with bitwise the same start offsets.
int forward(pdg_warmstart* w, cudaStream_t st)
{
    const int N = w->N;
    const Layout& y = w->lay;
    const float* p = w->p.p;
    // (the backward pass's; here it parts no two kernels)
    GK(cudaMemsetAsync(w->loss.p, 0, sizeof(double), st));
    gemm<bf16, NFP, H, EPI_RELU | EPI_STORE1>(st, w->xin.p, NFP, N, w->W.We, p + y.be, nullptr, 0, w->cat[0].p, 2 * H,
                                              nullptr, 0, nullptr, 0);
    for (int l = 0; l < L; ++l) {
        gemm<bf16, H, 2 * H, EPI_STORE1>(st, w->cat[l].p, 2 * H, N, w->W.AB[l], nullptr, nullptr, 0, w->pq[l].p, 2 * H,
                                         nullptr, 0, nullptr, 0);
        messages<true>(st, N, w->ptr.p, w->adj.p, w->ef.p, w->deg_inv.p, w->pq[l].p, p + y.C[l], p + y.c[l], w->cat[l].p,
                       w->mask[l].p);
        bf16* next = l + 1 < L ? w->cat[l + 1].p : w->hfin.p;
        const int ldn = l + 1 < L ? 2 * H : H;
        // h <- h + relu(U [h; a] + u): the residual h is the A operand's
        // first H columns
        gemm<bf16, 2 * H, H, EPI_RELU | EPI_STORE1 | EPI_RESIDA>(st, w->cat[l].p, 2 * H, N, w->W.U[l], p + y.u[l],
                                                                 nullptr, 0, w->uo[l].p, H, next, ldn, nullptr, 0);
    }
    gemm<bf16, H, 16, EPI_STOREF>(st, w->hfin.p, H, N, w->W.Wd, w->bdp.p, nullptr, 0, nullptr, 0, nullptr, 0,
                                  w->out.p, 16);
    GK(cudaGetLastError());
    return PDG_OK;
}

int wgrad_grid(int M) { return std::max(1, std::min(kWgradBlocks, nb(M, kWgradRows))); }
int msg_bwd_grid(int N) { return std::max(1, std::min(kMsgBwdBlocks, nb(N, 16))); }

// Floats of the partial sums of every gradient over N nodes (they are added up
// in one launch): 40 MB at most, which a network that only infers never needs.
size_t part_floats(int N)
{
    return (size_t)wgrad_grid(N) * ((NO * H + NO) + (H * NF + H) + L * ((2 * H * H + H) + (2 * H * H + 2 * H))) +
           (size_t)msg_bwd_grid(N) * L * H * (EF + 1);
}

// The partial sums of a backward pass: wgrad and the message backward append
// a segment each, `run` adds all of them up.
struct GradSums {
    SumTable t{};
    float* free_;
    int n = 0;
    explicit GradSums(float* part) : free_(part) {}
    float* add(int nblocks, int nw, int nbias, float* dW, float* db)
    {
        float* q = free_;
        t.part[n] = q; t.nblocks[n] = nblocks; t.nw[n] = nw; t.nbias[n] = nbias; t.dW[n] = dW; t.db[n] = db;
        t.first[n + 1] = t.first[n] + nb(nw + nbias, 32);
        free_ += (size_t)nblocks * (nw + nbias);
        ++n;
        return q;
    }
    void run(cudaStream_t st) { launch_after(k_sum_parts, t.first[n], 256, 0, st, t); }
};

// Partial sums of dW (nout x K) and db (nout, may be null) of dY^T X over M
// rows; ref: dY counts as zero where ref is not positive.
template <int NP, int KP, bool MASK>
void wgrad(GradSums& gs, const float* dY, int ldy, int nout, const bf16* ref, int ldr, const bf16* X, int ldx, int K,
           int M, float* dW, float* db, cudaStream_t st)
{
    const int gw = wgrad_grid(M);
    float* part = gs.add(gw, nout * K, nout, dW, db);
    launch_after(k_wgrad<NP, KP, MASK>, gw, 256, 0, st, dY, ldy, nout, ref, ldr, X, ldx, K, M, part);
}

// gradients of the loss w.r.t. all parameters into w->g; loss accumulated into
// w->loss (cleared by forward); ew: per-edge weights of the smoothness term (null: 1).  The ReLU
// masks are applied where their operand is read and the residual path is added
// where its partner is written.  With both in kernels of their own and one
// launch of sums per gradient a training step on 16 cloths took 2,220 us (now
// 2,108), the gradients of a 97x97 graph 452 us (385).
int backward(pdg_warmstart* w, float inv_cnt, const float* ew, cudaStream_t st)
{
    const int N = w->N;
    const Layout& y = w->lay;
    float* g = w->g.p;
    GK(w->part.reserve(part_floats(N)));   // (grows only with the graph, whose upload waits for earlier passes)
    GradSums gs(w->part.p);
    launch_after(k_loss, nb(N, 256), 256, 0, st, N, w->out.p, w->target.p, w->freew.p, w->ptr.p, w->adj.p, ew, w->smooth,
                                       inv_cnt, w->dout.p, w->loss.p);
    wgrad<16, H, false>(gs, w->dout.p, 16, NO, nullptr, 0, w->hfin.p, H, H, N, g + y.Wd, g + y.bd, st);
    float *dh = w->dh.p, *dn = w->dtmp.p;   // d loss / d h of layer l, of layer l - 1
    gemm<float, 16, H, EPI_STOREF>(st, w->dout.p, 16, N, w->W.Wdt, nullptr, nullptr, 0, nullptr, 0, nullptr, 0, dh, H);
    for (int l = L - 1; l >= 0; --l) {
        wgrad<H, 2 * H, true>(gs, dh, H, H, w->uo[l].p, H, w->cat[l].p, 2 * H, 2 * H, N, g + y.U[l], g + y.u[l], st);
        gemm<float, H, 2 * H, EPI_MASKA | EPI_SPLIT>(st, dh, H, N, w->W.Ut[l], nullptr, w->uo[l].p, H, nullptr, 0,
                                                     nullptr, 0, dn, H, w->da.p, H, w->deg_inv.p);
        const int gm = msg_bwd_grid(N);
        float* part = gs.add(gm, H * EF, H, g + y.C[l], g + y.c[l]);
        launch_after(k_msg_bwd, gm, 256, 0, st, N, w->ptr.p, w->adj.p, w->rev.p, w->ef.p, w->mask[l].p, w->da.p, w->dpq.p, part);
        wgrad<2 * H, H, false>(gs, w->dpq.p, 2 * H, 2 * H, nullptr, 0, w->cat[l].p, 2 * H, H, N, g + y.A[l], nullptr, st);
        gemm<float, 2 * H, H, EPI_ACCF>(st, w->dpq.p, 2 * H, N, w->W.ABt[l], nullptr, nullptr, 0, nullptr, 0, nullptr, 0,
                                        dn, H);
        std::swap(dh, dn);
    }
    wgrad<H, NFP, true>(gs, dh, H, H, w->cat[0].p, 2 * H, w->xin.p, NFP, NF, N, g + y.We, g + y.be, st);
    gs.run(st);
    GK(cudaGetLastError());
    return PDG_OK;
}

int adam_step(pdg_warmstart* w, float lr, cudaStream_t st)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    w->t += 1;
    const float bc1 = 1.f - (float)std::pow((double)b1, (double)w->t);
    const float bc2 = 1.f - (float)std::pow((double)b2, (double)w->t);
    launch_after(k_adam, nb(w->lay.total, 256), 256, 0, st, w->lay.total, w->p.p, w->g.p, w->m.p, w->v.p, lr, b1, b2, eps, bc1,
                                                  bc2, w->lay, w->W, w->bdp.p);
    GK(cudaGetLastError());
    return PDG_OK;
}

// Room for the graph, and its arrays on `st`: the reverse-edge index and the
// inverse degrees are formed on the device, where graph_ok finds whether the
// adjacency was symmetric.
int upload_graph(pdg_warmstart* w, int N, const int* ptr, int E, const int* adj, cudaStream_t st)
{
    // work that still reads the buffers
    GK(cudaStreamSynchronize(w->stream));
    if (w->solver) GK(cudaStreamSynchronize(w->solver->stream));
    const int rc = alloc_graph(w, N, E);
    if (rc) return rc;
    GK(cudaMemcpyAsync(w->ptr.p, ptr, sizeof(int) * ((size_t)N + 1), cudaMemcpyHostToDevice, st));
    if (E) GK(cudaMemcpyAsync(w->adj.p, adj, sizeof(int) * (size_t)E, cudaMemcpyHostToDevice, st));
    GK(cudaMemsetAsync(w->bad.p, 0, sizeof(int), st));
    k_graph<<<nb(N, 256), 256, 0, st>>>(N, E, w->ptr.p, w->adj.p, w->rev.p, w->deg_inv.p, w->bad.p);
    GK(cudaGetLastError());
    return PDG_OK;
}

// Waits for upload_graph's checks; nothing may read the graph before.
// backward_lists: some list ends before it begins (caller graphs; with one of
// those an entry may belong to several lists, or the graph may also be bad).
int graph_ok(pdg_warmstart* w, cudaStream_t st, bool* backward_lists = nullptr)
{
    int bad = 0;
    GK(cudaMemcpyAsync(&bad, w->bad.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    GK(cudaStreamSynchronize(st));
    if (backward_lists) *backward_lists = bad == 2;
    return bad && !(backward_lists && bad == 2) ? set_error(PDG_ERR_ARG, "warm start: adjacency is not symmetric") : PDG_OK;
}

// The same graph with every list of its own, one after another: ptr, and of
// each entry its place in the caller's arrays.  False where a list leaves them.
bool plain_lists(int N, const int* ptr, int E, std::vector<int>& p, std::vector<int>& from)
{
    p.assign(1, 0);
    for (int i = 0; i < N; ++i) {
        if (ptr[i] < 0 || ptr[i] > E || ptr[i + 1] < 0 || ptr[i + 1] > E) return false;
        for (int e = ptr[i]; e < ptr[i + 1]; ++e) from.push_back(e);
        if (from.size() > 0x7fffffffu) return false;
        p.push_back((int)from.size());
    }
    return true;
}

}  // namespace

// ---- solver-side hooks (declared in pdg_solver.h) -------------------------
namespace pdg {

int warm_infer_enqueue(pdg_warmstart* w, pdg_solver* s)
{
    cudaStream_t st = s->stream;
    const int N = w->N;
    k_node_feat<<<nb(N, 256), 256, 0, st>>>(N, s->X.p, s->V.p, s->Y.p, s->aux.p, w->stat.p, s->vcloth.p, s->cinfo.p,
                                            s->dprev.p, w->xin.p);
    launch_after(k_edge_feat, nb(N, 256), 256, 0, st, N, w->ptr.p, w->adj.p, w->rest.p, s->Y.p, w->ef.p);
    // encoder + layer 0's P, Q; per layer the messages, then the update fused
    // with the next layer's P, Q or, after the last layer, with the decoder
    // and the start offsets
    const Layout& y = w->lay;
    const float* p = w->p.p;
    fused<FUSE_ENC_PQ>(st, w->xin.p, NFP, N, w->W.We, p + y.be, w->W.AB[0], nullptr, w->cat[0].p, 2 * H, w->pq[0].p,
                       nullptr, nullptr, nullptr);
    for (int l = 0; l < L; ++l) {
        messages<false>(st, N, w->ptr.p, w->adj.p, w->ef.p, w->deg_inv.p, w->pq[l].p, p + y.C[l], p + y.c[l], w->cat[l].p,
                        nullptr);
        if (l + 1 < L)
            fused<FUSE_UPD_PQ>(st, w->cat[l].p, 2 * H, N, w->W.U[l], p + y.u[l], w->W.AB[l + 1], nullptr,
                               w->cat[l + 1].p, 2 * H, w->pq[l + 1].p, nullptr, nullptr, nullptr);
        else
            fused<FUSE_UPD_OUT>(st, w->cat[l].p, 2 * H, N, w->W.U[l], p + y.u[l], w->W.Wd, w->bdp.p, nullptr, 0,
                                nullptr, s->A.p, s->dprev.p, s->warm.p);
    }
    GK(cudaGetLastError());
    return PDG_OK;
}

// launches of one warm_infer_enqueue: features (2), encoder, per layer the
// messages and the fused update
int warm_kernel_count() { return 3 + 2 * L; }

void warm_detach(pdg_warmstart* w, const pdg_solver* s)
{
    if (w && w->solver == s) w->solver = nullptr;
}

int warm_judge_sweeps(const pdg_warmstart* w) { return w ? w->judge : 0; }

}  // namespace pdg

extern "C" {

int pdg_warmstart_create(unsigned long long seed, pdg_warmstart** out)
{
    if (!out) return set_error(PDG_ERR_ARG, "pdg_warmstart_create: null output");
    std::unique_ptr<pdg_warmstart> w(new pdg_warmstart);
    GK(cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking));
    w->own_stream = true;
    int rc = alloc_params(w.get());
    if (rc) return rc;
    // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights, zero biases; the
    // decoder starts at zero, so an untrained network predicts no change of
    // the offset: the previous frame's offset where it is valid, else y
    const Layout& y = w->lay;
    std::vector<float> h(y.total, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int rows, int cols, float gain) {
        std::uniform_real_distribution<float> U(-gain / std::sqrt((float)cols), gain / std::sqrt((float)cols));
        for (int i = 0; i < rows * cols; ++i) h[off + i] = U(rng);
    };
    fill(y.We, H, NF, 1.f);
    for (int l = 0; l < L; ++l) {
        fill(y.A[l], H, H, 1.f); fill(y.B[l], H, H, 1.f); fill(y.C[l], H, EF, 1.f); fill(y.U[l], H, 2 * H, 1.f);
    }
    // (decoder Wd, bd stay zero)
    GK(cudaMemcpyAsync(w->p.p, h.data(), sizeof(float) * y.total, cudaMemcpyHostToDevice, w->stream));
    rc = refresh_bf16(w.get(), w->stream);
    if (rc) return rc;
    GK(cudaStreamSynchronize(w->stream));
    *out = w.release();
    return PDG_OK;
}

int pdg_warmstart_param_count(const pdg_warmstart* w, int* n)
{
    if (!w || !n) return set_error(PDG_ERR_ARG, "null argument");
    *n = w->lay.total;
    return PDG_OK;
}

int pdg_warmstart_get_params(pdg_warmstart* w, float* host)
{
    if (!w || !host) return set_error(PDG_ERR_ARG, "null argument");
    GK(cudaStreamSynchronize(w->stream));
    if (w->solver) GK(cudaStreamSynchronize(w->solver->stream));
    GK(cudaMemcpyAsync(host, w->p.p, sizeof(float) * w->lay.total, cudaMemcpyDeviceToHost, w->stream));
    GK(cudaStreamSynchronize(w->stream));
    return PDG_OK;
}

int pdg_warmstart_set_params(pdg_warmstart* w, const float* host)
{
    if (!w || !host) return set_error(PDG_ERR_ARG, "null argument");
    for (int i = 0; i < w->lay.total; ++i)
        if (!std::isfinite(host[i])) return set_error(PDG_ERR_ARG, "non-finite parameter %d", i);
    GK(cudaStreamSynchronize(w->stream));
    if (w->solver) GK(cudaStreamSynchronize(w->solver->stream));
    GK(cudaMemcpyAsync(w->p.p, host, sizeof(float) * w->lay.total, cudaMemcpyHostToDevice, w->stream));
    GK(cudaMemsetAsync(w->m.p, 0, sizeof(float) * w->lay.total, w->stream));
    GK(cudaMemsetAsync(w->v.p, 0, sizeof(float) * w->lay.total, w->stream));
    w->t = 0;
    const int rc = refresh_bf16(w, w->stream);
    if (rc) return rc;
    GK(cudaStreamSynchronize(w->stream));
    return PDG_OK;
}

int pdg_warmstart_eval(pdg_warmstart* w, int N, const float* x, const int* ptr, const int* adj, const float* ef,
                       const float* target, const float* freew, const float* ew, float* out, float* loss,
                       float* grads)
{
    if (!w || N <= 0 || !x || !ptr || !target || !freew) return set_error(PDG_ERR_ARG, "pdg_warmstart_eval: bad arguments");
    if (w->solver) return set_error(PDG_ERR_STATE, "pdg_warmstart_eval: the network is attached to a solver");
    const int E = ptr[N];
    if (E < 0 || (E > 0 && (!adj || !ef))) return set_error(PDG_ERR_ARG, "pdg_warmstart_eval: bad adjacency");
    cudaStream_t st = w->stream;
    int rc = upload_graph(w, N, ptr, E, adj, st);
    if (rc) return rc;
    // features to bf16 on the device (staged where the backward pass later
    // keeps dh)
    GK(cudaMemcpyAsync(w->dh.p, x, sizeof(float) * NF * (size_t)N, cudaMemcpyHostToDevice, st));
    k_pack_feat<<<nb(N, 256), 256, 0, st>>>(N, w->dh.p, w->xin.p);
    if (E) GK(cudaMemcpyAsync(w->ef.p, ef, sizeof(float4) * E, cudaMemcpyHostToDevice, st));
    GK(cudaMemcpyAsync(w->target.p, target, sizeof(float) * 3 * N, cudaMemcpyHostToDevice, st));
    GK(cudaMemcpyAsync(w->freew.p, freew, sizeof(float) * N, cudaMemcpyHostToDevice, st));
    if (ew && E) GK(cudaMemcpyAsync(w->ew.p, ew, sizeof(float) * E, cudaMemcpyHostToDevice, st));
    bool backward_lists = false;
    rc = graph_ok(w, st, &backward_lists);
    if (rc) return rc;
    if (backward_lists) {   // the kernels keep one sign mask per entry: no entry may belong to two lists
        try {
            std::vector<int> p, from;
            if (!plain_lists(N, ptr, E, p, from)) return set_error(PDG_ERR_ARG, "pdg_warmstart_eval: bad adjacency");
            std::vector<int> a(from.size());
            std::vector<float4> f(from.size());
            std::vector<float> q(ew ? from.size() : 0);
            for (size_t i = 0; i < from.size(); ++i) {
                a[i] = adj[from[i]];
                std::memcpy(&f[i], ef + 4 * (size_t)from[i], sizeof(float4));
                if (ew) q[i] = ew[from[i]];
            }
            return pdg_warmstart_eval(w, N, x, p.data(), a.data(), f.empty() ? nullptr : &f[0].x, target, freew,
                                      q.empty() ? nullptr : q.data(), out, loss, grads);
        } catch (const std::bad_alloc&) {
            return set_error(PDG_ERR_ALLOC, "host allocation failed");
        }
    }
    double cnt = 0.0;
    for (int i = 0; i < N; ++i) cnt += freew[i] > 0.f ? 3.0 : 0.0;
    rc = forward(w, st);
    if (rc) return rc;
    rc = backward(w, (float)(1.0 / std::max(cnt, 1.0)), (ew && E) ? w->ew.p : nullptr, st);
    if (rc) return rc;
    double l = 0.0;
    if (out) {   // N x 3 of the padded outputs, through a buffer the backward pass is done with
        k_pack_out<<<nb(N, 256), 256, 0, st>>>(N, w->out.p, w->dtmp.p);
        GK(cudaMemcpyAsync(out, w->dtmp.p, sizeof(float) * NO * (size_t)N, cudaMemcpyDeviceToHost, st));
    }
    GK(cudaMemcpyAsync(&l, w->loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    if (grads) GK(cudaMemcpyAsync(grads, w->g.p, sizeof(float) * w->lay.total, cudaMemcpyDeviceToHost, st));
    GK(cudaStreamSynchronize(st));
    if (loss) *loss = (float)l;
    return PDG_OK;
}

int pdg_warmstart_adam_step(pdg_warmstart* w, float lr)
{
    if (!w || !(lr > 0.f)) return set_error(PDG_ERR_ARG, "pdg_warmstart_adam_step: bad arguments");
    cudaStream_t st = w->solver ? w->solver->stream : w->stream;
    const int rc = adam_step(w, lr, st);
    if (rc) return rc;
    GK(cudaStreamSynchronize(st));
    return PDG_OK;
}

int pdg_warmstart_attach(pdg_warmstart* w, pdg_solver* s)
{
    if (!w || !s) return set_error(PDG_ERR_ARG, "pdg_warmstart_attach: null argument");
    if (s->kernel != PDG_KERNEL_GRAPH && s->kernel != PDG_KERNEL_STREAM)
        return set_error(PDG_ERR_STATE, "pdg_warmstart_attach: the solver must use the per-sweep (graph) kernels");
    // a network serves one solver and a solver has one network: either's former
    // partner lets go (its frames then start from the inertial prediction)
    if (w->solver && w->solver != s) {
        pdg_solver* old = w->solver;
        GK(cudaStreamSynchronize(old->stream));
        old->ws = nullptr;
        if (old->graph) { cudaGraphExecDestroy(old->graph); old->graph = nullptr; }
        w->solver = nullptr;
    }
    if (s->ws && s->ws != w) {
        GK(cudaStreamSynchronize(s->stream));
        warm_detach(s->ws, s);
        s->ws = nullptr;
    }
    const HostLayout& Lh = s->L;
    const int N = Lh.ntot;
    // mesh adjacency in the solver's (reordered) numbering, both directions
    std::vector<std::vector<std::pair<int, float>>> nbr(N);
    std::vector<float4> stat(N);
    std::vector<int> iperm(N);
    for (int g = 0; g < N; ++g) iperm[Lh.perm_global[g]] = g;   // batch caller index -> reordered
    int vbase = 0;
    for (const auto& c : s->cloths) {
        const Topology& t = *c.topo;
        const size_t nE = t.edges.size() / 4;
        for (size_t e = 0; e < nE; ++e) {
            const int a = iperm[vbase + t.edges[4 * e]], b = iperm[vbase + t.edges[4 * e + 1]];
            const float r = std::max(t.rest_len[e], 1e-12f);
            nbr[a].push_back({b, r});
            nbr[b].push_back({a, r});
        }
        double ks = 0.0, kb = 0.0;
        for (float k : c.cons.k_stretch) ks += k;
        for (float k : c.cons.bend_k) kb += k;
        ks = c.cons.k_stretch.empty() ? 1.0 : ks / c.cons.k_stretch.size();
        kb = c.cons.bend_k.empty() ? 1e-3 : kb / c.cons.bend_k.size();
        for (int i = 0; i < c.mesh->N; ++i) {
            const int gidx = iperm[vbase + i];
            const float m = std::max(c.mesh->mass[i], 1e-12f);
            stat[gidx] = make_float4((std::log(m) + 11.f) / 2.f, (float)((std::log(std::max(ks, 1e-6)) - 6.9) / 1.2),
                                     (float)((std::log(std::max(kb, 1e-9)) + 4.6) / 1.2), 0.f);
        }
        vbase += c.mesh->N;
    }
    std::vector<int> ptr(N + 1, 0), adj;
    std::vector<float> rest;
    // a node's neighbours in the order of the usual plan, whatever plan the
    // solver has: the messages are summed in that order
    const std::vector<int>& order = usual_order(s);
    std::vector<int> pos(N), rank(N);
    for (int g = 0; g < N; ++g) pos[order[g]] = g;
    for (int g = 0; g < N; ++g) rank[g] = pos[Lh.perm_global[g]];
    for (int i = 0; i < N; ++i) {
        std::sort(nbr[i].begin(), nbr[i].end(), [&](const std::pair<int, float>& a, const std::pair<int, float>& b) {
            return rank[a.first] < rank[b.first];
        });
        for (auto& q : nbr[i]) { adj.push_back(q.first); rest.push_back(q.second); }
        ptr[i + 1] = (int)adj.size();
    }
    // Energy-norm weights of the loss's edge term: the PD system matrix
    // M + K approximated by M plus a graph Laplacian whose diagonal is K's
    // own (the Jacobi diagonal minus the mass), per unit mass: vertex i
    // spreads sigma_i = (D_i - m_i) / m_i evenly over its deg_i edges, and
    // an edge takes the mean of its two ends.  Pinned vertices contribute 0.
    std::vector<float> sig(N, 0.f), ew(adj.size(), 0.f);
    for (int i = 0; i < N; ++i) {
        const float4 a = Lh.aux[i];
        const float m = Lh.mass[i];
        const int deg = ptr[i + 1] - ptr[i];
        if (a.w > 0.f && m > 0.f && deg > 0) sig[i] = std::max(0.f, (1.f / (a.w * m) - 1.f) / (float)deg);
    }
    for (int i = 0; i < N; ++i)
        for (int e = ptr[i]; e < ptr[i + 1]; ++e) ew[e] = 0.5f * (sig[i] + sig[adj[e]]);
    cudaStream_t st = s->stream;
    int rc = upload_graph(w, N, ptr.data(), (int)adj.size(), adj.data(), st);
    if (rc) return rc;
    rc = graph_ok(w, st);
    if (rc) return rc;
    if (!rest.empty()) GK(cudaMemcpyAsync(w->rest.p, rest.data(), sizeof(float) * rest.size(), cudaMemcpyHostToDevice, st));
    if (!ew.empty()) GK(cudaMemcpyAsync(w->ew.p, ew.data(), sizeof(float) * ew.size(), cudaMemcpyHostToDevice, st));
    GK(cudaMemcpyAsync(w->stat.p, stat.data(), sizeof(float4) * N, cudaMemcpyHostToDevice, st));
    GK(s->warm.alloc(N));
    GK(cudaMemsetAsync(s->warm.p, 0, sizeof(float4) * N, st));
    // the solver's learned-start state: previous offsets (none valid yet)
    // and the learned chain of the judge
    if (s->dprev.n != (size_t)N) GK(s->dprev.alloc(N));
    GK(cudaMemsetAsync(s->dprev.p, 0, sizeof(float4) * N, st));
    GK(s->A2.alloc(N)); GK(s->B2.alloc(N));
    GK(s->crt2.alloc(Lh.ncloth));
    GK(s->acc2.alloc((size_t)Lh.ncloth * s->acc_stride));
    GK(cudaMemsetAsync(s->acc2.p, 0, sizeof(double) * (size_t)Lh.ncloth * s->acc_stride, st));
    GK(cudaStreamSynchronize(st));
    w->solver = s;
    s->ws = w;
    if (s->graph) { cudaGraphExecDestroy(s->graph); s->graph = nullptr; }
    return PDG_OK;
}

int pdg_warmstart_train_frame(pdg_warmstart* w, pdg_solver* s, float lr, float* loss)
{
    if (!w || !s || w->solver != s) return set_error(PDG_ERR_STATE, "pdg_warmstart_train_frame: not attached to this solver");
    cudaStream_t st = s->stream;
    const int N = w->N;
    GK(cudaMemcpyAsync(w->Xn.p, s->X.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    GK(cudaMemcpyAsync(w->Vn.p, s->V.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    GK(cudaMemcpyAsync(w->Dn.p, s->dprev.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    int rc = pdg_solver_step(s, 1, nullptr);
    if (rc) return rc;
    // inputs from (x_n, v_n, y, d_prev), target (x* - y - d_prev)/s from the solve
    k_node_feat<<<nb(N, 256), 256, 0, st>>>(N, w->Xn.p, w->Vn.p, s->Y.p, s->aux.p, w->stat.p, s->vcloth.p, s->cinfo.p,
                                            w->Dn.p, w->xin.p);
    launch_after(k_edge_feat, nb(N, 256), 256, 0, st, N, w->ptr.p, w->adj.p, w->rest.p, s->Y.p, w->ef.p);
    launch_after(k_target, nb(N, 256), 256, 0, st, N, s->X.p, s->Y.p, s->aux.p, w->Dn.p, w->target.p, w->freew.p);
    int nfree = 0;
    for (const auto& a : s->L.aux) nfree += a.w >= 0.f ? 1 : 0;
    rc = forward(w, st);
    if (rc) return rc;
    rc = backward(w, 1.f / (float)std::max(1, 3 * nfree), w->energy ? w->ew.p : nullptr, st);
    if (rc) return rc;
    if (lr > 0.f) {
        rc = adam_step(w, lr, st);
        if (rc) return rc;
    }
    // features and target 3, forward 2 + 3L, loss and backward 5 + 5L,
    // Adam 1
    s->launches += 3 + (2 + 3 * L) + (5 + 5 * L) + (lr > 0.f ? 1 : 0);
    double l = 0.0;
    GK(cudaMemcpyAsync(&l, w->loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    GK(cudaStreamSynchronize(st));
    if (loss) *loss = (float)l;
    return PDG_OK;
}

int pdg_warmstart_train_pair(pdg_warmstart* w, pdg_solver* traj, pdg_solver* deep, float lr, float* loss)
{
    if (!w || !traj || !deep || w->solver != traj)
        return set_error(PDG_ERR_STATE, "pdg_warmstart_train_pair: the network must be attached to `traj`");
    if (deep == traj || deep->L.ntot != traj->L.ntot || deep->L.ncloth != traj->L.ncloth ||
        deep->kernel == PDG_KERNEL_PERSISTENT || deep->kernel == PDG_KERNEL_RESIDENT)
        return set_error(PDG_ERR_ARG, "pdg_warmstart_train_pair: `deep` must solve the same cloths with the same "
                                      "vertex layout (same patch plan, per-sweep kernels)");
    // (patch sizes that the plans chose themselves may differ: the state then
    // goes from one vertex order to the other through the caller's)
    const bool same = deep->L.perm_global == traj->L.perm_global;
    int rc = PDG_OK;
    if (!same) {
        if (usual_order(traj) != usual_order(deep))
            return set_error(PDG_ERR_ARG, "pdg_warmstart_train_pair: `deep` must solve the same cloths with the same "
                                          "vertex layout (same patch plan, per-sweep kernels)");
    }
    cudaStream_t st = traj->stream;
    const int N = w->N;
    GK(cudaStreamSynchronize(deep->stream));
    // inputs (x_n, v_n, d_prev) of the trajectory; the deep solve starts from the same state
    GK(cudaMemcpyAsync(w->Xn.p, traj->X.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    GK(cudaMemcpyAsync(w->Vn.p, traj->V.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    GK(cudaMemcpyAsync(w->Dn.p, traj->dprev.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    if (same) {
        GK(cudaMemcpyAsync(deep->X.p, traj->X.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
        GK(cudaMemcpyAsync(deep->V.p, traj->V.p, sizeof(float4) * N, cudaMemcpyDeviceToDevice, st));
    } else {
        GK(w->Xd.reserve(N));
        GK(launch_take_state(traj->X.p, traj->V.p, traj->stage_x.p, traj->stage_v.p, traj->inv_global.p, N, st));
        GK(launch_put_state(traj->stage_x.p, traj->stage_v.p, deep->X.p, deep->V.p, deep->inv_global.p, N, st, nullptr));
    }
    GK(cudaStreamSynchronize(st));
    rc = pdg_solver_step(deep, 1, nullptr);   // the target: x* of this frame
    if (rc) return rc;
    GK(cudaStreamSynchronize(deep->stream));
    rc = pdg_solver_step(traj, 1, nullptr);       // the trajectory and its kept offsets advance
    if (rc) return rc;
    // y of both solvers is the same prediction from the same state
    k_node_feat<<<nb(N, 256), 256, 0, st>>>(N, w->Xn.p, w->Vn.p, traj->Y.p, traj->aux.p, w->stat.p, traj->vcloth.p,
                                            traj->cinfo.p, w->Dn.p, w->xin.p);
    launch_after(k_edge_feat, nb(N, 256), 256, 0, st, N, w->ptr.p, w->adj.p, w->rest.p, traj->Y.p, w->ef.p);
    const float4* xs = deep->X.p;
    if (!same) {
        GK(launch_take_state(deep->X.p, nullptr, traj->stage_x.p, nullptr, deep->inv_global.p, N, st));
        GK(launch_put_state(traj->stage_x.p, nullptr, w->Xd.p, nullptr, traj->inv_global.p, N, st, nullptr));
        xs = w->Xd.p;
    }
    launch_after(k_target, nb(N, 256), 256, 0, st, N, xs, traj->Y.p, traj->aux.p, w->Dn.p, w->target.p, w->freew.p);
    int nfree = 0;
    for (const auto& a : traj->L.aux) nfree += a.w >= 0.f ? 1 : 0;
    rc = forward(w, st);
    if (rc) return rc;
    rc = backward(w, 1.f / (float)std::max(1, 3 * nfree), w->energy ? w->ew.p : nullptr, st);
    if (rc) return rc;
    if (lr > 0.f) {
        rc = adam_step(w, lr, st);
        if (rc) return rc;
    }
    traj->launches += (same ? 3 : 7) + (2 + 3 * L) + (5 + 5 * L) + (lr > 0.f ? 1 : 0);
    double l = 0.0;
    GK(cudaMemcpyAsync(&l, w->loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    GK(cudaStreamSynchronize(st));
    if (loss) *loss = (float)l;
    return PDG_OK;
}

int pdg_warmstart_set_smoothness(pdg_warmstart* w, float lambda)
{
    if (!w || !(lambda >= 0.f) || !std::isfinite(lambda))
        return set_error(PDG_ERR_ARG, "pdg_warmstart_set_smoothness: lambda must be finite and >= 0");
    w->smooth = lambda;
    return PDG_OK;
}

int pdg_warmstart_time_inference(pdg_warmstart* w, int reps, float* ms)
{
    if (!w || reps <= 0 || !ms) return set_error(PDG_ERR_ARG, "pdg_warmstart_time_inference: bad arguments");
    pdg_solver* s = w->solver;
    if (!s) return set_error(PDG_ERR_STATE, "pdg_warmstart_time_inference: not attached to a solver");
    cudaEvent_t e0, e1;
    GK(cudaEventCreate(&e0));
    GK(cudaEventCreate(&e1));
    int rc = warm_infer_enqueue(w, s);   // untimed first run
    GK(cudaEventRecord(e0, s->stream));
    for (int r = 0; r < reps && rc == PDG_OK; ++r) rc = warm_infer_enqueue(w, s);
    GK(cudaEventRecord(e1, s->stream));
    GK(cudaEventSynchronize(e1));
    float t = 0.f;
    GK(cudaEventElapsedTime(&t, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    s->launches += (long long)(reps + 1) * warm_kernel_count();
    *ms = t / (float)reps;
    return PDG_OK;
}

int pdg_warmstart_set_energy_norm(pdg_warmstart* w, int enable)
{
    if (!w) return set_error(PDG_ERR_ARG, "pdg_warmstart_set_energy_norm: null argument");
    w->energy = enable ? 1 : 0;
    return PDG_OK;
}

int pdg_warmstart_set_judge_sweeps(pdg_warmstart* w, int sweeps)
{
    if (!w || sweeps < 0 || sweeps > 1000)
        return set_error(PDG_ERR_ARG, "pdg_warmstart_set_judge_sweeps: sweeps must be in [0, 1000]");
    w->judge = sweeps;
    // the frame graph of an attached solver holds the judge's launches
    if (w->solver && w->solver->graph) { cudaGraphExecDestroy(w->solver->graph); w->solver->graph = nullptr; }
    return PDG_OK;
}

int pdg_warmstart_get_judge_sweeps(const pdg_warmstart* w, int* sweeps)
{
    if (!w || !sweeps) return set_error(PDG_ERR_ARG, "pdg_warmstart_get_judge_sweeps: null argument");
    *sweeps = w->judge;
    return PDG_OK;
}

void pdg_warmstart_destroy(pdg_warmstart* w)
{
    if (!w) return;
    if (w->solver) { w->solver->ws = nullptr; if (w->solver->graph) { cudaGraphExecDestroy(w->solver->graph); w->solver->graph = nullptr; } }
    delete w;
}

}  // extern "C"
