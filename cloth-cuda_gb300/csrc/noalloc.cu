// pdg_step_noalloc: one frame of the consistent PD solve that allocates no
// device memory.
//
// Who needs it: callers that cannot call cudaMalloc -- applications that own
// all device memory through their own pool (engines and hosts that load this
// library as a plugin and forbid allocation behind their back), and real-time
// loops that cannot afford cudaMalloc/cudaFree, which synchronise the whole
// device.  They pass the cloth in the reference's own device layout (the
// arrays of ClothMesh, SimConstraints and Constraints) and get the frame
// solved in place.
//
// Where the scratch lives: the per-frame work arrays (inertial prediction,
// the two offset iterates, the force accumulator, the per-sweep residual
// sums and the control word) sit in one file-scope __device__ array of
// kScratchBytes (about 8.4 MB), which every GPU that loads the library holds
// until the process exits.  Sizes beyond PDG_NOALLOC_MAX_VERTS vertices or
// PDG_NOALLOC_MAX_ITERS sweeps are rejected.  Host code cannot use the
// array's name as a device address, so the first call on each device looks
// the address up with cudaGetSymbolAddress (with that device current) and
// caches it; make that first call before any stream capture.  All calls share
// the array and it keeps the last call's contents: each call clears what
// must start at zero, and calls that overlap on the GPU (different streams,
// or different host threads) race on it.
//
// The frame is one cooperative launch.  Its sweeps alternate two phases with a
// grid barrier after each: the elements (one thread per triangle or hinge)
// add their corner forces to the accumulator, the vertices take their update
// and clear it.  What bounds it is latency, not bytes: a 129x129 cloth moves
// about 5 MB per sweep through L2.  The former form issued five launches per
// sweep (control, clear, triangles, hinges, update; three scalar atomics per
// corner).  A frame of 32 sweeps at 129x129 took 875 us in that form, 355 us
// as one launch with one 16-byte reduction per corner, and takes 220 us with
// what a frame does not change kept in registers and one arrival per block
// and barrier.  The float reductions add in any order, so results match
// pdg_solver_step to rounding, not bitwise.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../../include/pdg.h"
#include "pd_kernels.cuh"
#include "pdg_host.h"

namespace pdg {
namespace {

constexpr int kMaxVerts = PDG_NOALLOC_MAX_VERTS;
constexpr int kMaxIters = PDG_NOALLOC_MAX_ITERS;

struct NaCtl {
    int active, used, status, pad;
    double res_y2, res0_2, resf_2;
    unsigned bar;      // grid barrier: arrivals so far (cleared before each frame)
    int err;           // a barrier wait gave up (cleared with them)
};

constexpr size_t kOffY = 0;
constexpr size_t kOffA = kOffY + 16 * (size_t)kMaxVerts;
constexpr size_t kOffB = kOffA + 16 * (size_t)kMaxVerts;
constexpr size_t kOffF = kOffB + 16 * (size_t)kMaxVerts;
constexpr size_t kOffAcc = kOffF + 16 * (size_t)kMaxVerts;
constexpr size_t kOffCtl = kOffAcc + 8 * (size_t)(kMaxIters + 2);
constexpr size_t kScratchBytes = kOffCtl + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

struct Scratch {
    float4* Y; float4* A; float4* B; float4* F; double* acc; NaCtl* ctl;
};

Scratch carve(unsigned char* base)
{
    Scratch s;
    s.Y = reinterpret_cast<float4*>(base + kOffY);
    s.A = reinterpret_cast<float4*>(base + kOffA);
    s.B = reinterpret_cast<float4*>(base + kOffB);
    s.F = reinterpret_cast<float4*>(base + kOffF);
    s.acc = reinterpret_cast<double*>(base + kOffAcc);
    s.ctl = reinterpret_cast<NaCtl*>(base + kOffCtl);
    return s;
}

constexpr int kNaThreads = 512;
constexpr long long kNaWaitCycles = 4000000000LL;   // about 2 s: bound of a barrier wait

struct NaArgs {
    Scratch s;
    int N, T, E, P;
    float *pos, *vel;
    const float *mass, *diag;
    const int* tris;
    const float *Dm_inv, *area, *ks;
    const int* quads;
    const float *w4, *nrest, *kb;
    const int* pin_idx;
    const float* pin_target;
    float h, ax, ay, az, damping, gamma, tol, rho2;
    int cap, have_final, use_cheb, cheb_delay;
};

// Barrier `phase` (1, 2, ...) of the frame over the grid: one arrival per
// block on a count that only grows, polled until all blocks of the phase are
// in.  False on every thread of a block once a wait, here or in another
// block, gave up.
__device__ __forceinline__ bool na_barrier(NaCtl* c, unsigned& phase)
{
    __shared__ int ok;
    __syncthreads();
    ++phase;
    if (threadIdx.x == 0) {
        const unsigned want = phase * gridDim.x;
        __threadfence();
        atomicAdd(&c->bar, 1u);
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(&c->bar)) : "memory");
        if (v < want) {
            const long long t0 = clock64();
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(&c->bar)) : "memory");
                if (clock64() - t0 > kNaWaitCycles) { atomicCAS(&c->err, 0, 1); break; }
            } while (v < want);
        }
        ok = v >= want;
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ void na_add(float4* F, int v, float x, float y, float z)
{
    atomicAdd(&F[v], make_float4(x, y, z, 0.f));   // one 16-byte reduction
}

// A triangle (quad i3 < 0) or hinge with what does not change over the
// sweeps of a frame: its corners, constants and the prediction's edge vectors.
struct NaElem {
    int i0, i1, i2, i3;
    float4 c;             // Dm_inv, or the hinge's weights
    float s, nrest;       // h^2 k area, or h^2 k and the rest norm
    float3 e1, e2, e3;    // y_1 - y_0, y_2 - y_0, y_3 - y_0
    float3 y0;
};

__device__ __forceinline__ float3 na_sub(float4 p, float4 q)
{
    return make_float3(fsub(p.x, q.x), fsub(p.y, q.y), fsub(p.z, q.z));
}

__device__ __forceinline__ NaElem na_element(const NaArgs& a, long long q)
{
    NaElem m;
    const float h2 = fmul(a.h, a.h);
    if (q < a.T) {
        const int t = (int)q;
        m.i0 = a.tris[3 * t]; m.i1 = a.tris[3 * t + 1]; m.i2 = a.tris[3 * t + 2]; m.i3 = -1;
        m.c = make_float4(a.Dm_inv[4 * t], a.Dm_inv[4 * t + 1], a.Dm_inv[4 * t + 2], a.Dm_inv[4 * t + 3]);
        m.s = h2 * (a.ks[t] * a.area[t]);
        m.nrest = 0.f;
    } else {
        const int e = (int)(q - a.T);
        m.i0 = a.quads[4 * e]; m.i1 = a.quads[4 * e + 1]; m.i2 = a.quads[4 * e + 2]; m.i3 = a.quads[4 * e + 3];
        m.c = make_float4(a.w4[4 * e], a.w4[4 * e + 1], a.w4[4 * e + 2], a.w4[4 * e + 3]);
        m.s = h2 * a.kb[e];
        m.nrest = a.nrest[e];
    }
    const float4 y0 = __ldcg(&a.s.Y[m.i0]), y1 = __ldcg(&a.s.Y[m.i1]), y2 = __ldcg(&a.s.Y[m.i2]);
    const float4 y3 = m.i3 >= 0 ? __ldcg(&a.s.Y[m.i3]) : y0;
    m.e1 = na_sub(y1, y0); m.e2 = na_sub(y2, y0); m.e3 = na_sub(y3, y0);
    m.y0 = f3(y0);
    return m;
}

// Adds the element's corner forces at offsets D to F.
__device__ __forceinline__ void na_apply(const NaElem& m, const float4* D, float4* F)
{
    const float4 d0 = __ldcg(&D[m.i0]), d1 = __ldcg(&D[m.i1]), d2 = __ldcg(&D[m.i2]);
    const float4 d3 = m.i3 >= 0 ? __ldcg(&D[m.i3]) : d0;
    const float3 e1 = fadd3(m.e1, na_sub(d1, d0)), e2 = fadd3(m.e2, na_sub(d2, d0));
    if (m.i3 < 0) {
        float3 c0, c1, c2;
        tri_force<kModeConsistent>(e1, e2, m.c, m.s, c0, c1, c2);
        na_add(F, m.i0, c0.x, c0.y, c0.z);
        na_add(F, m.i1, c1.x, c1.y, c1.z);
        na_add(F, m.i2, c2.x, c2.y, c2.z);
    } else {
        const float3 e3 = fadd3(m.e3, na_sub(d3, d0));
        const float3 x0 = make_float3(fadd(m.y0.x, d0.x), fadd(m.y0.y, d0.y), fadd(m.y0.z, d0.z));
        const float3 f = hinge_force<kModeConsistent>(e1, e2, e3, x0, m.c, m.s, m.nrest);
        na_add(F, m.i0, fmul(f.x, m.c.x), fmul(f.y, m.c.x), fmul(f.z, m.c.x));
        na_add(F, m.i1, fmul(f.x, m.c.y), fmul(f.y, m.c.y), fmul(f.z, m.c.y));
        na_add(F, m.i2, fmul(f.x, m.c.z), fmul(f.y, m.c.z), fmul(f.z, m.c.z));
        na_add(F, m.i3, fmul(f.x, m.c.w), fmul(f.y, m.c.w), fmul(f.z, m.c.w));
    }
}

// Two 512-thread blocks per SM at 64 registers: a 129x129 cloth's 80,000
// elements are then one per thread on all 152 SMs.
// ONE: no thread has more than one element; its element's constants and rest
// of the prediction then stay in registers for the frame, so that a sweep's
// only loads are the offsets of its corners (one trip to L2).  Likewise each
// thread keeps its first vertex's mass, prediction and last two offsets.
template <bool ONE>
__global__ void __launch_bounds__(kNaThreads, 2) k_na_frame(NaArgs a)
{
    __shared__ float red[kNaThreads / 32];
    __shared__ int done_s;
    const Scratch s = a.s;
    NaCtl* ctl = s.ctl;
    const int gtid = blockIdx.x * kNaThreads + threadIdx.x, gstride = gridDim.x * kNaThreads;
    const float h = a.h, h2 = fmul(h, h);
    const int nsweep = a.cap + a.have_final;
    unsigned phase = 0;

    // prediction, start offsets, cleared sums
    for (int i = gtid; i < a.cap + 2; i += gstride) s.acc[i] = 0.0;
    for (int i = gtid; i < a.N; i += gstride) {
        float4 y;
        y.x = ffma(h2, a.ax, ffma(h, a.vel[3 * i], a.pos[3 * i]));
        y.y = ffma(h2, a.ay, ffma(h, a.vel[3 * i + 1], a.pos[3 * i + 1]));
        y.z = ffma(h2, a.az, ffma(h, a.vel[3 * i + 2], a.pos[3 * i + 2]));
        y.w = a.mass[i];
        s.Y[i] = y;
        const float dg = a.diag[i];
        const float4 d0 = make_float4(0.f, 0.f, 0.f, dg > 1e-10f ? 1.0f / dg : 0.f);   // inertial start
        s.A[i] = d0;
        s.B[i] = d0;
        s.F[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!na_barrier(ctl, phase)) return;
    if (a.P > 0) {
        for (int q = gtid; q < a.P; q += gstride) {
            const int i = a.pin_idx[q];
            const float4 y = __ldcg(&s.Y[i]);
            const float4 d = make_float4(fsub(a.pin_target[3 * q], y.x), fsub(a.pin_target[3 * q + 1], y.y),
                                         fsub(a.pin_target[3 * q + 2], y.z), -1.f);
            s.A[i] = d;
            s.B[i] = d;
        }
        if (!na_barrier(ctl, phase)) return;
    }

    NaElem el;
    if (ONE && gtid < a.T + a.E) el = na_element(a, gtid);
    float4 vd = make_float4(0.f, 0.f, 0.f, 0.f), vp = vd, vy = vd;   // vertex gtid: d^k, d^(k-1), y
    if (gtid < a.N) { vd = __ldcg(&s.A[gtid]); vp = vd; vy = __ldcg(&s.Y[gtid]); }

    bool active = true;
    float om = 1.f;
    for (int k = 0; k < nsweep; ++k) {
        const bool res_only = k >= a.cap;
        if (!res_only) {   // Chebyshev weight of sweep k (the solver's recurrence)
            if (!a.use_cheb || k < a.cheb_delay) om = 1.f;
            else if (k == a.cheb_delay) om = fdiv(2.f, fsub(2.f, a.rho2));
            else om = fdiv(4.f, fsub(4.f, fmul(a.rho2, om)));
        }
        // the decision at the start of sweep k, the same in every block:
        // converged or failed frames end here
        if (k >= 1) {
            if (threadIdx.x == 0) {
                const double acc0 = __ldcg(&s.acc[0]), rk2 = __ldcg(&s.acc[k - 1]);
                const bool bad = !isfinite(rk2);
                const bool conv = a.tol > 0.f && rk2 <= (double)a.tol * (double)a.tol * acc0;
                done_s = bad || conv;
                if (blockIdx.x == 0) {
                    if (k == 1) { ctl->res0_2 = acc0; ctl->res_y2 = acc0; }
                    if (done_s) { ctl->status = bad ? -6 : 0; ctl->used = k - 1; ctl->resf_2 = rk2; ctl->active = 0; }
                }
            }
            __syncthreads();
            if (done_s) { active = false; break; }
        }
        const float4* D = (k & 1) ? s.B : s.A;
        float4* Dn = (k & 1) ? s.A : s.B;
        // elements
        if (ONE) {
            if (gtid < a.T + a.E) na_apply(el, D, s.F);
        } else {
            for (long long q = gtid; q < (long long)a.T + a.E; q += gstride) na_apply(na_element(a, q), D, s.F);
        }
        if (!na_barrier(ctl, phase)) return;
        // vertices; the accumulator is left clear for the next sweep
        float r2 = 0.f;
        for (int i = gtid; i < a.N; i += gstride) {
            const bool first = i == gtid;
            const float4 f4 = __ldcg(&s.F[i]);
            const float4 d = first ? vd : __ldcg(&D[i]), y = first ? vy : __ldcg(&s.Y[i]);
            const float4 dp = res_only ? d : (first ? vp : __ldcg(&Dn[i]));
            float rv;
            const float4 o = update_consistent(d, y, make_float3(f4.x, f4.y, f4.z), dp, a.gamma, res_only ? 1.f : om, rv);
            r2 += rv;
            if (!res_only) Dn[i] = o;
            s.F[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (first && !res_only) { vp = d; vd = o; }
        }
        block_residual<kNaThreads>(r2, red, s.acc + k);
        if (!na_barrier(ctl, phase)) return;
    }

    // the frame's record (block 0, a warp looks through the sums), known to
    // the other blocks after one more barrier
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        if (a.cap <= 1 && threadIdx.x == 0) { ctl->res0_2 = __ldcg(&s.acc[0]); ctl->res_y2 = __ldcg(&s.acc[0]); }
        if (active) {
            bool finite = true;
            for (int k = threadIdx.x; k <= a.cap; k += 32) {
                const double v = __ldcg(&s.acc[k]);
                finite = finite && isfinite(v);
            }
            finite = __all_sync(0xffffffffu, finite) != 0;
            if (threadIdx.x == 0) {
                ctl->used = a.cap;
                ctl->resf_2 = a.have_final ? __ldcg(&s.acc[a.cap]) : -1.0;
                ctl->status = finite ? 0 : -6;
                ctl->active = 0;
            }
        }
    }
    if (!na_barrier(ctl, phase)) return;
    const int status = __ldcg(&ctl->status), used = __ldcg(&ctl->used);
    const float4* D = (used & 1) ? s.B : s.A;
    const float sc = 1.f - a.damping, ih = fdiv(1.f, h);
    for (int i = gtid; i < a.N; i += gstride) {
        const float4 d = __ldcg(&D[i]);
        if (d.w < 0.f) continue;   // pinned: written below
        if (status != 0) {         // failed frame: keep x_n, stop the cloth
            a.vel[3 * i] = 0.f; a.vel[3 * i + 1] = 0.f; a.vel[3 * i + 2] = 0.f;
            continue;
        }
        const float4 y = __ldcg(&s.Y[i]);
        a.vel[3 * i] = fmul(sc, ffma(d.x, ih, ffma(h, a.ax, a.vel[3 * i])));
        a.vel[3 * i + 1] = fmul(sc, ffma(d.y, ih, ffma(h, a.ay, a.vel[3 * i + 1])));
        a.vel[3 * i + 2] = fmul(sc, ffma(d.z, ih, ffma(h, a.az, a.vel[3 * i + 2])));
        a.pos[3 * i] = fadd(y.x, d.x); a.pos[3 * i + 1] = fadd(y.y, d.y); a.pos[3 * i + 2] = fadd(y.z, d.z);
    }
    for (int q = gtid; q < a.P; q += gstride) {
        const int i = a.pin_idx[q];
        a.pos[3 * i] = a.pin_target[3 * q]; a.pos[3 * i + 1] = a.pin_target[3 * q + 1]; a.pos[3 * i + 2] = a.pin_target[3 * q + 2];
        a.vel[3 * i] = 0.f; a.vel[3 * i + 1] = 0.f; a.vel[3 * i + 2] = 0.f;
    }
}

// Device address of the scratch array, looked up once per device.
std::mutex g_mu;
unsigned char* g_addr[64] = {};
int g_blocks[64] = {};   // blocks of k_na_frame resident at once

int scratch_of(int dev, unsigned char** out, int* blocks)
{
    if (dev < 0 || dev >= 64) return set_error(PDG_ERR_ARG, "pdg_step_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return set_error(PDG_ERR_CUDA, "pdg_step_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        int nsm = 0, per = 0, per2 = 0;
        if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_na_frame<true>, kNaThreads, 0) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, k_na_frame<false>, kNaThreads, 0) != cudaSuccess ||
            std::min(per, per2) <= 0)
            return set_error(PDG_ERR_CUDA, "pdg_step_noalloc: occupancy query failed");
        g_blocks[dev] = nsm * std::min(per, per2);
        g_addr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_addr[dev];
    *blocks = g_blocks[dev];
    return PDG_OK;
}

}  // namespace
}  // namespace pdg

using namespace pdg;

#define NA_CK(call)                                                                                \
    do {                                                                                           \
        const cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) return set_error(PDG_ERR_CUDA, "pdg_step_noalloc: %s", cudaGetErrorString(e_)); \
    } while (0)

extern "C" int pdg_step_noalloc(const pdg_config* cfg, int N, float* d_pos, float* d_vel, const float* d_mass,
                                const float* d_jacobi_diag, int T, const int* d_tris, const float* d_Dm_inv,
                                const float* d_rest_area, const float* d_stretch_k, int E, const int* d_bend_quads,
                                const float* d_bend_w, const float* d_bend_n, const float* d_bend_k, int P,
                                const int* d_pin_idx, const float* d_pin_target, void* stream,
                                pdg_frame_stats* stats)
{
    if (!cfg) return set_error(PDG_ERR_ARG, "pdg_step_noalloc: null config");
    if (N <= 0 || N > kMaxVerts)
        return set_error(PDG_ERR_ARG, "pdg_step_noalloc: %d vertices; this entry point handles 1..%d", N, kMaxVerts);
    if (cfg->max_iterations < 0 || cfg->max_iterations > kMaxIters)
        return set_error(PDG_ERR_ARG, "pdg_step_noalloc: max_iterations %d; this entry point handles 0..%d",
                         cfg->max_iterations, kMaxIters);
    if (T < 0 || E < 0 || P < 0) return set_error(PDG_ERR_ARG, "pdg_step_noalloc: negative count");
    if (cfg->mode != PDG_MODE_CONSISTENT || cfg->init != PDG_INIT_INERTIAL)
        return set_error(PDG_ERR_ARG, "pdg_step_noalloc: only the consistent mode from the inertial start");
    if (!(cfg->dt > 0.f) || !(cfg->damping >= 0.f && cfg->damping <= 1.f) || !(cfg->gamma > 0.f) ||
        (cfg->use_chebyshev && !(cfg->rho >= 0.f && cfg->rho < 1.f)) || cfg->cheb_delay < 0)
        return set_error(PDG_ERR_ARG, "pdg_step_noalloc: invalid dt, damping, gamma, rho or cheb_delay");
    if (!d_pos || !d_vel || !d_mass || !d_jacobi_diag || (T && (!d_tris || !d_Dm_inv || !d_rest_area || !d_stretch_k)) ||
        (E && (!d_bend_quads || !d_bend_w || !d_bend_n || !d_bend_k)) || (P && (!d_pin_idx || !d_pin_target)))
        return set_error(PDG_ERR_ARG, "pdg_step_noalloc: null device array");

    int dev = 0;
    NA_CK(cudaGetDevice(&dev));
    if (stream) {   // the scratch address is this device's: the stream must belong to it
        int sdev = -1;
        NA_CK(cudaStreamGetDevice(static_cast<cudaStream_t>(stream), &sdev));
        if (sdev != dev)
            return set_error(PDG_ERR_ARG, "pdg_step_noalloc: the stream belongs to device %d, the current device is %d",
                             sdev, dev);
    }
    unsigned char* base = nullptr;
    int max_blocks = 0;
    const int rc = scratch_of(dev, &base, &max_blocks);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    NaArgs a{};
    a.s = carve(base);
    a.N = N; a.T = T; a.E = E; a.P = P;
    a.pos = d_pos; a.vel = d_vel; a.mass = d_mass; a.diag = d_jacobi_diag;
    a.tris = d_tris; a.Dm_inv = d_Dm_inv; a.area = d_rest_area; a.ks = d_stretch_k;
    a.quads = d_bend_quads; a.w4 = d_bend_w; a.nrest = d_bend_n; a.kb = d_bend_k;
    a.pin_idx = d_pin_idx; a.pin_target = d_pin_target;
    a.h = cfg->dt; a.ax = cfg->wind[0]; a.ay = cfg->gravity + cfg->wind[1]; a.az = cfg->wind[2];
    a.damping = cfg->damping; a.gamma = cfg->gamma; a.tol = cfg->tolerance; a.rho2 = cfg->rho * cfg->rho;
    a.cap = cfg->max_iterations;
    a.have_final = (cfg->compute_final_residual || cfg->tolerance > 0.f) ? 1 : 0;
    a.use_cheb = cfg->use_chebyshev; a.cheb_delay = cfg->cheb_delay;
    // one element per thread as far as the resident blocks go
    const long long work = std::max((long long)T + E, (long long)N);
    const int grid = (int)std::max(1LL, std::min((long long)max_blocks, (work + kNaThreads - 1) / kNaThreads));
    NA_CK(cudaMemsetAsync(a.s.ctl, 0, sizeof(NaCtl), st));
    void* args[] = {&a};
    const void* kernel = (long long)T + E <= (long long)grid * kNaThreads ? (const void*)k_na_frame<true>
                                                                          : (const void*)k_na_frame<false>;
    NA_CK(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kNaThreads), args, 0, st));

    if (stats) {
        NaCtl c;
        NA_CK(cudaMemcpyAsync(&c, a.s.ctl, sizeof(NaCtl), cudaMemcpyDeviceToHost, st));
        NA_CK(cudaStreamSynchronize(st));
        if (c.err) return set_error(PDG_ERR_TIMEOUT, "pdg_step_noalloc: bounded wait ran out (grid barrier)");
        stats->iterations = c.used;
        stats->warm_start_used = 0;
        stats->status = c.status;
        stats->res_inertial = std::sqrt(std::fmax(0.0, c.res_y2));
        stats->res_initial = std::sqrt(std::fmax(0.0, c.res0_2));
        stats->res_final = c.resf_2 >= 0.0 ? std::sqrt(c.resf_2) : -1.0;
        stats->rel_residual = (stats->res_final >= 0.0 && stats->res_inertial > 0.0)
                                  ? stats->res_final / stats->res_inertial : -1.0;
        stats->converged = (c.status == 0 && cfg->tolerance > 0.f && stats->res_final >= 0.0 &&
                            stats->res_final <= (double)cfg->tolerance * stats->res_inertial) ? 1 : 0;
    }
    return PDG_OK;
}
