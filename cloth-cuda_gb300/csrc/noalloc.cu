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
// The frame is one cooperative launch: the elements (one thread per triangle
// or hinge) add their corner forces to an accumulator, grid barrier, the
// vertices are updated from it.  Where every element and vertex has its own
// thread each element updates its corners itself (k_na_one), which leaves one
// barrier per sweep; larger cloths take two (k_na_frame).  What bounds it is
// latency, not bytes: a 129x129 cloth moves about 5 MB per sweep through L2.
// A frame of 32 sweeps at 129x129 took 875 us as five launches per sweep
// (control, clear, triangles, hinges, update; three scalar atomics per
// corner), 220 us as one launch with two barriers per sweep, one 16-byte
// reduction per corner and what a frame does not change kept in registers, and
// takes 141 us now.  The float reductions add in any order, so results match
// pdg_solver_step to rounding, not bitwise.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../../include/pdg.h"
#include "noalloc_wait.h"
#include "pd_kernels.cuh"
#include "pdg_host.h"

namespace pdg {
namespace {

constexpr int kMaxVerts = PDG_NOALLOC_MAX_VERTS;
constexpr int kMaxIters = PDG_NOALLOC_MAX_ITERS;

struct NaCtl {
    int active, used, status, pad;
    double res_y2, res0_2, resf_2;
    unsigned bar;      // grid barrier: arrivals so far, kNaGaveUp (cleared before each frame)
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

// The frame's barrier word (noalloc_wait.h) on the device.
struct NaBarWord {
    unsigned* p;
    long long t0;
    __device__ __forceinline__ void arrive()
    {
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(1u) : "memory");
    }
    __device__ __forceinline__ unsigned look()
    {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)) : "memory");
        return v;
    }
    __device__ __forceinline__ void start() { t0 = clock64(); }
    __device__ __forceinline__ bool late() { return clock64() - t0 > kNaWaitCycles; }
    __device__ __forceinline__ void replace(unsigned v, unsigned to) { atomicCAS(p, v, to); }
};

// Barrier `phase` (1, 2, ...) of the frame over the grid: one arrival per
// block on a count that only grows, polled until all blocks of the phase are
// in.  False once a wait, here or in another block, gave up.  na_wait is the
// part of one thread, between two block barriers; its arrival releases what
// the block did before (with a full fence and a relaxed arrival 32 sweeps of a
// 129x129 cloth took 156 us instead of 150).
__device__ __forceinline__ bool na_wait(NaCtl* c, unsigned phase)
{
    NaBarWord w{&c->bar, 0};
    return na_wait_on(w, phase * gridDim.x);
}
__device__ __forceinline__ bool na_barrier(NaCtl* c, unsigned& phase)
{
    __shared__ int ok;
    __syncthreads();
    ++phase;
    if (threadIdx.x == 0) ok = na_wait(c, phase);
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

// STEP 1: the predictions in an array, 2: paired with the offsets.
template <int STEP>
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
    const float4 y0 = a.s.Y[STEP * m.i0], y1 = a.s.Y[STEP * m.i1], y2 = a.s.Y[STEP * m.i2];
    const float4 y3 = m.i3 >= 0 ? a.s.Y[STEP * m.i3] : y0;
    m.e1 = na_sub(y1, y0); m.e2 = na_sub(y2, y0); m.e3 = na_sub(y3, y0);
    m.y0 = f3(y0);
    return m;
}

// Adds the element's corner forces at its corners' offsets to F.
__device__ __forceinline__ void na_apply(const NaElem& m, float4 d0, float4 d1, float4 d2, float4 d3, float4* F)
{
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

// The frame's outcome from the sums, found by a warp of every block for itself:
// its status, and the frame's record (block 0).  stop: the sweep after which
// the tolerance ended the frame, or -1.
__device__ __forceinline__ void na_outcome(const NaArgs& a, int stop, int& status)
{
    const Scratch s = a.s;
    const int lane = threadIdx.x, nsweep = a.cap + a.have_final;
    // without a tolerance no decision was taken: the first sum that is not
    // finite ended the frame
    int bad = 0x7fffffff;
    bool finite = true;
    for (int k = lane; k <= a.cap; k += 32) {
        const bool f = isfinite(__ldcg(&s.acc[k]));
        finite = finite && f;
        if (stop < 0 && !f && k + 1 < nsweep) bad = min(bad, k);
    }
    bad = __reduce_min_sync(0xffffffffu, bad);
    finite = __all_sync(0xffffffffu, finite) != 0;
    if (lane == 0) {
        const int j = stop >= 0 ? stop : (bad != 0x7fffffff ? bad : -1);   // ended after sweep j
        const int used = j >= 0 ? j : a.cap;
        const double rf = j >= 0 || a.have_final ? __ldcg(&s.acc[used]) : -1.0;
        status = j >= 0 ? (isfinite(rf) ? 0 : -6) : (finite ? 0 : -6);
        if (blockIdx.x == 0) {
            const double acc0 = __ldcg(&s.acc[0]);
            s.ctl->res0_2 = acc0; s.ctl->res_y2 = acc0; s.ctl->resf_2 = rf;
            s.ctl->used = used; s.ctl->status = status; s.ctl->active = 0;
        }
    }
}

// The barrier that ends sweep k: the block's residual (r2 of its threads) is
// added to the sweep's sum, and with a tolerance the decision about sweep k
// follows, the same in every block (done).  With a tolerance the residual is
// added before the arrival, otherwise only after the last sweep: the next
// barrier makes it visible (129x129: 145 us instead of 150).  False once a
// wait gave up.
template <int NT>
__device__ __forceinline__ bool na_end_sweep(const NaArgs& a, unsigned& phase, int k, bool last, bool has_own, float r2,
                                             int& done)
{
    __shared__ float red[NT / 32];
    __shared__ int ok_s, done_s;
    const bool sum = has_own && k >= 0;
    if (sum) {
        r2 = warp_sum(r2);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = r2;
    }
    __syncthreads();
    ++phase;
    const bool late = !(a.tol > 0.f) && !last;
    if (sum && (threadIdx.x >> 5) == (late ? 1 : 0)) {
        const int lane = threadIdx.x & 31;
        const float v = warp_sum(lane < NT / 32 ? red[lane] : 0.f);
        if (lane == 0) atomicAdd(a.s.acc + k, (double)v);
    }
    if (threadIdx.x == 0) {
        ok_s = na_wait(a.s.ctl, phase);
        int d = 0;
        if (a.tol > 0.f && k >= 0 && !last) {
            const double acc0 = __ldcg(&a.s.acc[0]), rk2 = __ldcg(&a.s.acc[k]);
            d = !isfinite(rk2) || rk2 <= (double)a.tol * (double)a.tol * acc0;
        }
        done_s = d;
    }
    __syncthreads();
    done = done_s;
    return ok_s != 0;
}

// Chebyshev weight of sweep k from that of the sweep before (the solver's
// recurrence).
__device__ __forceinline__ float na_omega(const NaArgs& a, int k, float om)
{
    if (!a.use_cheb || k < a.cheb_delay) return 1.f;
    if (k == a.cheb_delay) return fdiv(2.f, fsub(2.f, a.rho2));
    return fdiv(4.f, fsub(4.f, fmul(a.rho2, om)));
}

// A vertex's new state after the sweeps (d: its offset), or what a failed
// frame leaves.
__device__ __forceinline__ void na_finalize(const NaArgs& a, int i, float4 y, float3 d, int status)
{
    if (status != 0) {         // keep x_n, stop the cloth
        a.vel[3 * i] = 0.f; a.vel[3 * i + 1] = 0.f; a.vel[3 * i + 2] = 0.f;
        return;
    }
    const float h = a.h, sc = 1.f - a.damping, ih = fdiv(1.f, h);
    a.vel[3 * i] = fmul(sc, ffma(d.x, ih, ffma(h, a.ax, a.vel[3 * i])));
    a.vel[3 * i + 1] = fmul(sc, ffma(d.y, ih, ffma(h, a.ay, a.vel[3 * i + 1])));
    a.vel[3 * i + 2] = fmul(sc, ffma(d.z, ih, ffma(h, a.az, a.vel[3 * i + 2])));
    a.pos[3 * i] = fadd(y.x, d.x); a.pos[3 * i + 1] = fadd(y.y, d.y); a.pos[3 * i + 2] = fadd(y.z, d.z);
}

// Pinned vertices to their targets, at rest.
__device__ __forceinline__ void na_pins(const NaArgs& a, int gtid, int gstride)
{
    for (int q = gtid; q < a.P; q += gstride) {
        const int i = a.pin_idx[q];
        a.pos[3 * i] = a.pin_target[3 * q]; a.pos[3 * i + 1] = a.pin_target[3 * q + 1]; a.pos[3 * i + 2] = a.pin_target[3 * q + 2];
        a.vel[3 * i] = 0.f; a.vel[3 * i + 1] = 0.f; a.vel[3 * i + 2] = 0.f;
    }
}

// Prediction y of vertex i and its offset at the inertial start (d.w: 1 /
// diagonal).
__device__ __forceinline__ float4 na_predict(const NaArgs& a, int i, float4& d0)
{
    const float h = a.h, h2 = fmul(h, h);
    const float dg = a.diag[i];
    d0 = make_float4(0.f, 0.f, 0.f, dg > 1e-10f ? 1.0f / dg : 0.f);
    float4 y;
    y.x = ffma(h2, a.ax, ffma(h, a.vel[3 * i], a.pos[3 * i]));
    y.y = ffma(h2, a.ay, ffma(h, a.vel[3 * i + 1], a.pos[3 * i + 1]));
    y.z = ffma(h2, a.az, ffma(h, a.vel[3 * i + 2], a.pos[3 * i + 2]));
    y.w = a.mass[i];
    return y;
}

// Offset of pin q's vertex, whose prediction is y.
__device__ __forceinline__ float4 na_pin_offset(const NaArgs& a, int q, float4 y)
{
    return make_float4(fsub(a.pin_target[3 * q], y.x), fsub(a.pin_target[3 * q + 1], y.y),
                       fsub(a.pin_target[3 * q + 2], y.z), -1.f);
}

// The frame at any size, two barriers per sweep: threads may have several
// elements and vertices.  Two 512-thread blocks per SM at 64 registers.  y and
// d of a vertex lie in one 32-byte pair (the arrays Y and A as one), which an
// element reads through L1: in two arrays read from L2 32 sweeps of a 257x257
// cloth took 505 us, now 424; 360x360 738, now 615.  What bounds it is the
// reductions and corner reads in L2 (327,000 elements a sweep at 257x257).
// Each thread keeps its first vertex's mass, prediction and last two offsets.
__global__ void __launch_bounds__(kNaThreads, 2) k_na_frame(NaArgs a)
{
    __shared__ int status_s;
    const Scratch s = a.s;
    float4* YD = s.Y;
    const int gtid = blockIdx.x * kNaThreads + threadIdx.x, gstride = gridDim.x * kNaThreads;
    const int nsweep = a.cap + a.have_final;
    const bool has_own = (int)(blockIdx.x * kNaThreads) < a.N;
    unsigned phase = 0;

    // prediction, start offsets, cleared sums
    for (int i = gtid; i < a.cap + 2; i += gstride) s.acc[i] = 0.0;
    for (int i = gtid; i < a.N; i += gstride) {
        float4 d0;
        YD[2 * i] = na_predict(a, i, d0);
        YD[2 * i + 1] = d0;
        s.B[i] = d0;
        s.F[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!na_barrier(s.ctl, phase)) return;
    if (a.P > 0) {
        for (int q = gtid; q < a.P; q += gstride) {
            const int i = a.pin_idx[q];
            const float4 d = na_pin_offset(a, q, YD[2 * i]);
            YD[2 * i + 1] = d;
            s.B[i] = d;
        }
        if (!na_barrier(s.ctl, phase)) return;
    }

    float4 vd = make_float4(0.f, 0.f, 0.f, 0.f), vp = vd, vy = vd;   // vertex gtid: d^k, d^(k-1), y
    if (gtid < a.N) { vy = YD[2 * gtid]; vd = YD[2 * gtid + 1]; vp = vd; }

    int nstop = -1;
    float om = 1.f;
    for (int k = 0; k < nsweep; ++k) {
        const bool res_only = k >= a.cap;
        if (!res_only) om = na_omega(a, k, om);
        for (long long q = gtid; q < (long long)a.T + a.E; q += gstride) {
            const NaElem m = na_element<2>(a, q);
            const float4 d0 = YD[2 * m.i0 + 1];
            na_apply(m, d0, YD[2 * m.i1 + 1], YD[2 * m.i2 + 1], m.i3 >= 0 ? YD[2 * m.i3 + 1] : d0, s.F);
        }
        if (!na_barrier(s.ctl, phase)) return;
        // vertices; the accumulator is left clear for the next sweep
        float r2 = 0.f;
        for (int i = gtid; i < a.N; i += gstride) {
            const bool first = i == gtid;
            const float4 f4 = s.F[i];
            const float4 d = first ? vd : YD[2 * i + 1], y = first ? vy : YD[2 * i];
            const float4 dp = res_only ? d : (first ? vp : s.B[i]);
            float rv;
            const float4 o = update_consistent(d, y, make_float3(f4.x, f4.y, f4.z), dp, a.gamma, res_only ? 1.f : om, rv);
            r2 += rv;
            s.F[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (res_only) continue;
            YD[2 * i + 1] = o;
            if (first) { vp = d; vd = o; } else s.B[i] = d;
        }
        int done;
        if (!na_end_sweep<kNaThreads>(a, phase, k, k + 1 == nsweep, has_own, r2, done)) return;
        if (done) { nstop = k; break; }
    }

    if (threadIdx.x < 32) na_outcome(a, nstop, status_s);
    __syncthreads();
    // (stopped after sweep k: d^k, which the sweep's update moved on from)
    for (int i = gtid; i < a.N; i += gstride) {
        const bool first = i == gtid;
        const float4 d = first ? (nstop >= 0 ? vp : vd) : (nstop >= 0 ? s.B[i] : YD[2 * i + 1]);
        if (d.w >= 0.f) na_finalize(a, i, first ? vy : YD[2 * i], f3(d), status_s);   // (pinned: below)
    }
    na_pins(a, gtid, gstride);
}

// The frame where no thread has more than one element or vertex: a sweep then
// takes one grid barrier.  Each thread keeps its element's constants and its
// corners' last two offsets in registers and forms the corners' updates itself
// from the summed forces, as every other element at that corner does with the
// same operations; the force sums rotate through three arrays (the one read,
// the one added to, the one being cleared).  Phase p evaluates the forces at
// d^p after taking the update of sweep p - 1; thread i < N also takes vertex i,
// for the residual, the cleared sum and the frame's end.
// With the corners' offsets read back from memory a sweep took two barriers
// and two more trips to L2: 32 sweeps of a 129x129 cloth 220 us, now 141;
// 100x100 195 us, now 125; 9x9 144 us, now 83.  (The sums are read through L1,
// which the barrier's acquiring load empties: 141 us, from L2 145.)
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_na_one(NaArgs a)
{
    __shared__ int status_s;
    const Scratch s = a.s;
    NaCtl* ctl = s.ctl;
    const int gtid = blockIdx.x * NT + threadIdx.x;
    const int nsweep = a.cap + a.have_final;
    const bool own = gtid < a.N, elem = gtid < a.T + a.E, has_own = (int)(blockIdx.x * NT) < a.N;
    unsigned phase = 0;

    // prediction, start offsets (A), cleared sums
    if (gtid < a.cap + 2) s.acc[gtid] = 0.0;
    for (int i = gtid + (int)gridDim.x * NT; i < a.cap + 2; i += (int)gridDim.x * NT) s.acc[i] = 0.0;
    float4 vy = make_float4(0.f, 0.f, 0.f, 0.f), vd = vy;   // vertex gtid: y, d^k
    if (own) {
        vy = na_predict(a, gtid, vd);
        s.Y[gtid] = vy;
        s.A[gtid] = vd;
        s.F[gtid] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!na_barrier(ctl, phase)) return;
    if (a.P > 0) {
        for (int q = gtid; q < a.P; q += (int)gridDim.x * NT) {
            const int i = a.pin_idx[q];
            s.A[i] = na_pin_offset(a, q, s.Y[i]);
        }
        if (!na_barrier(ctl, phase)) return;
    }

    NaElem el;
    float4 cd[4];            // corners: d^k, 1 / diagonal (pinned: -1)
    float3 cp[4];            // d^(k-1)
    float cm[4];             // mass
    if (elem) {
        el = na_element<1>(a, gtid);
        const int id[4] = {el.i0, el.i1, el.i2, el.i3 >= 0 ? el.i3 : el.i0};
        #pragma unroll
        for (int c = 0; c < 4; ++c) {
            cd[c] = s.A[id[c]];
            cp[c] = f3(cd[c]);
            cm[c] = s.Y[id[c]].w;
        }
    }
    if (own) vd = s.A[gtid];
    float3 vp = f3(vd);

    // Y is not read again: the third array of the rotation
    float4 *fr = s.Y, *fw = s.F, *fc = s.B;   // read, add to, clear
    float om = 1.f;
    int nstop = -1;
    for (int p = 0; p <= nsweep; ++p) {
        const int k = p - 1;   // the sweep whose update is taken
        float r2 = 0.f;
        if (p > 0) {
            const bool res_only = k >= a.cap;
            if (!res_only) om = na_omega(a, k, om);
            const float w = res_only ? 1.f : om;
            auto update = [&](float4& d, float3& dp, float m, float4 f, float& rv) {
                const float4 dq = res_only ? d : make_float4(dp.x, dp.y, dp.z, 0.f);
                const float4 o = update_consistent(d, make_float4(0.f, 0.f, 0.f, m), f3(f), dq, a.gamma, w, rv);
                if (!res_only) { dp = f3(d); d = o; }
            };
            if (elem && p < nsweep) {
                const float4 f0 = fr[el.i0], f1 = fr[el.i1], f2 = fr[el.i2];
                const float4 f3_ = el.i3 >= 0 ? fr[el.i3] : f0;
                float rv;
                update(cd[0], cp[0], cm[0], f0, rv);
                update(cd[1], cp[1], cm[1], f1, rv);
                update(cd[2], cp[2], cm[2], f2, rv);
                update(cd[3], cp[3], cm[3], f3_, rv);
            }
            if (own) update(vd, vp, vy.w, fr[gtid], r2);
        }
        if (p < nsweep) {
            if (elem) na_apply(el, cd[0], cd[1], cd[2], cd[3], fw);
            if (own) fc[gtid] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        int done;
        if (!na_end_sweep<NT>(a, phase, k, p == nsweep, has_own, r2, done)) return;
        if (done) { nstop = k; break; }
        float4* t = fr; fr = fw; fw = fc; fc = t;
    }

    if (threadIdx.x < 32) na_outcome(a, nstop, status_s);
    __syncthreads();
    if (own && vd.w >= 0.f) na_finalize(a, gtid, vy, nstop >= 0 ? vp : f3(vd), status_s);   // (pinned: below)
    na_pins(a, gtid, (int)gridDim.x * NT);
}

// Device address of the scratch array, looked up once per device.
std::mutex g_mu;
unsigned char* g_addr[64] = {};
int g_blocks[64] = {};   // blocks of k_na_frame resident at once (of k_na_one: one per SM)
int g_sms[64] = {};

int scratch_of(int dev, unsigned char** out, int* blocks, int* sms)
{
    if (dev < 0 || dev >= 64) return set_error(PDG_ERR_ARG, "pdg_step_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return set_error(PDG_ERR_CUDA, "pdg_step_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        int nsm = 0, per = 0;
        if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_na_frame, kNaThreads, 0) != cudaSuccess || per <= 0)
            return set_error(PDG_ERR_CUDA, "pdg_step_noalloc: occupancy query failed");
        g_blocks[dev] = nsm * per;
        g_sms[dev] = nsm;
        g_addr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_addr[dev];
    *blocks = g_blocks[dev];
    *sms = g_sms[dev];
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
    int max_blocks = 0, nsm = 0;
    const int rc = scratch_of(dev, &base, &max_blocks, &nsm);
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
    const long long work = std::max((long long)T + E, (long long)N);
    NA_CK(cudaMemsetAsync(a.s.ctl, 0, sizeof(NaCtl), st));
    void* args[] = {&a};
    // One block per SM, of the fewest threads that give each element and vertex
    // its own: a barrier waits for few arrivals and a block's barrier for few
    // warps.  Measured beside one another, 32 sweeps of a 33x33 cloth take 97 us in blocks of 128 threads,
    // 139 of 640; 100x100 134 us in blocks of 512 (one per SM), 135 of 256 and
    // 140 of 128 (two and four per SM); 129x129 156 us in blocks of 640, 160
    // of 320 and 192 of 128.
    struct { int nt; const void* kernel; } const one[] = {
        {128, (const void*)k_na_one<128>}, {256, (const void*)k_na_one<256>}, {512, (const void*)k_na_one<512>},
        {640, (const void*)k_na_one<640>}, {768, (const void*)k_na_one<768>}, {1024, (const void*)k_na_one<1024>}};
    int nt = kNaThreads, blocks = max_blocks;
    const void* kernel = (const void*)k_na_frame;
    for (const auto& o : one)
        if (work <= (long long)nsm * o.nt) { nt = o.nt; blocks = nsm; kernel = o.kernel; break; }
    const int grid = (int)std::min((long long)blocks, (work + nt - 1) / nt);
    NA_CK(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(nt), args, 0, st));

    if (stats) {
        NaCtl c;
        NA_CK(cudaMemcpyAsync(&c, a.s.ctl, sizeof(NaCtl), cudaMemcpyDeviceToHost, st));
        NA_CK(cudaStreamSynchronize(st));
        if (c.bar & kNaGaveUp)
            return set_error(PDG_ERR_TIMEOUT, "pdg_step_noalloc: bounded wait ran out (grid barrier)");
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
