// Resident persistent PD kernel: one cooperative launch per frame, one patch
// per block for the whole frame.  The patch's cell and hinge records, the
// hinges' slot addresses, the gather pointers, y and d^k live in shared
// memory (vertex-major contribution slots, as in the per-sweep kernels), and
// each thread keeps its owned vertex's previous offset d^(k-1) in a register.  Per sweep only the owned
// offsets go out to L2 and the halo offsets come back.
//
// Synchronisation between sweeps: with fixed sweep counts a block waits only
// for the halo offsets it reads.  Each boundary vertex publishes d^(k+1) as
// three 64-bit words, value bits | tag << 32, with the tag naming the frame
// and the sweep; a reader polls the words of its halo vertices until all
// three carry the tag it expects, so the data itself is the completion flag
// (one write and one read per exchange, no separate mark and no fence).
// With a residual tolerance (the TOL instance) the sweeps run the same way, and
// the convergence decision lags: a spare warp adds the block's residual of
// sweep k while the others go on, and before sweep k + 2 the block reads the
// complete sum of sweep k.  If the cloth stops there, its vertices step back to
// d^k, which each thread still holds.  (A grid barrier per sweep, which the
// complete sum of the last sweep would need, made a 129x129 sweep 5.7 us.)
// Every wait is bounded by a clock64 budget; on expiry the block records an
// error code and leaves, and so do all others at their next wait.
//
// Used when every patch fits one block (nown <= NT) and all patches are
// co-resident.
//
// The instance with IO = true also moves the caller's state for the
// host-buffer frame (pdg_solver_step_host): it reads x and v from the caller's
// arrays for the prediction and writes them back after the finalisation, both
// walked in caller order so that page-locked host memory is accessed
// contiguously, which replaces the two copy launches around the frame.
#include "pd_kernels.cuh"
#include "pdg_kernels.h"

namespace pdg {

// Barrier over the grid on a 64-bit count of arrivals that is never reset:
// every barrier adds gridDim.x, so a block's own arrival number tells which
// count ends its barrier.  False once a wait, here or in another block, gave
// up (the host then clears the count when it reports the error).
__device__ __forceinline__ bool grid_barrier_r(unsigned* bar, int* err, long long budget)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* cnt = reinterpret_cast<unsigned long long*>(bar);
        __threadfence();
        const unsigned long long old = atomicAdd(cnt, 1ull);
        const unsigned long long want = (old / gridDim.x + 1ull) * gridDim.x;
        unsigned long long v = old + 1ull;
        if (v < want) {
            const long long t0 = clock64();
            do {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(__cvta_generic_to_global(cnt)) : "memory");
                if (v < want && (clock64() - t0 > budget || *(volatile int*)err != 0)) { atomicCAS(err, 0, 2); break; }
            } while (v < want);
        }
        __threadfence();
        ok = (v >= want && *(volatile int*)err == 0);
    }
    __syncthreads();
    return ok != 0;
}

// Caller vertex o of an AoS xyz array, or zeros without one.
__device__ __forceinline__ float3 caller_vec(const float* a, int o)
{
    return a ? make_float3(a[3 * o], a[3 * o + 1], a[3 * o + 2]) : make_float3(0.f, 0.f, 0.f);
}

// Predicts layout vertex g from the caller's x and v (xi, vi: its entries in
// the caller's arrays), which replace the solver's state as the scatter copy
// before a frame would have.
__device__ __forceinline__ void predict_caller_vertex(const PersistArgs& p, int g, float3 xi, float3 vi)
{
    const float4 x = p.in_x ? make_float4(xi.x, xi.y, xi.z, 0.f) : __ldcg(&p.X[g]);
    const float4 v = p.in_v ? make_float4(vi.x, vi.y, vi.z, 0.f) : __ldcg(&p.V[g]);
    if (p.in_x) p.Xw[g] = x;
    if (p.in_v) p.V[g] = v;
    predict_vertex_xv(g, x, v, p.aux, p.mass, p.vcloth, p.it.cinfo, p.warm, p.Y, p.it.buf[0], p.it.buf[1]);
}

// Layout vertex g's state into the caller's arrays at caller vertex o (the
// gather copy after a frame).
__device__ __forceinline__ void store_frame_state(const PersistArgs& p, int o, int g)
{
    if (p.out_x) {
        const float4 x = __ldcg(&p.Xw[g]);
        p.out_x[3 * o] = x.x; p.out_x[3 * o + 1] = x.y; p.out_x[3 * o + 2] = x.z;
    }
    if (p.out_v) {
        const float4 v = __ldcg(&p.V[g]);
        p.out_v[3 * o] = v.x; p.out_v[3 * o + 1] = v.y; p.out_v[3 * o + 2] = v.z;
    }
}

// Named barriers (barrier 0 is __syncthreads).  `count` threads, a multiple
// of 32, take part.
__device__ __forceinline__ void named_sync(int id, int count)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// Arrival without waiting (the waiting side uses named_sync).
__device__ __forceinline__ void named_arrive(int id, int count)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// named_sync that also returns whether `v` held on every taking part thread.
__device__ __forceinline__ bool named_and(int id, int count, bool v)
{
    unsigned r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                 "barrier.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r)
                 : "r"((unsigned)v), "r"(id), "r"(count)
                 : "memory");
    return r != 0;
}

// Tagged exchange of one vertex offset: each component is one 64-bit word
// (value bits | tag << 32).  A 64-bit access is single-copy atomic, so a
// reader that finds `tag` in all three words holds the value written with
// it; the words are read and written at GPU scope, bypassing L1.
__device__ __forceinline__ void st_tagged(unsigned long long* w, float4 o, unsigned tag)
{
    const unsigned long long t = (unsigned long long)tag << 32;
    const unsigned long long a = t | __float_as_uint(o.x), b = t | __float_as_uint(o.y), c = t | __float_as_uint(o.z);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(a), "l"(b) : "memory");
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w + 2), "l"(c) : "memory");
}

// Reads the words of one vertex; true (and v.xyz set) when all carry `tag`.
__device__ __forceinline__ bool ld_tagged(const unsigned long long* w, unsigned tag, float4& v)
{
    unsigned long long a, b, c;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(w + 2) : "memory");
    if ((unsigned)(a >> 32) != tag || (unsigned)(b >> 32) != tag || (unsigned)(c >> 32) != tag) return false;
    v.x = __uint_as_float((unsigned)a);
    v.y = __uint_as_float((unsigned)b);
    v.z = __uint_as_float((unsigned)c);
    return true;
}

// The three words of one vertex, read once (no tag check).
__device__ __forceinline__ void ld_words(const unsigned long long* w, unsigned long long& a, unsigned long long& b,
                                         unsigned long long& c)
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(c) : "l"(w + 2) : "memory");
}

// Polls one vertex's words until they carry `tag`, bounded by the clock64
// budget; false on timeout or when another block reported an error.
__device__ __forceinline__ bool poll_tagged(const unsigned long long* w, unsigned tag, float4& v, int* err,
                                            long long budget)
{
    if (ld_tagged(w, tag, v)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (ld_tagged(w, tag, v)) return true;
        if (clock64() - t0 > budget || *(volatile int*)err != 0) {
            atomicCAS(err, 0, 3);
            return false;
        }
    }
}

constexpr int kResOmega = 1024;   // Chebyshev weights kept in shared memory

// Local step over the records with list index in [t0, t1) (cells) and
// [e0, e1) (lone hinges), read from the patch's copy in shared memory.  With
// `rev` the records go to the threads in reverse order (the last thread takes
// the first record), which leaves the first threads free; a record's
// contributions and slots do not depend on the thread that computes them.
template <int MODE, int NT>
__device__ __forceinline__ void local_records(const CellRec* rc, const HingeRec* rh, const uint2* hvs,
                                              const float4* sy, const float4* sd, int ncell, int nhin, int t0, int t1,
                                              int e0, int e1, float2* cxy, float* cz, bool rev = false)
{
    const int j0 = rev ? NT - 1 - (int)threadIdx.x : (int)threadIdx.x;
    for (int t = t0 + j0; t < t1; t += NT) cell_contrib_vm_p<MODE>(rc[t], sy, sd, cxy, cz);
    for (int e = e0 + j0; e < e1; e += NT) hinge_contrib_vm<MODE>(rh[e], hvs[e], sy, sd, cxy, cz);
}

// Jacobi update of owned vertex l with force f: o = d^(k+1), d = d^k.
template <int MODE>
__device__ __forceinline__ void vertex_update_f(float3 f, int l, const float4* sy, const float4* sd, float4 dprev,
                                                float gamma, float omega, float4& o, float4& d, float& r2)
{
    d = sd[l];
    const float4 y = sy[l];
    if (MODE == kModeConsistent) o = update_consistent(d, y, f, dprev, gamma, omega, r2);
    else                         o = update_literal(d, y, f);
}

// Gather by one thread and update.
template <int MODE>
__device__ __forceinline__ void vertex_update(int npad, const int* sptr, int l, const float4* sy,
                                              const float4* sd, const float2* cxy, const float* cz,
                                              float4 dprev, float gamma, float omega, float4& o, float4& d, float& r2)
{
    const int deg = sptr[l + 1] - sptr[l], h = gather_half(deg);
    const float3 f = deg <= 10 ? fadd3(gather_vm_u<5>(l, 0, h, npad, cxy, cz), gather_vm_u<5>(l, h, deg, npad, cxy, cz))
                               : fadd3(gather_vm(l, 0, h, npad, cxy, cz), gather_vm(l, h, deg, npad, cxy, cz));
    vertex_update_f<MODE>(f, l, sy, sd, dprev, gamma, omega, o, d, r2);
}

// Block sum of r2 over the NT compute threads (named barrier 1), added to
// *acc by one double atomic.
template <int NT>
__device__ __forceinline__ void compute_residual(float r2, float* red, double* acc)
{
    const int tid = threadIdx.x;
    r2 = warp_sum(r2);
    if ((tid & 31) == 0) red[tid >> 5] = r2;
    named_sync(1, NT);
    if (tid < 32) {
        float v = tid < NT / 32 ? red[tid] : 0.f;
        v = warp_sum(v);
        if (tid == 0) atomicAdd(acc, (double)v);
    }
}

// Block layout: NT compute threads (thread l < nown owns local vertex l;
// the patch's records in shared memory) and one more warp that helps stage
// the records at the start of the frame.  In the TOL instance that warp adds
// the residuals and takes the decisions; otherwise it only takes part in the
// block-wide barriers.  (It was the signal warp of a completion-mark
// protocol, which the tagged exchange replaced: 257x257 sweep 5.5 -> 4.7 us,
// 33x33 4.8 -> 4.3 us, bitwise equal.)
//
// One sweep of the compute threads:
//   [k > 0: poll the halo's tagged d^k words into shared memory] -> bar 1
//   (a vote: a failed poll makes every compute thread leave the sweep loop)
//   -> phase A records -> bar 1 -> update of the boundary vertices (d^(k+1)
//   to global memory and as tagged words) -> phase B records -> bar 1 ->
//   [first read of the next sweep's halo words] -> interior update.
// Barrier 1 counts the NT compute threads.  TOL: before the vote of sweep
// k >= 2 the compute threads take the spare warp's decision about sweep k - 2
// (barrier 4 + (k & 1)), after sweep k they hand it their partial sums
// (barrier 2 + (k & 1)).  Two of each, so that neither side can arrive twice
// at a barrier that the other has not left.
// IO: the instance that also moves the caller's state (p.in_x ... p.out_v);
// the other one compiles without that code.
// RANGE (with TOL): sweeps p.k0 .. p.k1 - 1 of a frame whose prediction, start
// and finalisation are other launches: the streaming plan's sweeps where its
// patches all fit on the chip at once.  At 54,000 vertices in 128-vertex
// patches a sweep takes 3.7 us, as launches of the streaming kernel 7.3 us.
template <int MODE, int NT, bool IO, bool TOL, bool RANGE>
__global__ void __launch_bounds__(NT + 32, 512 / (NT + 32)) k_resident(PersistArgs p)
{
    static_assert(!RANGE || (TOL && !IO), "ranges take decisions and move no caller state");
    constexpr int NTT = NT + 32;   // 512 and 256: 4 warps per SM sub-partition
    extern __shared__ float4 smem[];
    __shared__ PatchHdr ph;
    __shared__ float red[TOL ? 2 : 1][NTT / 32];
    __shared__ int dec[2];             // TOL: decision, 0 go on, 1 stop, 2 leave (a wait ran out)
    __shared__ int gone;               // TOL: the compute threads left early
    __shared__ int over;               // RANGE: the cloth is done before the range
    __shared__ FrameEnd end_s;         // outcome of this cloth's frame; TOL: set early when it stops
    __shared__ int stopped;            // TOL: it did
    __shared__ float som[kResOmega];   // Chebyshev weights of this cloth
    const IterArgs& a = p.it;
    const int tid = threadIdx.x;
    const bool comp = tid < NT;
    // With caller arrays, this thread's first caller vertex is loaded before
    // the patch's records are staged: the host round trip overlaps the staging.
    const bool caller_in = IO && (p.in_x || p.in_v), caller_out = IO && (p.out_x || p.out_v);
    const int o0 = (int)blockIdx.x * NT + tid;
    float3 xi0 = make_float3(0.f, 0.f, 0.f), vi0 = xi0;
    int gi0 = 0;
    if (caller_in && comp && o0 < p.n) {
        gi0 = __ldg(&p.io_inv[o0]);
        xi0 = caller_vec(p.in_x, o0);
        vi0 = caller_vec(p.in_v, o0);
    }
    if (tid == 0) ph = a.patches[blockIdx.x];
    __syncthreads();
    const int nown = ph.nown, nlocal = ph.nlocal, ncell = ph.ncell, nhin = ph.nhinge;
    // shared memory: the patch's records (read every sweep), the hinges' slot
    // addresses, y and d of the local vertices, the vertex-major contribution
    // slots and the gather pointers
    CellRec* rc = reinterpret_cast<CellRec*>(smem);
    HingeRec* rh = reinterpret_cast<HingeRec*>(rc + ncell);
    uint2* hvs = reinterpret_cast<uint2*>(rh + nhin);
    float4* sy = reinterpret_cast<float4*>(hvs + ((nhin + 1) & ~1));
    float4* sd = sy + nlocal;
    float2* cxy = reinterpret_cast<float2*>(sd + nlocal);
    float* cz = reinterpret_cast<float*>(cxy + ph.vm_nslot);
    int* sptr = reinterpret_cast<int*>(cz + ph.vm_nslot);
    const int npad = ph.vm_npad;

    {
        // records from the device format (groups of kCellGroup, piece-major),
        // read in that order, into shared memory record after record
        const uint4* src = reinterpret_cast<const uint4*>(a.cells + ph.cell_off);
        uint4* dst = reinterpret_cast<uint4*>(rc);
        const int n4 = (ncell + kCellGroup - 1) / kCellGroup * (9 * kCellGroup);
        for (int q = tid; q < n4; q += NTT) {
            const int grp = q / (9 * kCellGroup), r = q - grp * (9 * kCellGroup);
            const int i = r / kCellGroup, cc = grp * kCellGroup + r % kCellGroup;
            if (cc < ncell) dst[cc * 9 + i] = __ldg(&src[q]);
        }
        const uint4* hsrc = reinterpret_cast<const uint4*>(a.hinges + ph.hinge_off);
        uint4* hdst = reinterpret_cast<uint4*>(rh);
        for (int q = tid; q < 2 * nhin; q += NTT) hdst[q] = __ldg(&hsrc[q]);
        for (int q = tid; q < nhin; q += NTT) hvs[q] = __ldg(&a.hvm[ph.hinge_off + q]);
    }
    // gather pointers (per-vertex contribution counts) and Chebyshev weights
    for (int l = tid; l <= nown; l += NTT) sptr[l] = a.csr_ptr[ph.csr_off + l];
    for (int k = tid; k < a.omega_stride && k < kResOmega; k += NTT) som[k] = a.omega[ph.cloth * a.omega_stride + k];
    __syncthreads();


    // predict the owned vertices, or with caller arrays the vertices in caller
    // order (a grid-stride walk over the compute threads); the cloth's first
    // block resets its record
    const int c = ph.cloth;
    const ClothInfo& ci = a.cinfo[c];
    const bool own = tid < nown;
    const bool first = (int)blockIdx.x == ci.patch_begin;
    const int g = ph.vbegin + tid;
    float4 dprev = make_float4(0.f, 0.f, 0.f, 0.f);
    const int k0 = RANGE ? p.k0 : 0;   // first sweep
    // The per-sweep sums and arrivals of a whole frame come in two sets: a
    // frame uses the one that p.frame's parity names and clears the other, so
    // that no block needs to wait for the clearing.  Frames with fixed sweep
    // counts have no arrivals but clear them too (in the spare warp, below):
    // the frame that uses the set next may have a tolerance.  (A range uses
    // the sums that the frame's first launch cleared.)
    const unsigned par = RANGE ? 0u : __ldcg(p.frame) & 1u;
    const size_t set = (size_t)a.ncloth * a.acc_stride;
    double* acc = a.acc + (RANGE ? 0 : par * set) + (size_t)c * a.acc_stride;
    int* cnt = TOL ? p.cnt + par * set + (size_t)c * a.acc_stride : nullptr;
    if (first) {
        if (!RANGE && tid == 0) {
            ClothRT r;
            r.active = 1; r.used = 0; r.status = 0; r.warm = 0;
            r.res_y2 = 0.0; r.res0_2 = 0.0; r.resf_2 = -1.0;
            a.crt[c] = r;
        }
        for (int k = tid; k < a.acc_stride; k += NTT) {
            if (!RANGE) a.acc[(par ^ 1u) * set + (size_t)c * a.acc_stride + k] = 0.0;
            if (TOL) p.cnt[(RANGE ? 0u : par ^ 1u) * set + (size_t)c * a.acc_stride + k] = 0;
        }
    }
    if (TOL && tid == 0) { gone = 0; stopped = 0; }
    // The frame's exchange tags: tag0 + k for d^k, tag0 from the device word
    // that the previous frame advanced (so a replayed launch gets new tags).
    // Before the 32-bit tags would wrap, every block clears its boundary
    // vertices' words in both buffers and the frame starts again from 0, after
    // a grid barrier that orders the clearing before any neighbour's poll.
    const int nsweep = RANGE ? p.k1 : p.max_iter + (p.have_final ? 1 : 0);   // end of the sweeps
    unsigned tag0 = __ldcg(p.xch_tag);
    const bool wrap = (unsigned long long)tag0 + (unsigned long long)nsweep > 0xffffffffULL;
    if (wrap) {
        tag0 = 0;
        for (int q = tid; q < 8 * ph.nbnd; q += NTT) {
            const int l = q >> 3, b = (q >> 2) & 1, w = q & 3;
            p.xch[((size_t)b * (size_t)p.n + (size_t)(ph.vbegin + l)) * 4 + w] = 0ull;
        }
    }
    // Prediction.  A block predicts its halo vertices too: the state is not
    // written before every block has met the barrier after the sweeps, so no
    // block waits for another's prediction.  (With a barrier after the owners'
    // prediction, and one more between the record and the finalisation, a
    // 33x33 frame of 10 sweeps took 43.0 us, now 36.9.)  With caller arrays
    // the vertices are walked in caller order, a grid stride over the compute
    // threads, and the halo is read after a barrier.
    if (RANGE) {
        // the decision about the sweep before the range, the same in every
        // block of the cloth; all have taken it when the barrier below opens
        if (tid == 0) over = cloth_done(a, c, k0, first, true) ? 1 : 0;
        if (own) dprev = __ldcg(&((k0 & 1) ? a.buf[0] : a.buf[1])[g]);
    } else if (caller_in) {
        if (comp && o0 < p.n) predict_caller_vertex(p, gi0, xi0, vi0);
        for (int o = o0 + (int)gridDim.x * NT; comp && o < p.n; o += (int)gridDim.x * NT)
            predict_caller_vertex(p, __ldg(&p.io_inv[o]), caller_vec(p.in_x, o), caller_vec(p.in_v, o));
    } else {
        for (int l = tid; l < nlocal; l += NTT) {
            const int gg = l < nown ? ph.vbegin + l : __ldg(&a.halo[ph.halo_off + l - nown]);
            float4 y, s;
            predict_values(__ldcg(&p.X[gg]), __ldcg(&p.V[gg]), __ldcg(&p.aux[gg]), __ldg(&p.mass[gg]), ci, p.warm, gg, y, s);
            sy[l] = y;
            sd[l] = s;
            if (l < nown) {
                p.Y[gg] = y;
                a.buf[0][gg] = s;
                a.buf[1][gg] = s;
                if (l == tid) dprev = s;
            }
        }
    }
    if ((RANGE || caller_in || wrap) && !grid_barrier_r(p.bar, p.err, p.spin_budget)) return;
    if (RANGE || caller_in) {
        // (the barrier: every block of a range has read the tag word)
        if (RANGE && blockIdx.x == 0 && tid == 0) *p.xch_tag = tag0 + (unsigned)nsweep;
        if (caller_in && own) dprev = __ldcg(&a.buf[0][g]);
        for (int l = tid; l < nlocal; l += NTT) {
            const int gg = l < nown ? ph.vbegin + l : __ldg(&a.halo[ph.halo_off + l - nown]);
            sy[l] = __ldcg(&a.Y[gg]);
            sd[l] = __ldcg(&(RANGE && (k0 & 1) ? a.buf[1] : a.buf[0])[gg]);
        }
    }
    // this compute thread's first halo vertex, re-read every sweep
    const int hl0 = nown + tid;
    const int hg0 = (comp && hl0 < nlocal) ? __ldg(&a.halo[ph.halo_off + tid]) : 0;
    __syncthreads();

    const float gamma = ci.gamma;
    // TOL: kept in a register, because the acquiring loads of the spare warp
    // empty L1 and the reloads would miss it (129x129 to a tolerance 597 ->
    // 520 us per 200 sweeps).  Otherwise the reloads hit, and the instances
    // with the register were slower (65x65 111 -> 123 us per 50 sweeps).
    const int max_iter_r = TOL ? ci.max_iter : 0;
    auto max_iter = [&]() { return TOL ? max_iter_r : ci.max_iter; };
    // TOL: the end of this cloth's sweeps
    const int kend = RANGE && over ? k0 : min(nsweep, max_iter() + 1);
    if (comp) {
        // ---- compute threads ----
        float4 dpp = make_float4(0.f, 0.f, 0.f, 0.f);   // TOL: own d^(k-2)
        bool left = false;
        // the words of this thread's first halo vertex for the next sweep, read
        // ahead while the interior is updated: when they already carry the
        // tag the top of the next sweep needs no round trip (257x257 sweep
        // 4.72 -> 4.60 us; read before phase B instead: 4.76 us)
        unsigned long long pw0 = 0, pw1 = 0, pw2 = 0;
        // A patch whose records all fit one round of the threads computes them
        // together: one local step and barrier less on the sweep's chain.
        const bool one_phase = ncell + nhin <= NT;
        const int na = one_phase ? ncell : ph.ncell_a, nha = one_phase ? nhin : ph.nhin_a;
        for (int k = k0; k < (TOL ? kend : nsweep); ++k) {
            if (TOL && k >= k0 + 2) {
                named_sync(4 + (k & 1), NTT);
                const int go = dec[k & 1];
                if (go) {
                    // the cloth stops at d^(k-2), or a wait ran out
                    if (go == 1 && own) ((k & 1) ? a.buf[1] : a.buf[0])[g] = dpp;
                    left = true;
                    break;
                }
            }
            if (k > k0 && k <= max_iter()) {
                // the neighbours' d^k (written in their sweep k - 1, which
                // every sweep up to the cloth's cap has): poll the tagged
                // words of this thread's halo vertices
                const unsigned tag = tag0 + (unsigned)k;
                const unsigned long long* xb = p.xch + (size_t)(k & 1) * (size_t)p.n * 4;
                bool ok = true;
                for (int l = hl0; ok && l < nlocal; l += NT) {
                    const int gg = l == hl0 ? hg0 : __ldg(&a.halo[ph.halo_off + l - nown]);
                    float4 v = sd[l];
                    if (l == hl0 && (unsigned)(pw0 >> 32) == tag && (unsigned)(pw1 >> 32) == tag &&
                        (unsigned)(pw2 >> 32) == tag) {
                        v.x = __uint_as_float((unsigned)pw0);
                        v.y = __uint_as_float((unsigned)pw1);
                        v.z = __uint_as_float((unsigned)pw2);
                    } else {
                        ok = poll_tagged(xb + (size_t)gg * 4, tag, v, p.err, p.spin_budget);
                    }
                    sd[l] = v;
                }
                if (!named_and(1, NT, ok)) {   // the grid barrier below reports the error
                    if (TOL) {
                        if (tid == 0) gone = 1;
                        named_arrive(2 + (k & 1), NTT);
                        left = true;
                    }
                    break;
                }
            } else {
                named_sync(1, NT);
            }
            // the cap alone decides: the cloth's record stays active through the sweeps
            const bool skip_k = k >= max_iter() && (k > max_iter() || !a.have_final);
            const float omega_k =
                k < a.omega_stride ? (k < kResOmega ? som[k] : a.omega[c * a.omega_stride + k]) : 1.f;
            const bool res_only = k >= max_iter();
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f), d = o;
            float r2 = 0.f;
            // Phase A: the records through boundary vertices (a prefix of
            // each list), then the boundary vertices, which the neighbouring
            // patches read: their tagged words go out before phase B runs.
            if (!skip_k)
                local_records<MODE, NT>(rc, rh, hvs, sy, sd, ncell, nhin, 0, na, 0, nha, cxy, cz);
            named_sync(1, NT);
            // The boundary vertices' sums are on the neighbours' critical path:
            // one thread per vertex, every slot load issued before the
            // additions.  (Splitting each sum over an owner and a helper
            // thread joined by a named barrier, the two halves of its
            // definition, was slower once the loads were hoisted.)
            if (!skip_k && tid < ph.nbnd) {
                vertex_update<MODE>(npad, sptr, tid, sy, sd, cxy, cz, dprev, gamma, omega_k, o, d, r2);
                if (!res_only) {
                    ((k & 1) ? a.buf[0] : a.buf[1])[g] = o;
                    st_tagged(p.xch + ((size_t)((k + 1) & 1) * (size_t)p.n + g) * 4, o, tag0 + (unsigned)(k + 1));
                }
            }
            // Phase B: the remaining records, then the interior vertices.  At
            // most a warp's worth of records goes to the last threads, which
            // are idle while the first ones sum the boundary vertices; a larger
            // phase B stays on the first threads, which reach it after the
            // boundary offsets are out, so that it does not compete with the
            // boundary sums the neighbouring patches wait for.
            if (!one_phase) {
                if (!skip_k)
                    local_records<MODE, NT>(rc, rh, hvs, sy, sd, ncell, nhin, ph.ncell_a, ncell, ph.nhin_a, nhin, cxy,
                                            cz, (ncell - ph.ncell_a) + (nhin - ph.nhin_a) <= 32);
                named_sync(1, NT);
            }
            if (k + 1 < nsweep && k + 1 <= max_iter() && hl0 < nlocal)
                ld_words(p.xch + ((size_t)((k + 1) & 1) * (size_t)p.n + hg0) * 4, pw0, pw1, pw2);
            if (!skip_k && own && tid >= ph.nbnd) {
                vertex_update<MODE>(npad, sptr, tid, sy, sd, cxy, cz, dprev, gamma, omega_k, o, d, r2);
                if (!res_only) ((k & 1) ? a.buf[0] : a.buf[1])[g] = o;
            }
            // every record has read d^k: the owned offsets move on
            if (!skip_k && own && !res_only) {
                sd[tid] = o;
                if (TOL) dpp = dprev;
                dprev = d;
            }
            if (TOL) {
                // the block's residual is added by the spare warp
                r2 = warp_sum(r2);
                if ((tid & 31) == 0) red[k & 1][tid >> 5] = r2;
                named_arrive(2 + (k & 1), NTT);
            } else if (MODE == kModeConsistent && !skip_k && (k == 0 || k >= max_iter() - 1)) {
                // fixed sweep counts read only the residual of the start and
                // of the last sweeps
                compute_residual<NT>(r2, red[0], acc + k);
            }
        }
        if (TOL && !left && kend >= k0 + 2) {
            // the last decision, about sweep kend - 2; the last sweep may have
            // only evaluated the residual
            named_sync(4 + (kend & 1), NTT);
            if (dec[kend & 1] == 1 && own && kend - 1 < max_iter()) ((kend & 1) ? a.buf[1] : a.buf[0])[g] = dpp;
        }
    } else if (TOL) {
        // ---- the spare warp: residual sums and decisions ----
        const int npc = ci.patch_end - ci.patch_begin;
        const int lane = tid & 31;
        // waits for the complete sum of sweep j; false when a wait ran out
        auto complete = [&](int j) {
            const long long t0 = clock64();
            for (;;) {
                int n;
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];"
                             : "=r"(n) : "l"(__cvta_generic_to_global(cnt + j)) : "memory");
                if (n >= npc) return true;
                if (clock64() - t0 > p.spin_budget || *(volatile int*)p.err != 0) {
                    atomicCAS(p.err, 0, 3);
                    return false;
                }
            }
        };
        bool ended = false;
        for (int k = k0; k < kend; ++k) {
            if (k > k0) {
                // the decision about sweep k - 1, taken at the top of sweep
                // k + 1: every patch of the cloth has added its part of the
                // sum by now or is about to
                const int j = k - 1;
                int go = 0;
                if (lane == 0) {
                    if (!complete(j)) go = 2;
                    if (go == 0) {
                        // the normaliser, as in cloth_done
                        const bool own_start = !(RANGE && ci.init >= 2 && a.warm_active);
                        const double ry2 = ld_cg_f64(own_start ? acc : &a.crt[c].res_y2), rk2 = ld_cg_f64(acc + j);
                        const float tol = ci.tol;
                        const bool bad = !isfinite(rk2);
                        if (bad || (tol > 0.f && rk2 <= (double)tol * (double)tol * ry2)) {
                            go = 1;
                            end_s = FrameEnd{j, bad ? -6 : 0};
                            stopped = 1;
                            if (first) {
                                ClothRT* rt = a.crt + c;
                                if (RANGE) {
                                    rt->res0_2 = ld_cg_f64(acc);
                                    if (own_start) rt->res_y2 = ry2;
                                }
                                rt->used = j; rt->resf_2 = rk2; rt->active = 0;
                                if (bad) rt->status = -6;
                            }
                        }
                    }
                    dec[(k + 1) & 1] = go;
                }
                go = __shfl_sync(0xffffffffu, go, 0);
                __syncwarp();
                named_arrive(4 + ((k + 1) & 1), NTT);
                if (go) {
                    // the compute threads finish sweep k and stop at the top
                    // of the next one: their partial sums are not needed
                    named_sync(2 + (k & 1), NTT);
                    ended = true;
                    break;
                }
            }
            named_sync(2 + (k & 1), NTT);
            if (*(volatile int*)&gone) { ended = true; break; }
            float v = lane < NT / 32 ? red[k & 1][lane] : 0.f;
            v = warp_sum(v);
            if (lane == 0) {
                atomicAdd(acc + k, (double)v);
                __threadfence();
                atomicAdd(cnt + k, 1);
            }
        }
        // a cloth whose cap lies inside the range: its record, as the sweep
        // after its last one would have left it
        const int kq = max_iter() + (a.have_final ? 1 : 0);
        if (RANGE && first && lane == 0 && !ended && kend > k0 && kq < nsweep && complete(kend - 1))
            cloth_done(a, c, kq, true, true);
    } else if (first) {
        for (int k = tid - NT; k < a.acc_stride; k += 32) p.cnt[(par ^ 1u) * set + (size_t)c * a.acc_stride + k] = 0;
    }
    if (RANGE) return;
    // every per-sweep sum is complete after this barrier, and every block has
    // read the frame's words
    if (!grid_barrier_r(p.bar, p.err, p.spin_budget)) return;
    if (blockIdx.x == 0 && tid == 0) {
        *p.xch_tag = tag0 + (unsigned)nsweep;
        *p.frame = par ^ 1u;
    }
    if (tid < 32) {
        const FrameEnd end = end_frame(a, c, acc, TOL && stopped ? &end_s : nullptr, first);
        if (tid == 0) end_s = end;
    }
    if (caller_out) {
        // (vertices of any cloth: their records)
        if (!grid_barrier_r(p.bar, p.err, p.spin_budget)) return;
        for (int o = o0; comp && o < p.n; o += (int)gridDim.x * NT) {
            const int gv = __ldg(&p.io_inv[o]);
            finalize_vertex(gv, p.Xw, p.V, p.Y, a.buf[0], a.buf[1], p.aux, p.vcloth, a.cinfo, a.crt);
            store_frame_state(p, o, gv);
        }
        return;
    }
    __syncthreads();
    if (own) finalize_vertex(g, end_s, ci, p.Xw, p.V, p.Y, a.buf[0], a.buf[1], p.aux);
}

// NT compute threads plus one warp: 480 + 32 threads, one block (one patch)
// per SM; 224 + 32, two half-size patches per SM; 128 + 32, three patches per
// SM (ranges only).  Instances: fixed sweep counts (the consistent solve, the
// reference-literal solve, the consistent solve that moves the caller's
// state), the consistent solve to a tolerance without and with the caller's
// state, and its ranges of sweeps.
struct ResVariant { int nt; void* f[6]; };

static const ResVariant* res_variants(int* n)
{
    static const ResVariant v[] = {
        {480, {(void*)k_resident<kModeConsistent, 480, false, false, false>,
               (void*)k_resident<kModeLiteral, 480, false, false, false>,
               (void*)k_resident<kModeConsistent, 480, true, false, false>,
               (void*)k_resident<kModeConsistent, 480, false, true, false>,
               (void*)k_resident<kModeConsistent, 480, true, true, false>,
               (void*)k_resident<kModeConsistent, 480, false, true, true>}},
        {224, {(void*)k_resident<kModeConsistent, 224, false, false, false>,
               (void*)k_resident<kModeLiteral, 224, false, false, false>,
               (void*)k_resident<kModeConsistent, 224, true, false, false>,
               (void*)k_resident<kModeConsistent, 224, false, true, false>,
               (void*)k_resident<kModeConsistent, 224, true, true, false>,
               (void*)k_resident<kModeConsistent, 224, false, true, true>}},
        {128, {nullptr, nullptr, nullptr, nullptr, nullptr, (void*)k_resident<kModeConsistent, 128, false, true, true>}},
    };
    *n = 3;
    return v;
}

int resident_pick(int nt)
{
    int n = 0;
    const ResVariant* v = res_variants(&n);
    for (int i = 0; i < n; ++i)
        if (v[i].nt == nt) return i;
    return -1;
}

static void* variant_fn(int variant, int mode, bool io, bool tol)
{
    int n = 0;
    const ResVariant* v = res_variants(&n);
    if (variant < 0 || variant >= n) return nullptr;
    if (mode != kModeConsistent) return io || tol ? nullptr : v[variant].f[1];
    return v[variant].f[tol ? (io ? 4 : 3) : (io ? 2 : 0)];
}

// Blocks of instance f that are resident at once (0: it cannot run).
static int resident_blocks_of(void* f, int threads, size_t smem)
{
    int dev = 0, nsm = 0, nb = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) return 0;
    if (smem > 220 * 1024 || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, threads, smem) != cudaSuccess) return 0;
    return nb * nsm;
}

bool resident_moves_state(int mode) { return mode == kModeConsistent; }

int resident_max_blocks(int mode, int variant, size_t smem)
{
    int n = 0, nb = 0;
    const int nt = variant_fn(variant, mode, false, false) ? res_variants(&n)[variant].nt : 0;
    // the solver may run any instance of its mode (the tolerance can change)
    for (int i = 0; i < 4 && nt; ++i) {
        void* f = variant_fn(variant, mode, (i & 1) != 0, (i & 2) != 0);
        if (!f) continue;
        const int b = resident_blocks_of(f, nt + 32, smem);
        nb = i == 0 || b < nb ? b : nb;
    }
    return nb;
}

int resident_range_pick(int max_nown, int max_rec, int npatch, size_t smem)
{
    // the smallest blocks that hold the patches, more of them per SM, but
    // larger ones where a patch's records then take one round of the threads
    // (128-vertex patches, 189 records: 5,289 vertices 168 -> 139 us per 50
    // sweeps, 32,001 190 -> 166)
    int n = 0, pick = -1;
    const ResVariant* v = res_variants(&n);
    for (int i = n - 1; i >= 0; --i) {
        if (max_nown > v[i].nt || npatch > resident_blocks_of(v[i].f[5], v[i].nt + 32, smem)) continue;
        if (max_rec <= v[i].nt) return i;
        if (pick < 0) pick = i;
    }
    return pick;
}

cudaError_t launch_resident_range(const PersistArgs& p, int variant, int grid, size_t smem, cudaStream_t s)
{
    int n = 0;
    const ResVariant* v = res_variants(&n);
    if (variant < 0 || variant >= n || grid <= 0) return cudaErrorInvalidValue;
    if (p.k1 <= p.k0) return cudaSuccess;
    PersistArgs copy = p;
    void* args[] = {&copy};
    return cudaLaunchCooperativeKernel(v[variant].f[5], dim3(grid), dim3(v[variant].nt + 32), args, smem, s);
}

cudaError_t launch_resident(const PersistArgs& p, int variant, int grid, size_t smem, cudaStream_t s)
{
    const bool io = p.in_x || p.in_v || p.out_x || p.out_v;
    void* f = variant_fn(variant, p.mode, io, p.nbr_sync == 0);
    if (!f || grid <= 0) return cudaErrorInvalidValue;
    int n = 0;
    const int nt = res_variants(&n)[variant].nt;
    PersistArgs copy = p;
    void* args[] = {&copy};
    return cudaLaunchCooperativeKernel(f, dim3(grid), dim3(nt + 32), args, smem, s);
}

}  // namespace pdg
