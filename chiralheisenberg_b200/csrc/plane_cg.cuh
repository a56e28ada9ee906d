// plane_cg.cuh -- conjugate gradients on M^dagger M (+ sigma) for a batch of
// independent systems whose vectors are planes (planes.cuh).
//
// Three kinds of system share the kernels:
//   T = double2  congrad (rhmc/cheisdwf.f:1064-1157): FP64 vectors, REAL*4
//                scalars, sums formed in FP64 and rounded once (the reference
//                adds element by element in REAL*4, an order that no parallel
//                sum can follow), the reference's stopping rule;
//   T = hmc32    congrad of the HMC predecessor (hmc_planes.cuh): the same
//                rule on FP32 vectors with every operation rounded;
//   T = float2   the inner solver of the per-shift defect correction: FP32
//                vectors, FP64 scalars, (M^dagger M + sigma) e = r to a
//                relative residual.
// One iteration is three kernels over the blocks of all systems:
//   k_pcg1  x1 = M p, |x1|^2
//   k_pcg2  r -= alpha (M^dagger x1 + sigma p), |r|^2, x += alpha p
//   k_pcg3  p = r + beta p (and |p|^2 where sigma enters), the scalars
// x is updated beside the stencil, whose latencies hide it (in k_pcg3, which
// moves bytes only, 32 FP64 solves took 202 ms instead of 193); hmc32 does it
// in k_pcg3, where it spares registers and a load of p (11.6 -> 10.8 ms).
// A block leaves its partial; the kernel that needs a sum adds the system's
// partials itself, in one order.  A system's scalars are kept in two slots by
// the parity of the iteration: k_pcg3 reads one while its first block of the
// system writes the other.  All systems of a batch start together, so the
// iteration number is common; finished systems' blocks return at once.
//
// A system's blocks and the order of its sums depend on its lattice alone,
// so a system's solution has the same bits alone and in any batch.
//
// The batch's layout (lattices, plans, where each system's blocks and vectors
// start) is a kernel argument: a block finds its system by a search over
// argument memory on blockIdx, so the plan and the vectors' addresses stay in
// uniform registers as in a single solve.  Read from a table in shared memory
// they cost the stencil 100-250 bytes of spills at 80 registers: 32 solves up
// to 16^3x24 224 ms instead of the figure at kBatchBytes.
#pragma once
#include <cstring>
#include <vector>

#include "chunk_graph.h"
#include "planes.cuh"
#include "row_stage.cuh"

namespace chdwf {

constexpr int kPcgThreads = 192;      // a block; 4 an SM at kPlaneRegs
constexpr int kPcgMaxBlocks = 2048;   // stencil blocks of one system
// bytes of a vector a thread takes in k_pcg3
constexpr int kPcgBytes = 64;
template <class T> constexpr int pcg_units_thread() {
    return kPcgBytes / (int)sizeof(typename unit_of<T>::type);
}

struct PcgSlot {
    float alphan, betad;     // congrad
    double rr;               // shifted: |r|^2
    int done, iters;
};

constexpr int kPcgSys = 32;           // systems of one set of launches
constexpr int kPcgGeo = 6;            // distinct lattices and parameters among them

template <class T>
struct PcgGeo {
    typedef typename real_of<T>::type Real;
    PlanePlan pl;
    Real diag, hpin;
    int apbc;
    int nblk, neblk;                  // stencil blocks, element blocks (k_pcg3)
};
// What may change from call to call in a batch of the same layout (device).
template <class T>
struct PcgDyn {
    typedef typename unit_of<T>::type V;
    V* x;
    typename real_of<T>::type sigma;
    float resid;                      // congrad: stop when betan < resid
    double rstop;                     // shifted: stop when |r|^2 <= rstop
    int niterc;                       // iteration cap
};
struct PcgRun {                       // iterations before this chunk, before the next
    int base, next;
    int active;                       // systems still running
};

template <class T>
struct PcgArgs {
    typedef typename unit_of<T>::type V;
    PcgGeo<T> geo[kPcgGeo];
    int64_t vec0[kPcgSys];            // system's vectors p, r, x1 (units from vec)
    int chi0[kPcgSys];                // its REAL*4 chi (from chif)
    int part0[kPcgSys];               // its partials of |x1|^2, |r|^2, |p|^2, and alpha (from part)
    int blk0[kPcgSys + 1], eblk0[kPcgSys + 1];
    unsigned char gid[kPcgSys];
    int nsys, ngeo;
    V* vec;
    const float* chif;
    double* part;
    const PcgDyn<T>* dyn;
    PcgSlot* slot;                    // [nsys][2]
    PcgRun* run;
    int* hflag;                       // mapped host flag: set when none is running
};

// The system that block b belongs to: the last s with first[s] <= b.
__device__ __forceinline__ int pcg_find(const int* first, int nsys, int b) {
    int lo = 0, hi = nsys;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (b >= first[mid]) lo = mid;
        else hi = mid;
    }
    return lo;
}

static __global__ void k_pcg_tick(PcgRun* run, int chunk) {
    run->base = run->next;
    run->next += chunk;
}

// What a kind of system brings: its stencil, and s*a + b of its updates.
// congrad's without fused multiply-add, as the reference rounds them; the FP32
// correction's with.
template <class T> struct PcgOp {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    static constexpr bool kShifted = std::is_same<T, float2>::value;
    static constexpr bool kLateX = false;              // x in k_pcg3
    template <bool DAG, int IMASS, class Epi>
    static __device__ __forceinline__ void item(const V* in, const PlanePlan& pl,
                                                const PlaneThread& th, uint32_t it,
                                                const float* chif, Real diag, Real hpin,
                                                bool apbc, Epi& epi) {
        plane_item<DAG, IMASS, true, std::is_same<T, double2>::value || IMASS == 3>(
            in, pl, th, it, chif, diag, hpin, apbc, epi);
    }
    static __device__ __forceinline__ double2 axpy(double s, double2 a, double2 b) {
        return zadd(b, zscal(s, a));
    }
    static __device__ __forceinline__ cpair axpy(float s, const cpair& a, const cpair& b) {
        return zaxpy(s, a, b);
    }
    static __device__ __forceinline__ double norm2(const V& v) { return unit_norm2(v); }
};

template <class T>
struct PcgEpi1 {
    typedef typename unit_of<T>::type V;
    V* x1;
    double loc;
    __device__ __forceinline__ bool operator()(V acc[4], int64_t e, int64_t cst, uint32_t o,
                                               bool act, int, uint32_t) {
        if (!act) return true;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            st_unit(unit_at(x1 + e + d * cst, o), acc[d]);
            loc += PcgOp<T>::norm2(acc[d]);
        }
        return true;
    }
};
template <class T>
struct PcgEpi2 {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    const V* p;
    V *r, *x;
    Real alpha, sigma;
    bool upd;                         // x is updated (congrad: nx > 1)
    double loc;
    __device__ __forceinline__ bool operator()(V acc[4], int64_t e, int64_t cst, uint32_t o,
                                               bool act, int, uint32_t) {
        if (!act) return true;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int64_t ed = e + d * cst;
            V a = acc[d];
            if (!PcgOp<T>::kLateX && (PcgOp<T>::kShifted || upd)) {
                const V pv = ld_unit(unit_at(p + ed, o));
                if (PcgOp<T>::kShifted) a = PcgOp<T>::axpy(sigma, pv, a);
                if (upd)
                    st_unit(unit_at(x + ed, o),
                            PcgOp<T>::axpy(alpha, pv, ld_unit(unit_at(x + ed, o))));
            }
            const V rv = PcgOp<T>::axpy(-alpha, a, ld_unit(unit_at(r + ed, o)));
            st_unit(unit_at(r + ed, o), rv);
            loc += PcgOp<T>::norm2(rv);
        }
        return true;
    }
};

template <bool DAG, int IMASS, class T, class Epi>
__device__ __forceinline__ void pcg_sweep(const PcgArgs<T>& a, const PcgGeo<T>& G, int s, int b,
                                          const typename unit_of<T>::type* in,
                                          const PlaneThread& th, Epi& epi) {
    for (uint32_t it = (uint32_t)b; it < G.pl.nitem; it += (uint32_t)G.nblk)
        PcgOp<T>::template item<DAG, IMASS>(in, G.pl, th, it, a.chif + a.chi0[s], G.diag, G.hpin,
                                            G.apbc != 0, epi);
}
template <class T>
__device__ __forceinline__ int64_t pcg_units(const PlanePlan& pl) {
    return 8 * (int64_t)pl.U * pl.kvol;
}

template <class T, int IMASS>
__global__ void __maxnreg__(kPlaneRegs) k_pcg1(const __grid_constant__ PcgArgs<T> a, int k) {
    typedef typename unit_of<T>::type V;
    const int s = pcg_find(a.blk0, a.nsys, (int)blockIdx.x);
    const PcgGeo<T>& G = a.geo[a.gid[s]];
    const int b = (int)blockIdx.x - a.blk0[s];
    const PlaneThread th = plane_thread(G.pl);
    V* p = a.vec + a.vec0[s];
    pdl_wait();
    if (a.slot[2 * s + (k & 1)].done) return;
    PcgEpi1<T> epi{p + 2 * pcg_units<T>(G.pl), 0.0};
    pcg_sweep<false, IMASS>(a, G, s, b, p, th, epi);
    __shared__ double sh[32];
    const double loc = block_sum_any(epi.loc, sh);
    if (threadIdx.x == 0) a.part[a.part0[s] + b] = loc;
}

template <class T, int IMASS>
__global__ void __maxnreg__(kPlaneRegs) k_pcg2(const __grid_constant__ PcgArgs<T> a, int k) {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    const int s = pcg_find(a.blk0, a.nsys, (int)blockIdx.x);
    const PcgGeo<T>& G = a.geo[a.gid[s]];
    const int b = (int)blockIdx.x - a.blk0[s];
    const PlaneThread th = plane_thread(G.pl);
    V* p = a.vec + a.vec0[s];
    double* part = a.part + a.part0[s];
    PcgEpi2<T> epi{p, p + pcg_units<T>(G.pl), a.dyn[s].x, (Real)1, a.dyn[s].sigma, true, 0.0};
    pdl_wait();
    const PcgSlot c = a.slot[2 * s + (k & 1)];
    if (c.done) return;
    const double tot = sum_partials_any(part, G.nblk);
    if constexpr (!PcgOp<T>::kShifted) {
        // alphad = |x1|^2 ; alpha = alphan/alphad from the second iteration on
        // (:1093-1117)
        const int nx = a.run->base + k + 1;
        epi.upd = nx > 1;
        if (nx > 1) epi.alpha = (Real)(c.alphan / (float)tot);
    } else {
        // p^dagger (M^dagger M + sigma) p = |M p|^2 + sigma |p|^2; a value that
        // is not positive ends the system in k_pcg3
        __syncthreads();
        const double pap = tot + (double)epi.sigma * sum_partials_any(part + 2 * G.nblk, G.neblk);
        epi.alpha = pap > 0.0 ? (float)(c.rr / pap) : 0.0f;
    }
    if (PcgOp<T>::kLateX && b == 0 && threadIdx.x == 0) part[2 * G.nblk + G.neblk] = (double)epi.alpha;
    pcg_sweep<true, IMASS>(a, G, s, b, p + 2 * pcg_units<T>(G.pl), th, epi);
    __shared__ double sh[32];
    const double loc = block_sum_any(epi.loc, sh);
    if (threadIdx.x == 0) part[G.nblk + b] = loc;
}

template <class T>
__global__ void __launch_bounds__(kPcgThreads) k_pcg3(const __grid_constant__ PcgArgs<T> a, int k) {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    const int s = pcg_find(a.eblk0, a.nsys, (int)blockIdx.x);
    const PcgGeo<T>& G = a.geo[a.gid[s]];
    const int b = (int)blockIdx.x - a.eblk0[s];
    const int64_t nu = pcg_units<T>(G.pl);
    V *p = a.vec + a.vec0[s], *r = p + nu;
    double* part = a.part + a.part0[s];
    const float resid = a.dyn[s].resid;
    const double rstop = a.dyn[s].rstop;
    const int niterc = a.dyn[s].niterc;
    V* x = a.dyn[s].x;
    constexpr bool LX = PcgOp<T>::kLateX;
    constexpr int N = pcg_units_thread<T>();
    const int64_t i0 = (int64_t)b * (kPcgThreads * N) + threadIdx.x;
    V pv[N], rv[N], xv[LX ? N : 1];
    auto load = [&] {
#pragma unroll
        for (int q = 0; q < N; q++) {
            const int64_t i = i0 + q * kPcgThreads;
            if (i >= nu) break;
            pv[q] = ld_unit(p + i);
            rv[q] = ld_unit(r + i);
            if (LX) xv[q] = ld_unit(x + i);
        }
    };
    pdl_wait();
    // hmc32: on their way while the sum is formed (12.2 -> 10.9 ms); the others'
    // batches have blocks enough to hide it, and are 5% slower so
    if (LX) load();
    const PcgSlot c = a.slot[2 * s + (k & 1)];
    PcgSlot* next = a.slot + 2 * s + ((k + 1) & 1);
    if (c.done) {
        if (b == 0 && threadIdx.x == 0) *next = c;
        return;
    }
    const Real alpha = LX ? (Real)part[2 * G.nblk + G.neblk] : (Real)0;
    const double tot = sum_partials_any(part + G.nblk, G.nblk);
    const int nx = a.run->base + k + 1;
    PcgSlot n = c;
    Real beta;
    if constexpr (!PcgOp<T>::kShifted) {
        const float betan = (float)tot;                    // :1133-1141
        float bt = betan / c.betad;
        n.betad = betan;
        n.alphan = betan;
        if (nx == 1) bt = 0.0f;
        if (betan < resid) n.done = 1;
        else if (nx >= niterc) n.done = 2;
        if (!(betan == betan)) n.done = 3;
        beta = (Real)bt;
    } else {
        n.rr = tot;
        beta = (float)(tot / c.rr);
        if (tot <= rstop || !(tot == tot)) n.done = 1;
        else if (nx >= niterc) n.done = 2;
        else if (tot == c.rr) n.done = 2;                  // alpha 0: no progress
    }
    if (n.done) n.iters = nx;
    if (b == 0 && threadIdx.x == 0) {
        *next = n;
        if (n.done && atomicSub(&a.run->active, 1) == 1 && a.hflag) {
            *(volatile int*)a.hflag = 1;
            __threadfence_system();
        }
    }
    if (!LX) {
        if (n.done) return;
        load();
    }
    // x += alpha p (from the second iteration on), p = r + beta p (:1121-1127,
    // :1147-1150)
    double loc = 0.0;
#pragma unroll
    for (int q = 0; q < N; q++) {
        const int64_t i = i0 + q * kPcgThreads;
        if (i >= nu) break;
        if (LX && nx > 1) st_unit(x + i, PcgOp<T>::axpy(alpha, pv[q], xv[q]));
        if (n.done) continue;
        const V v = PcgOp<T>::axpy(beta, pv[q], rv[q]);
        st_unit(p + i, v);
        if (PcgOp<T>::kShifted) loc += PcgOp<T>::norm2(v);
    }
    if (n.done) return;
    if constexpr (PcgOp<T>::kShifted) {
        __shared__ double sh[32];
        loc = block_sum_any(loc, sh);
        if (threadIdx.x == 0) part[2 * G.nblk + b] = loc;
    }
}

// ABI layout <-> planes of one system (FP64): p = x, r = Phi, and the solution
// kept in planes in its own buffer while the solve runs.
static __global__ void k_pcg_in(double2* __restrict__ out, const double2* __restrict__ in, Geom g) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < g.kferm) out[i] = in[plane_unit_of<double2>(g, g.Ls, i).e];
}
static __global__ void k_pcg_out(double2* __restrict__ out, const double2* __restrict__ in, Geom g) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < g.kferm) out[plane_unit_of<double2>(g, g.Ls, i).e] = in[i];
}

// ---- host side ---------------------------------------------------------------------
inline int pcg_sms() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm > 0 ? nsm : 1;
}
// A batch under construction: systems are added while they fit.
template <class T>
struct PcgBatch {
    typedef typename real_of<T>::type Real;
    static constexpr bool kPair = std::is_same<typename unit_of<T>::type, cpair>::value;
    PcgArgs<T> a;                     // layout; the pointers are set when it runs
    int imass = 1;
    int64_t units = 0;
    int chis = 0, parts = 0;
    PcgBatch() { memset(&a, 0, sizeof(a)); }   // padding too: it is a graph's key
    // Vectors of a system: p, r, x1 and extra more.  False: the batch is full.
    bool add(const Geom& g, Real diag, Real hpin, int apbc, int im, int extra, int nsm) {
        if (a.nsys == kPcgSys || (a.nsys > 0 && im != imass)) return false;
        PcgGeo<T> G;
        memset(&G, 0, sizeof(G));
        G.pl = plane_plan(g, kPair, nsm, kPcgThreads);
        G.diag = diag;
        G.hpin = hpin;
        G.apbc = apbc;
        G.nblk = G.pl.nitem < (uint32_t)kPcgMaxBlocks ? (int)G.pl.nitem : kPcgMaxBlocks;
        const int64_t nu = 8 * (int64_t)G.pl.U * g.kvol;
        const int per = kPcgThreads * pcg_units_thread<T>();
        const int64_t ne = (nu + per - 1) / per;
        if (ne > (int64_t)1 << 30) return false;
        G.neblk = (int)ne;
        int id = 0;
        while (id < a.ngeo && memcmp(&a.geo[id], &G, sizeof(G)) != 0) id++;
        if (id == kPcgGeo) return false;
        if ((int64_t)a.eblk0[a.nsys] + ne > (int64_t)1 << 30 ||
            (int64_t)chis + 3 * (int64_t)g.kvol > (int64_t)1 << 30)
            return false;
        if (id == a.ngeo) a.geo[a.ngeo++] = G;
        const int s = a.nsys++;
        imass = im;
        a.gid[s] = (unsigned char)id;
        a.vec0[s] = units;
        a.chi0[s] = chis;
        a.part0[s] = parts;
        a.blk0[s + 1] = a.blk0[s] + G.nblk;
        a.eblk0[s + 1] = a.eblk0[s] + G.neblk;
        units += (3 + extra) * nu;
        chis += 3 * g.kvol;
        parts += 2 * G.nblk + G.neblk + 1;
        return true;
    }
    const PcgGeo<T>& geo(int s) const { return a.geo[a.gid[s]]; }
    int64_t vec_units(int s) const {
        return 8 * (int64_t)geo(s).pl.U * geo(s).pl.kvol;
    }
};

template <class T>
void pcg_launch_chunk(const PcgArgs<T>& a, int imass, int chunk, cudaStream_t st) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{}, ce{};
    c.gridDim = dim3((unsigned)a.blk0[a.nsys]);
    c.blockDim = dim3(kPcgThreads);
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    ce = c;
    ce.gridDim = dim3((unsigned)a.eblk0[a.nsys]);
    k_pcg_tick<<<1, 1, 0, st>>>(a.run, chunk);
    for (int k = 0; k < chunk; k++) {
        if (imass == 3) {
            cudaLaunchKernelEx(&c, k_pcg1<T, 3>, a, k);
            cudaLaunchKernelEx(&c, k_pcg2<T, 3>, a, k);
        } else {
            cudaLaunchKernelEx(&c, k_pcg1<T, 1>, a, k);
            cudaLaunchKernelEx(&c, k_pcg2<T, 1>, a, k);
        }
        cudaLaunchKernelEx(&ce, k_pcg3<T>, a, k);
    }
}

// Vectors and device state of a batch, kept between solves and grown when a
// larger batch arrives.
template <class T>
struct PcgWork {
    typedef typename unit_of<T>::type V;
    int64_t cap_units = 0;
    int cap_chi = 0, cap_part = 0;
    V* vec = nullptr;
    float* chif = nullptr;
    double* part = nullptr;
    PcgDyn<T>* dyn = nullptr;
    PcgSlot* slot = nullptr;
    PcgRun* run = nullptr;
    int *hflag_host = nullptr, *hflag_dev = nullptr;
    ChunkGraphs graphs;
    void release() {
        graphs.release();
        cudaFree(vec); cudaFree(chif); cudaFree(part); cudaFree(dyn); cudaFree(slot); cudaFree(run);
        if (hflag_host) cudaFreeHost(hflag_host);
        vec = nullptr; chif = nullptr; part = nullptr; dyn = nullptr; slot = nullptr; run = nullptr;
        hflag_host = hflag_dev = nullptr;
        cap_units = 0;
        cap_chi = cap_part = 0;
    }
    cudaError_t reserve(int64_t units, int chis, int parts) {
        if (run && units <= cap_units && chis <= cap_chi && parts <= cap_part) return cudaSuccess;
        release();
        cudaError_t e;
        if ((e = cudaMalloc(&vec, sizeof(V) * (size_t)units)) ||
            (e = cudaMalloc(&chif, sizeof(float) * (size_t)(chis ? chis : 1))) ||
            (e = cudaMalloc(&part, sizeof(double) * (size_t)parts)) ||
            (e = cudaMalloc(&dyn, sizeof(PcgDyn<T>) * kPcgSys)) ||
            (e = cudaMalloc(&slot, sizeof(PcgSlot) * 2 * kPcgSys)) ||
            (e = cudaMalloc(&run, sizeof(PcgRun))) ||
            (e = cudaHostAlloc(&hflag_host, sizeof(int), cudaHostAllocMapped)) ||
            (e = cudaHostGetDevicePointer((void**)&hflag_dev, hflag_host, 0))) {
            release();
            return e;
        }
        cap_units = units; cap_chi = chis; cap_part = parts;
        return cudaSuccess;
    }
    // chi: one field for all systems instead of the workspace's
    void bind(PcgBatch<T>& b, const float* chi = nullptr) {
        if (chi) memset(b.a.chi0, 0, sizeof(b.a.chi0));
        b.a.vec = vec;
        b.a.chif = chi ? chi : chif;
        b.a.part = part;
        b.a.dyn = dyn;
        b.a.slot = slot;
        b.a.run = run;
        b.a.hflag = hflag_dev;
    }
    // Runs a bound batch to its end.  Vectors initialised on st; dyn: the
    // systems' solutions, scalars and caps; slots: their initial slots (FP32:
    // |p|^2's partials as well), on return the final ones.
    cudaError_t solve(const PcgBatch<T>& b, const std::vector<PcgDyn<T>>& hd,
                      std::vector<PcgSlot>& slots, cudaStream_t st) {
        const int nsys = b.a.nsys;
        int cap = 0;
        for (const PcgDyn<T>& d : hd)
            if (d.niterc > cap) cap = d.niterc;
        std::vector<PcgSlot> s2(2 * nsys);
        for (int i = 0; i < nsys; i++) s2[2 * i] = s2[2 * i + 1] = slots[i];
        PcgRun hr{0, 0, nsys};
        cudaError_t e;
        if ((e = cudaMemcpyAsync(dyn, hd.data(), sizeof(PcgDyn<T>) * nsys, cudaMemcpyHostToDevice, st)) ||
            (e = cudaMemcpyAsync(slot, s2.data(), sizeof(PcgSlot) * 2 * nsys, cudaMemcpyHostToDevice, st)) ||
            (e = cudaMemcpyAsync(run, &hr, sizeof(hr), cudaMemcpyHostToDevice, st)))
            return e;
        *hflag_host = 0;
        constexpr int kChunk = 16;
        const cudaGraphExec_t ge =
            graphs.get(b.a, b.imass, st, [&] { pcg_launch_chunk(b.a, b.imass, kChunk, st); });
        cudaEvent_t ev[2];
        cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
        cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
        int64_t launched = 0;
        for (int n = 0; launched < cap; n++) {
            if (ge) cudaGraphLaunch(ge, st);
            else pcg_launch_chunk(b.a, b.imass, kChunk, st);
            launched += kChunk;
            count_launches(3 * kChunk + 1);
            cudaEventRecord(ev[n & 1], st);
            // one chunk is queued beyond the one that is looked at
            if (n >= 1) {
                cudaEventSynchronize(ev[(n - 1) & 1]);
                if (*(volatile int*)hflag_host) break;
            }
        }
        cudaEventDestroy(ev[0]);
        cudaEventDestroy(ev[1]);
        if ((e = cudaGetLastError())) return e;
        if ((e = cudaMemcpyAsync(s2.data(), slot, sizeof(PcgSlot) * 2 * nsys, cudaMemcpyDeviceToHost,
                                 st)) ||
            (e = cudaStreamSynchronize(st)))
            return e;
        // a finished system's final slot is carried along in both
        for (int i = 0; i < nsys; i++) slots[i] = s2[2 * i].done ? s2[2 * i] : s2[2 * i + 1];
        return cudaSuccess;
    }
};

// congrad's initial state (:1086-1091) and limits
inline PcgSlot pcg_congrad_slot() {
    PcgSlot s;
    memset(&s, 0, sizeof(s));
    s.betad = 1.0f;
    return s;
}
inline PcgDyn<double2> pcg_congrad_dyn(const Geom& g, float res, double2* x) {
    PcgDyn<double2> d;
    memset(&d, 0, sizeof(d));
    d.x = x;
    d.resid = (float)g.kferm * res * res;                    // :1076
    d.niterc = (int)(g.Ls * (int64_t)g.kvol);
    return d;
}
// p = x ; r = Phi (:1086-1089) in planes, and x in planes in its own buffer
inline void pcg_congrad_enter(const Geom& g, double2* p, double2* x, const double2* phi,
                              cudaStream_t st) {
    const unsigned nb = (unsigned)((g.kferm + kThreads - 1) / kThreads);
    k_pcg_in<<<nb, kThreads, 0, st>>>(p, x, g);
    k_pcg_in<<<nb, kThreads, 0, st>>>(p + g.kferm, phi, g);
    cudaMemcpyAsync(x, p, sizeof(double2) * g.kferm, cudaMemcpyDeviceToDevice, st);
    count_launches(2);
}
// x back in the ABI's layout (through x1)
inline void pcg_congrad_leave(const Geom& g, double2* p, double2* x, cudaStream_t st) {
    double2* x1 = p + 2 * g.kferm;
    k_pcg_out<<<(unsigned)((g.kferm + kThreads - 1) / kThreads), kThreads, 0, st>>>(x1, x, g);
    cudaMemcpyAsync(x, x1, sizeof(double2) * g.kferm, cudaMemcpyDeviceToDevice, st);
    count_launches(1);
}
inline int pcg_status(const PcgSlot& s) { return s.done == 1 ? 0 : (s.done == 2 ? 1 : 2); }

}  // namespace chdwf
