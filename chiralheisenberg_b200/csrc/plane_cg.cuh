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
// A system's blocks (of its sums: a block of the launch may hold several, see
// PcgTile) and the order of its sums depend on its lattice alone, so a system's
// solution has the same bits alone and in any batch.
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

constexpr int kPcgThreads = 192;      // a block
constexpr int kPcgPerSm = 4;          // stencil blocks an SM holds at kPlaneRegs
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

// Systems of one set of launches, at most, and the same of chdwf_congrad_batch for
// sets that are wider.  Their arguments take 17 KB a kernel, which the first pass on a
// layout pays for (graph of 49 kernels: 5 to 10 ms more).
constexpr int kPcgSys = 32, kPcgSysBatch = 256;
// distinct lattices among NS systems
constexpr int pcg_geos(int NS) { return NS / 8 + 2; }

template <class T>
struct alignas(8) PcgGeo {        // with 4 the stencil kernels spill 30 to 50 bytes more
    PlanePlan pl;
    int nblk, neblk;                  // blocks of the stencil's sums, element blocks (k_pcg3)
    int pack;                         // of the former in a block of the launch
};
// What may change from call to call in a batch of the same layout (device).
template <class T>
struct PcgDyn {
    typedef typename unit_of<T>::type V;
    V* x;
    const V* phi;                     // congrad: right-hand side,
    const double* chi;                // and chi to be rounded (null: it is already)
    typename real_of<T>::type sigma;
    float resid;                      // congrad: stop when betan < resid
    double rstop;                     // shifted: stop when |r|^2 <= rstop
    int niterc;                       // iteration cap
};
struct PcgRun {                       // iterations before this chunk, before the next
    int base, next;
    int active;                       // systems still running
};

template <class T_, int NS>
struct PcgArgs {
    typedef T_ T;
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    static constexpr int kMost = NS;
    PcgGeo<T> geo[pcg_geos(NS)];
    int64_t vec0[NS];                 // system's vectors p, r, x1 (units from vec)
    Real diag[NS], hpin[NS];          // its parameters
    int apbc[NS];
    int chi0[NS];                     // its REAL*4 chi (from chif)
    int part0[NS];                    // its partials of |x1|^2, |r|^2, |p|^2, and alpha (from part)
    int blk0[NS + 1], eblk0[NS + 1];  // its first block in the launches
    unsigned char gid[NS];            // its lattice's entry of geo
    int nsys, ngeo, packed;
    V* vec;
    const float* chif;
    float* chi_out;                   // the same where the batch holds it
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

// The thread's place among a system's blocks.  With PACK a block of the launch
// holds G.pack of them: warps g*kw to g*kw + kw - 1 (kw: a tile's warps) are block
// b = pack * (block of the launch) + g; warps behind the last tile hold no site.
// g is the same for a warp, and the shuffle lets the compiler know, so that what
// hangs on b stays in uniform registers.  It costs k_pcg1 64 bytes of spills all
// the same (FP64, 24^3x24: 107 ms a solve instead of 103), so launches that are
// not packed have kernels without it.
struct PcgTile {
    int b, w0;                        // block, its first warp
    PlaneThread th;
};
template <bool PACK, class T>
__device__ __forceinline__ PcgTile pcg_tile(const PcgGeo<T>& G, int blk) {
    if (!PACK) return PcgTile{blk, 0, plane_thread(G.pl)};
    const int kw = G.pl.threads >> 5;
    int g = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0) / kw;
    g = g < G.pack ? g : G.pack - 1;
    return PcgTile{blk * G.pack + g, g * kw,
                   plane_thread(G.pl, (int)threadIdx.x - g * G.pl.threads)};
}
template <bool DAG, int IMASS, bool PACK, class A, class T, class Epi>
__device__ __forceinline__ void pcg_sweep(const A& a, const PcgGeo<T>& G, int s,
                                          const PcgTile& t, const typename unit_of<T>::type* in,
                                          Epi& epi) {
    if (PACK && t.b >= G.nblk) return;
    for (uint32_t it = (uint32_t)t.b; it < G.pl.nitem; it += (uint32_t)G.nblk)
        PcgOp<T>::template item<DAG, IMASS>(in, G.pl, t.th, it, a.chif + a.chi0[s], a.diag[s],
                                            a.hpin[s], a.apbc[s] != 0, epi);
}
// Block b's partial, its warps' sums added in order: the same however many
// blocks share a block of the launch.
template <class T>
__device__ __forceinline__ void pcg_partial(const PcgGeo<T>& G, const PcgTile& t, double loc,
                                            double* part) {
    __shared__ double sh[kPcgThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loc += __shfl_down_sync(0xffffffffu, loc, o);
    const int w = (int)threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sh[w] = loc;
    __syncthreads();
    if ((int)threadIdx.x != 32 * t.w0 || t.b >= G.nblk) return;
    double r = 0.0;
    for (int i = 0; i < G.pl.threads >> 5; i++) r += sh[w + i];
    part[t.b] = r;
}
template <class T>
__device__ __forceinline__ int64_t pcg_units(const PlanePlan& pl) {
    return 8 * (int64_t)pl.U * pl.kvol;
}

template <class A, int IMASS, bool PACK>
__global__ void __maxnreg__(kPlaneRegs) k_pcg1(const __grid_constant__ A a, int k) {
    typedef typename A::T T;
    typedef typename unit_of<T>::type V;
    const int s = pcg_find(a.blk0, a.nsys, (int)blockIdx.x);
    const PcgGeo<T>& G = a.geo[a.gid[s]];
    const PcgTile t = pcg_tile<PACK>(G, (int)blockIdx.x - a.blk0[s]);
    V* p = a.vec + a.vec0[s];
    pdl_wait();
    if (a.slot[2 * s + (k & 1)].done) return;
    PcgEpi1<T> epi{p + 2 * pcg_units<T>(G.pl), 0.0};
    pcg_sweep<false, IMASS, PACK>(a, G, s, t, p, epi);
    if constexpr (PACK) {
        pcg_partial(G, t, epi.loc, a.part + a.part0[s]);
    } else {
        __shared__ double sh[32];
        const double loc = block_sum_any(epi.loc, sh);
        if (threadIdx.x == 0) a.part[a.part0[s] + t.b] = loc;
    }
}

template <class A, int IMASS, bool PACK>
__global__ void __maxnreg__(kPlaneRegs) k_pcg2(const __grid_constant__ A a, int k) {
    typedef typename A::T T;
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    const int s = pcg_find(a.blk0, a.nsys, (int)blockIdx.x);
    const PcgGeo<T>& G = a.geo[a.gid[s]];
    const PcgTile t = pcg_tile<PACK>(G, (int)blockIdx.x - a.blk0[s]);
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
    if (PcgOp<T>::kLateX && t.b == 0 && threadIdx.x == 0)
        part[2 * G.nblk + G.neblk] = (double)epi.alpha;
    pcg_sweep<true, IMASS, PACK>(a, G, s, t, p + 2 * pcg_units<T>(G.pl), epi);
    if constexpr (PACK) {
        pcg_partial(G, t, epi.loc, part + G.nblk);
    } else {
        __shared__ double sh[32];
        const double loc = block_sum_any(epi.loc, sh);
        if (threadIdx.x == 0) part[G.nblk + t.b] = loc;
    }
}

template <class A>
__global__ void __launch_bounds__(kPcgThreads) k_pcg3(const __grid_constant__ A a, int k) {
    typedef typename A::T T;
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

// ABI layout <-> planes, congrad's systems (FP64), k_pcg3's blocks.  The solution
// is kept in planes in its own buffer while the solve runs, so it passes through p
// on the way in and through x1 on the way out:
//   0  p = x, r = Phi (:1086-1089), chi rounded where the system brings it
//   1  x = p
//   2  x1 = x in the ABI's layout
//   3  x = x1
// One launch a step for all systems: launched one by one, a kernel or copy for
// each, 128 solves on 4^4 spent 2.7 of their 4.5 ms there.
template <int STEP, class A>
__global__ void __launch_bounds__(kPcgThreads) k_pcg_move(const __grid_constant__ A a) {
    typedef typename A::V V;
    const int s = pcg_find(a.eblk0, a.nsys, (int)blockIdx.x);
    const auto& G = a.geo[a.gid[s]];
    const int64_t nu = pcg_units<typename A::T>(G.pl), kv = G.pl.kvol;
    V *p = a.vec + a.vec0[s], *r = p + nu, *x1 = r + nu, *x = a.dyn[s].x;
    const V* phi = a.dyn[s].phi;
    const double* chi = a.dyn[s].chi;
    float* chif = a.chi_out + a.chi0[s];
    constexpr int N = pcg_units_thread<typename A::T>();
    const int64_t i0 = (int64_t)((int)blockIdx.x - a.eblk0[s]) * (kPcgThreads * N) + threadIdx.x;
#pragma unroll
    for (int q = 0; q < N; q++) {
        const int64_t i = i0 + q * kPcgThreads;
        if (i >= nu) break;
        if (STEP == 0 || STEP == 2) {
            // unit (component c, s, site) of the planes; element s + Ls (site + kvol c)
            const int64_t cs = (int64_t)((uint64_t)i / (uint64_t)kv), site = i - cs * kv;
            const int c = (int)cs / G.pl.Ls;
            const int64_t e = (cs - (int64_t)c * G.pl.Ls) + G.pl.Ls * (site + kv * c);
            if (STEP == 0) {
                p[i] = x[e];
                r[i] = phi[e];
                if (chi && i < 3 * kv) chif[i] = (float)chi[i];
            } else x1[e] = x[i];
        } else if (STEP == 1) x[i] = p[i];
        else x[i] = x1[i];
    }
}

// ---- host side ---------------------------------------------------------------------
inline int pcg_sms() {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm > 0 ? nsm : 1;
}
// A batch under construction: systems are added while they fit.
template <class T, int NS = kPcgSys>
struct PcgBatch {
    typedef PcgArgs<T, NS> Args;
    typedef typename real_of<T>::type Real;
    static constexpr bool kPair = std::is_same<typename unit_of<T>::type, cpair>::value;
    static_assert(sizeof(Args) + 16 <= 32764, "beyond what kernel arguments may take");
    Args a;                           // layout; the pointers are set when it runs
    int imass = 1;
    int64_t units = 0;
    int chis = 0, parts = 0;
    PcgBatch() { memset(&a, 0, sizeof(a)); }   // padding too: it is a graph's key
    // Vectors of a system: p, r, x1 and extra more.  False: the batch is full.
    bool add(const Geom& g, Real diag, Real hpin, int apbc, int im, int extra, int nsm) {
        if (a.nsys == NS || (a.nsys > 0 && im != imass)) return false;
        int id = 0;
        while (id < a.ngeo &&
               !(a.geo[id].pl.L == g.L && a.geo[id].pl.Lt == g.Lt && a.geo[id].pl.Ls == g.Ls))
            id++;
        if (id == pcg_geos(NS)) return false;
        PcgGeo<T> G;
        if (id < a.ngeo) G = a.geo[id];
        else {
            memset(&G, 0, sizeof(G));
            G.pl = plane_plan(g, kPair, nsm, kPcgThreads);
            G.nblk = G.pl.nitem < (uint32_t)kPcgMaxBlocks ? (int)G.pl.nitem : kPcgMaxBlocks;
            const int per = kPcgThreads * pcg_units_thread<T>();
            const int64_t ne = (8 * (int64_t)G.pl.U * g.kvol + per - 1) / per;
            if (ne > (int64_t)1 << 30) return false;
            G.neblk = (int)ne;
            G.pack = 1;
        }
        if ((int64_t)a.eblk0[a.nsys] + G.neblk > (int64_t)1 << 30 ||
            (int64_t)chis + 3 * (int64_t)g.kvol > (int64_t)1 << 30)
            return false;
        if (id == a.ngeo) a.geo[a.ngeo++] = G;
        const int s = a.nsys++;
        imass = im;
        a.gid[s] = (unsigned char)id;
        a.diag[s] = diag;
        a.hpin[s] = hpin;
        a.apbc[s] = apbc != 0;
        a.vec0[s] = units;
        a.chi0[s] = chis;
        a.part0[s] = parts;
        a.blk0[s + 1] = a.blk0[s] + G.nblk;
        a.eblk0[s + 1] = a.eblk0[s] + G.neblk;
        units += (3 + extra) * vec_units(s);
        chis += 3 * g.kvol;
        parts += 2 * G.nblk + G.neblk + 1;
        return true;
    }
    // Packs a launch of more stencil blocks than fit the device at once (wave).  A
    // small lattice's plan spreads tiles of one or two warps over the SMs, which
    // suits one solve; in a batch each such block holds the place of six warps.
    // Solves to 1e-6, ms not packed and packed: 5 on 8^4 (640 blocks, 320 packed) 3.5 and
    // 2.8, 16 on 8^4 6.9 and 4.8, 32 on 6^4 9.8 and 3.8, 128 on 4^4 4.4 and 1.9.  Below
    // one wave there is nothing to gain (4 on 8^4, 512 blocks: 2.7), and where only some
    // lattices pack, the spills (PcgTile) cost 2% (20 lattices from 12^3 to 16^3: 76.7
    // and 78.2), so a launch is packed where that takes a third of its blocks away.
    void pack(int wave) {
        if constexpr (NS > 1) {
            const int before = a.blk0[a.nsys];
            for (int m = 2; m <= kPcgThreads / 32 && a.blk0[a.nsys] > wave; m++) pack_by(m);
            a.packed = a.blk0[a.nsys] <= before / 3 * 2;
            if (!a.packed) pack_by(1);
        }
    }
    // At most m blocks in one.
    void pack_by(int m) {
        for (int i = 0; i < a.ngeo; i++) {
            const int most = kPcgThreads / a.geo[i].pl.threads;
            a.geo[i].pack = m < most ? m : most;
        }
        for (int s = 0; s < a.nsys; s++)
            a.blk0[s + 1] = a.blk0[s] + (geo(s).nblk + geo(s).pack - 1) / geo(s).pack;
    }
    // The same systems with room for M only: shorter kernel arguments.
    template <int M> bool fits() const { return a.nsys <= M && a.ngeo <= pcg_geos(M); }
    template <int M> PcgBatch<T, M> cut() const {
        PcgBatch<T, M> b;
        b.imass = imass;
        b.units = units;
        b.chis = chis;
        b.parts = parts;
        b.a.nsys = a.nsys;
        b.a.ngeo = a.ngeo;
        memcpy(b.a.geo, a.geo, sizeof(b.a.geo[0]) * a.ngeo);
        for (int s = 0; s < a.nsys; s++) {
            b.a.vec0[s] = a.vec0[s];
            b.a.diag[s] = a.diag[s];
            b.a.hpin[s] = a.hpin[s];
            b.a.apbc[s] = a.apbc[s];
            b.a.chi0[s] = a.chi0[s];
            b.a.part0[s] = a.part0[s];
            b.a.gid[s] = a.gid[s];
            b.a.blk0[s + 1] = a.blk0[s + 1];
            b.a.eblk0[s + 1] = a.eblk0[s + 1];
        }
        return b;
    }
    const PcgGeo<T>& geo(int s) const { return a.geo[a.gid[s]]; }
    int64_t vec_units(int s) const {
        return 8 * (int64_t)geo(s).pl.U * geo(s).pl.kvol;
    }
};

template <class A>
void pcg_launch_chunk(const A& a, int imass, int chunk, cudaStream_t st) {
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
    auto launch = [&](auto k1, auto k2) {
        for (int k = 0; k < chunk; k++) {
            cudaLaunchKernelEx(&c, k1, a, k);
            cudaLaunchKernelEx(&c, k2, a, k);
            cudaLaunchKernelEx(&ce, k_pcg3<A>, a, k);
        }
    };
    if constexpr (A::kMost > 1) {
        if (a.packed) {
            if (imass == 3) launch(k_pcg1<A, 3, true>, k_pcg2<A, 3, true>);
            else launch(k_pcg1<A, 1, true>, k_pcg2<A, 1, true>);
            return;
        }
    }
    if (imass == 3) launch(k_pcg1<A, 3, false>, k_pcg2<A, 3, false>);
    else launch(k_pcg1<A, 1, false>, k_pcg2<A, 1, false>);
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
            (e = cudaMalloc(&dyn, sizeof(PcgDyn<T>) * kPcgSysBatch)) ||
            (e = cudaMalloc(&slot, sizeof(PcgSlot) * 2 * kPcgSysBatch)) ||
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
    template <int NS> void bind(PcgBatch<T, NS>& b, const float* chi = nullptr) {
        b.pack(pcg_sms() * kPcgPerSm);
        if (chi) memset(b.a.chi0, 0, sizeof(b.a.chi0));
        b.a.vec = vec;
        b.a.chif = chi ? chi : chif;
        b.a.chi_out = chif;
        b.a.part = part;
        b.a.dyn = dyn;
        b.a.slot = slot;
        b.a.run = run;
        b.a.hflag = hflag_dev;
    }
    // Runs a bound batch to its end.  Vectors initialised on st (congrad: by
    // pcg_congrad_enter, between begin and run); dyn: the systems' solutions, scalars
    // and caps; slots: their initial slots (FP32: |p|^2's partials as well), on return
    // the final ones.
    template <int NS>
    cudaError_t solve(const PcgBatch<T, NS>& b, const std::vector<PcgDyn<T>>& hd,
                      std::vector<PcgSlot>& slots, cudaStream_t st) {
        const cudaError_t e = begin(b, hd, slots, st);
        return e ? e : run_to_end(b, hd, slots, st);
    }
    template <int NS>
    cudaError_t begin(const PcgBatch<T, NS>& b, const std::vector<PcgDyn<T>>& hd,
                      const std::vector<PcgSlot>& slots, cudaStream_t st) {
        const int nsys = b.a.nsys;
        std::vector<PcgSlot> s2(2 * nsys);
        for (int i = 0; i < nsys; i++) s2[2 * i] = s2[2 * i + 1] = slots[i];
        const PcgRun hr{0, 0, nsys};
        cudaError_t e;
        (void)((e = cudaMemcpyAsync(dyn, hd.data(), sizeof(PcgDyn<T>) * nsys, cudaMemcpyHostToDevice, st)) ||
               (e = cudaMemcpyAsync(slot, s2.data(), sizeof(PcgSlot) * 2 * nsys, cudaMemcpyHostToDevice, st)) ||
               (e = cudaMemcpyAsync(run, &hr, sizeof(hr), cudaMemcpyHostToDevice, st)));
        return e;
    }
    template <int NS>
    cudaError_t run_to_end(const PcgBatch<T, NS>& b, const std::vector<PcgDyn<T>>& hd,
                           std::vector<PcgSlot>& slots, cudaStream_t st) {
        const int nsys = b.a.nsys;
        int cap = 0;
        for (const PcgDyn<T>& d : hd)
            if (d.niterc > cap) cap = d.niterc;
        std::vector<PcgSlot> s2(2 * nsys);
        cudaError_t e;
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
inline PcgDyn<double2> pcg_congrad_dyn(const Geom& g, float res, double2* x, const double2* phi,
                                       const double* chi = nullptr) {
    PcgDyn<double2> d;
    memset(&d, 0, sizeof(d));
    d.x = x;
    d.phi = phi;
    d.chi = chi;
    d.resid = (float)g.kferm * res * res;                    // :1076
    d.niterc = (int)(g.Ls * (int64_t)g.kvol);
    return d;
}
// The systems' vectors set up from x and Phi, and x back in the ABI's layout.
template <int STEP, class A>
void pcg_move(const A& a, cudaStream_t st) {
    k_pcg_move<STEP><<<(unsigned)a.eblk0[a.nsys], kPcgThreads, 0, st>>>(a);
    k_pcg_move<STEP + 1><<<(unsigned)a.eblk0[a.nsys], kPcgThreads, 0, st>>>(a);
    count_launches(2);
}
template <class A> void pcg_congrad_enter(const A& a, cudaStream_t st) { pcg_move<0>(a, st); }
template <class A> void pcg_congrad_leave(const A& a, cudaStream_t st) { pcg_move<2>(a, st); }
// A bound batch from begin to end.  x is the solver's own in between, so it goes
// back into the ABI's layout after an error too, and the GPU is done with it then.
template <int NS>
cudaError_t pcg_congrad(PcgWork<double2>& w, const PcgBatch<double2, NS>& b,
                        const std::vector<PcgDyn<double2>>& dyn, std::vector<PcgSlot>& slots,
                        cudaStream_t st) {
    cudaError_t e = w.begin(b, dyn, slots, st);
    if (e) return e;
    pcg_congrad_enter(b.a, st);
    e = w.run_to_end(b, dyn, slots, st);
    pcg_congrad_leave(b.a, st);
    if (e) cudaStreamSynchronize(st);
    return e;
}
inline int pcg_status(const PcgSlot& s) { return s.done == 1 ? 0 : (s.done == 2 ? 1 : 2); }

}  // namespace chdwf
