// lanczos.cu -- multi-shift solver for (M^dagger M + sigma_k) x_k = Phi over
// the Remez poles: the reference's qmrherm (rhmc/cheisdwf.f:599-745).
//
// The reference runs the Lanczos-based multi-shift recurrence and keeps two
// ndiag x kferm arrays (p_k, x_k), so every iteration streams (10 + 4n)
// spinors.  This implementation runs the SAME Lanczos process and the SAME
// scalar recurrences (d_k, mu_k, rho_k and the stopping rule, :670-715) but
// in two passes:
//   pass 1  Lanczos vectors + scalar recurrences only; 6 spinor streams per
//           iteration (M with a fused |Mq|^2, M^dagger with the fused
//           three-term update and |r|^2);
//   pass 2  regenerate the identical Lanczos vectors (same kernels, same
//           stored scalars, bit-identical) and accumulate the solution
//           x = a0 Phi + sum_j c_j q_j, where c_j = sum_k a_k y_kj and y_kj is
//           the coefficient of q_j in x_k, obtained from rho and mu by the
//           backward recurrence y_km = rho_km, y_ki = rho_ki - mu_k,i+1 y_k,i+1
//           (x_k = sum_j rho_kj p_kj, p_kj = q_j - mu_kj p_k,j-1).
// For iflag=1 only the two wall slices of each x_k are accumulated: the force
// (derivs) reads x_k and M x_k on s=1 and s=Ls only, and M x_k there depends
// on x_k on those two slices alone.
// alpha~_j = q_j^dagger M^dagger M q_j is evaluated as |M q_j|^2, which lets
// the three-term update be fused into the M^dagger kernel.
//
// The Krylov vectors are site-fastest planes (planes.cuh).
// CHDWF_STENCIL=rows selects the row-staged kernels for pass 1 instead, whose
// vectors have the ABI's layout (FP64, and FP32 with odd Ls).
#include <cmath>
#include <cstddef>
#include <cstring>
#include <type_traits>
#include <utility>

#include "chunk_graph.h"
#include "dwf_stencil.cuh"
#include "lanczos.h"
#include "planes.cuh"

namespace chdwf {

template <class T> struct LdPlainT {
    const T* __restrict__ p;
    __device__ __forceinline__ T operator()(int64_t j) const { return __ldg(p + j); }
};

__device__ __forceinline__ double2 widen(double2 v) { return v; }
__device__ __forceinline__ double2 widen(float2 v) { return make_double2((double)v.x, (double)v.y); }

template <class T>
__device__ __forceinline__ T* ring(const LzArgsT<T>& a, int j) {
    if (j < a.hcap) return a.basis + (int64_t)j * a.vs;
    const int r = j % 3;
    return r == 0 ? a.rb0 : (r == 1 ? a.rb1 : a.rb2);
}

// Element (c, s, site) of a Krylov vector, in planes or in the ABI's layout.
__device__ __forceinline__ double2 vget(const LzArgsT<double2>& a, const double2* v, int c, int s,
                                        int64_t site) {
    return a.pl ? v[((int64_t)c * a.pp.U + s) * a.g.kvol + site]
                : v[s + (int64_t)a.g.Ls * site + a.g.cs * c];
}
__device__ __forceinline__ float2 vget(const LzArgsT<float2>& a, const float2* v, int c, int s,
                                       int64_t site) {
    if (!a.pl) return v[s + (int64_t)a.g.Ls * site + a.g.cs * c];
    const float* f = reinterpret_cast<const float*>(
        v + 2 * (((int64_t)c * a.pp.U + (s >> 1)) * a.g.kvol + site));
    return make_float2(f[s & 1], f[2 + (s & 1)]);
}

static_assert(kSplitThreads == kThreads, "the reductions assume kThreads-wide blocks");

// KernelTimer class of a launch: c for FP64 Krylov vectors, c + 4 for FP32.
template <class T>
static inline int timer_class(int c) {
    return c + (std::is_same<T, float2>::value ? 4 : 0);
}

// The stop flag, read once per block: every thread of a block takes the same
// branch (the scalar step may set it while an M^dagger block starts).
__device__ __forceinline__ bool block_stopped(const LzCtl* ctl) {
    __shared__ int s_done;
    if (threadIdx.x == 0) s_done = *(const volatile int*)&ctl->done;
    __syncthreads();
    return s_done != 0;
}

// ---- thread mapping of the regenerating pass 2 on the ABI's layout -----------
// FP64 vectors: two threads per point, one per flavour (split_point /
// split_flavour).  FP32 vectors: one thread per point and both flavours.
template <class T> struct LzShape;
template <> struct LzShape<double2> {
    static constexpr bool split = true;
    static constexpr int min_blocks = 3;          // <= 85 registers: no spills
    static constexpr int unit = kSplitPoints;     // points per block
};
template <> struct LzShape<float2> {
    static constexpr bool split = false;
    static constexpr int min_blocks = 3;          // <= 85 registers a thread
    static constexpr int unit = kThreads;
};

template <class T>
__device__ __forceinline__ void lz_lane(int64_t base, int64_t* p, int* f0) {
    if (LzShape<T>::split) {
        *p = base + (threadIdx.x & (kSplitPoints - 1));
        *f0 = split_flavour();
    } else {
        *p = base + threadIdx.x;
        *f0 = 0;
    }
}

// vt = M q_j with q_j = r_j / beta_j, formed as (1/beta_j) (M r_j): one
// scaling per output element instead of one per stencil load.
template <bool DAG, int IMASS, class T>
__device__ __forceinline__ void apply_scaled(T acc[4], const T* r, typename real_of<T>::type ib,
                                             const LzArgsT<T>& a, const PointIdx& q, int f) {
    dwf_apply_flavour<DAG, IMASS>(acc, LdPlainT<T>{r}, a.g, q, f, a.chif, a.diag, a.hpin,
                                  a.apbc != 0);
#pragma unroll
    for (int d = 0; d < 4; d++) acc[d] = zscal(ib, acc[d]);
}

// Scalar recurrences of qmrherm for iteration j (cheisdwf.f:666-715), one
// lane per pole (the poles are independent), and the stopping test.  d and
// rho are the lane's pole state; returns the stop code (0: go on).
struct PoleConst {       // what the scalar step reads of the control block
    int npole, niter_cap;
    double phimod, thresh, sigma;
};
__device__ __forceinline__ PoleConst pole_const(const LzCtl* ctl) {
    const int k = threadIdx.x;
    return PoleConst{ctl->npole, ctl->niter_cap, ctl->phimod, ctl->thresh,
                     k < kMaxPoles ? ctl->sigma[k] : 0.0};
}
template <class T>
__device__ __forceinline__ int pole_step(const LzArgsT<T>& a, const PoleConst& pc, int j, double at,
                                         double beta0, double& d, double& rho) {
    LzCtl* ctl = a.ctl;
    const int k = threadIdx.x;
    if (k == 0) a.h.alphat[j] = at;
    const int n = pc.npole;
    const int64_t H = kMaxIter + 2;
    double v = -1.0;
    if (k < n) {
        const double alpha = __dadd_rn(at, pc.sigma);
        double mu = 0.0;
        if (j == 1) {
            d = alpha;
            rho = __ddiv_rn(beta0, alpha);
        } else {
            const double dm1 = d;
            mu = __ddiv_rn(beta0, dm1);
            const double dn = __dsub_rn(alpha, __dmul_rn(beta0, mu));
            d = dn;
            rho = -__ddiv_rn(__dmul_rn(__dmul_rn(mu, dm1), rho), dn);
        }
        a.h.rho[k * H + j] = rho;
        a.h.mu[k * H + j] = mu;
        v = fabs(__dmul_rn(pc.phimod, rho));
    }
    // rhomax as the sequential scan over the poles forms it: start from pole
    // 0 and take any larger value (a NaN in pole 0 stays, NaNs of the other
    // poles are skipped)
    const double v0 = __shfl_sync(0xffffffffu, v, 0);
    double m1 = k >= 1 ? v : -1.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    const double rhomax = (v0 != v0) ? v0 : fmax(v0, m1);
    int done = 0;
    if (j >= 2 && rhomax < pc.thresh) done = 1;
    else if (j >= pc.niter_cap) done = 2;
    if (!(rhomax == rhomax)) done = 3;   // NaN: stop, reported as non-finite
    if (done && k == 0) {
        ctl->m = j;
        ctl->done = done;
        if (a.hflag) {
            *(volatile int*)a.hflag = done;
            __threadfence_system();
        }
    }
    return done;
}

// alpha~_j from M(j)'s partials (the same sum, in the same order, as the
// M^dagger blocks form), the pole recurrences and the stopping test, as a
// one-block kernel beside M^dagger(j) on a side stream (row-staged pass 1).
// A converged solve stops before M(j+1).
template <class T>
__global__ void __launch_bounds__(kThreads) k_lz_pole(LzArgsT<T> a, int nb) {
    LzCtl* ctl = a.ctl;
    if (block_stopped(ctl)) return;
    const int j = ctl->it_md;
    const double at = sum_partials_any(a.part, nb);
    if (threadIdx.x == 0) ctl->it_m = j + 1;
    if (threadIdx.x < 32) {
        const int k = threadIdx.x;
        double d = k < kMaxPoles ? ctl->d[k] : 0.0, rho = k < kMaxPoles ? ctl->rho[k] : 0.0;
        pole_step(a, pole_const(ctl), j, at, a.h.beta[j], d, rho);
        if (k < ctl->npole) {
            ctl->d[k] = d;
            ctl->rho[k] = rho;
        }
    }
}

// r_{j+1} = x3 - alpha~ q_j - beta_j q_{j-1} at one point (cheisdwf.f:655)
template <class T>
__device__ __forceinline__ T three_term(const LzArgsT<T>& a, T x3, int64_t e, int j,
                                        double alphat) {
    typedef typename real_of<T>::type Real;
    const T* rj = ring(a, j);
    const T* rjm = ring(a, j - 1);
    const Real ib = (Real)a.h.invbeta[j], at = (Real)alphat, bj = (Real)a.h.beta[j];
    const T qj = zscal(ib, rj[e]);
    T v = zsub(x3, zscal(at, qj));
    if (j > 1) v = zsub(v, zscal(bj, zscal((Real)a.h.invbeta[j - 1], rjm[e])));
    return v;
}

// Force solves with a wall store: element e of r_{j+1} at point (s, site),
// component c, also goes to the wall store when s is a wall.
template <class T>
__device__ __forceinline__ void wall_put(const LzArgsT<T>& a, int j1, int s, int site, int c,
                                         T v) {
    if (a.wcap == 0 || j1 >= a.wcap) return;
    const int Ls = a.g.Ls;
    if (s != 0 && s != Ls - 1) return;
    const int64_t cs2 = 2 * (int64_t)a.g.kvol;
    a.wbasis[(int64_t)j1 * 8 * cs2 + (s == 0 ? 0 : 1) + 2 * (int64_t)site + cs2 * c] = v;
}

// ---- pass 1 on planes ----------------------------------------------------------
// Two kernels an iteration: vt = M r_j with |vt|^2, and r_{j+1} =
// (1/beta_j) M^dagger vt - alpha~_j q_j - beta_j q_{j-1} with |r_{j+1}|^2, where
// q_j = r_j/beta_j and alpha~_j = |vt|^2/beta_j^2.  Leaving vt unscaled keeps
// beta_j, a sum over the previous kernel's blocks, out of M.  Block b (of nb
// workers) takes the items b, b + nb, ... and leaves its |.|^2 partial in
// part[b] (M) or part[nb + b] (M^dagger); one more block a kernel does the
// scalar work.
//
// Kernels k = 0..15 of M and M^dagger, after k_lz_tick, are captured as a
// graph: iteration j = ctl->base + k + 1.  Programmatic dependent launch lets
// a kernel's blocks start while the previous kernel drains: they work out
// their item and read base (constant during a replay), then wait for the
// previous kernel's end.  A kernel lets its dependents start only after its
// own wait, so base has been set before any other kernel of the replay reads
// it.
__device__ __forceinline__ int pass1_begin(const LzCtl* ctl, int k, bool after_tick) {
    int base = 0;
    if (!after_tick) base = *(volatile const int*)&ctl->base;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (after_tick) base = *(volatile const int*)&ctl->base;
    return base + k + 1;
}
__global__ void k_lz_tick(LzCtl* ctl, int chunk) {
    ctl->base = ctl->next;
    ctl->next += chunk;
}

// The sum of a kernel's nb partials and the recurrence's scalars, in two
// steps: asynchronous copies into shared memory when the kernel starts, in
// front of its stencil loads and holding no registers, and the sum, in one
// order for all blocks, where it is first needed, after the first unit.
// Loaded and summed in one step there, the L2 round trip made the kernel
// about 2 us longer (24^3x24): all blocks run one wave and wait together.
// Dynamic shared memory: nb + 3 doubles.
extern __shared__ double lz_smem[];
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
struct PartSum {
    __device__ __forceinline__ static void start(const double* part, int n, const double* x0,
                                                 const double* x1, const double* x2) {
        for (int i = (int)threadIdx.x; i < n; i += (int)blockDim.x) cp_async8(lz_smem + i, part + i);
        if (threadIdx.x == 0 && x0) {
            cp_async8(lz_smem + n, x0);
            cp_async8(lz_smem + n + 1, x1);
            cp_async8(lz_smem + n + 2, x2);
        }
    }
    __device__ __forceinline__ static double total(int n) {
        __shared__ double sh[32];
        __shared__ double res;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        double s = 0.0;
        for (int i = (int)threadIdx.x; i < n; i += (int)blockDim.x) s += lz_smem[i];
        s = block_sum_any(s, sh);
        if (threadIdx.x == 0) res = s;
        __syncthreads();
        return res;
    }
};
// alpha~_j from |vt|^2 = |M r_j|^2
__device__ __forceinline__ double alpha_of(double s, double ibj) { return s * ibj * ibj; }

template <class T>
struct PlaneM {
    typedef typename unit_of<T>::type V;
    V* vt;
    int done;              // the solve has stopped: no item is begun
    double loc;
    __device__ __forceinline__ bool operator()(V acc[4], int64_t e, int64_t cst, uint32_t o,
                                               bool act, int, uint32_t) {
        if (!act) return true;
        // |vt|^2 is summed in FP64 from the first term: a pair's partial sum
        // in FP32 made the FP32 force solves 7% longer (alpha~ and beta steer
        // the recurrences)
#pragma unroll
        for (int d = 0; d < 4; d++) {
            st_unit(unit_at(vt + e + d * cst, o), acc[d]);
            loc += unit_norm2(acc[d]);
        }
        return true;
    }
};

// Element of a unit that lies on wall sw (0: s = 1, 1: s = Ls).
__device__ __forceinline__ double2 unit_wall(double2 v, int, int) { return v; }
__device__ __forceinline__ float2 unit_wall(const cpair& v, int sw, int Ls) {
    return cpair_pt(v, sw == 0 ? 0 : (Ls & 1 ? 0 : 1));
}

template <class T, bool WALLS>
struct PlaneMd {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    const LzArgsT<T>& a;
    const V *rj, *rjm;
    V* rn;
    int nb, j, done;
    bool have;
    double loc;
    Real c0, c1, c2;                  // 1/beta_j, -alpha~/beta_j, -beta_j/beta_{j-1}
    __device__ __forceinline__ void scalars(double at, double bj, double ibj, double ibm) {
        c0 = (Real)ibj;
        c1 = (Real)(-at * ibj);
        c2 = (Real)(-bj * ibm);
        have = true;
    }
    __device__ __forceinline__ void ready() {
        if (have) return;
        const double s = PartSum::total(nb), ibj = lz_smem[nb + 1];
        scalars(alpha_of(s, ibj), lz_smem[nb], ibj, lz_smem[nb + 2]);
    }
    __device__ __forceinline__ bool operator()(V acc[4], int64_t e, int64_t cst, uint32_t o,
                                               bool act, int u, uint32_t site) {
        // FP64: q_j and q_{j-1} are loaded in front of the sum's block barriers.
        // FP32: behind them; the stencil of a pair leaves no registers for
        // them (100 bytes of spills; 24^3x24 M^dagger 2.5 us longer, against
        // 1.9 us shorter for FP64 20^3x20)
        constexpr bool EARLY = std::is_same<T, double2>::value;
        V q[4], qm[4];
        if (EARLY) {
#pragma unroll
            for (int d = 0; d < 4; d++) {
                q[d] = ld_unit(unit_at(rj + e + d * cst, o));
                qm[d] = j > 1 ? ld_unit(unit_at(rjm + e + d * cst, o)) : V{};
            }
        }
        ready();
        if (!act) return true;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            // r_{j+1} = x3 - alpha~ q_j - beta_j q_{j-1} (cheisdwf.f:655)
            if (!EARLY) {
                q[d] = ld_unit(unit_at(rj + e + d * cst, o));
                qm[d] = j > 1 ? ld_unit(unit_at(rjm + e + d * cst, o)) : V{};
            }
            V v = zaxpy(c1, q[d], zscal2(c0, acc[d]));
            if (j > 1) v = zaxpy(c2, qm[d], v);
            st_unit(unit_at(rn + e + d * cst, o), v);
            loc += unit_norm2(v);
            if (WALLS && j + 1 < a.wcap && (u == 0 || u == a.pp.U - 1)) {
                // the two wall slices of r_{j+1}, element (wall, site, c)
                const int64_t cs2 = 2 * (int64_t)a.g.kvol;
                const int c = (int)(e >= 4 * cst ? 4 : 0) + d;
                T* w = a.wbasis + (int64_t)(j + 1) * 8 * cs2 + 2 * (int64_t)site + cs2 * c;
                if (u == 0) w[0] = unit_wall(v, 0, a.g.Ls);
                if (u == a.pp.U - 1) w[1] = unit_wall(v, 1, a.g.Ls);
            }
        }
        return true;
    }
};

template <class T, int IMASS>
__device__ __forceinline__ void plane_phase_M(const LzArgsT<T>& a, const PlaneThread& th,
                                              int b, int nb, PlaneM<T>& epi, const T* rj) {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    for (uint32_t it = (uint32_t)b; it < a.pp.nitem && !epi.done; it += (uint32_t)nb)
        plane_item<false, IMASS>(reinterpret_cast<const V*>(rj), a.pp, th, it, a.chif, (Real)a.diag,
                                 (Real)a.hpin, a.apbc != 0, epi);
}
template <class T, int IMASS, bool WALLS>
__device__ __forceinline__ void plane_phase_Md(const LzArgsT<T>& a, const PlaneThread& th,
                                               int b, int nb, PlaneMd<T, WALLS>& epi) {
    typedef typename unit_of<T>::type V;
    typedef typename real_of<T>::type Real;
    for (uint32_t it = (uint32_t)b; it < a.pp.nitem && !epi.done; it += (uint32_t)nb)
        plane_item<true, IMASS>(reinterpret_cast<const V*>(a.vt), a.pp, th, it, a.chif,
                                (Real)a.diag, (Real)a.hpin, a.apbc != 0, epi);
}

// Pass 1 (REGEN false, k0 the place in the replay): iteration j unless the
// solve has stopped.  Block 0 is
// the scalar block: it forms beta_j from M^dagger(j-1)'s partials (beta_1
// comes from the source).  The regenerating pass 2 (REGEN true, k0 = j) takes
// every scalar from the history and has no scalar block.
template <class T, int IMASS, bool REGEN>
__global__ void __maxnreg__(kPlaneRegs) k_lz1_M(LzArgsT<T> a, int k0) {
    typedef typename unit_of<T>::type V;
    LzCtl* ctl = a.ctl;
    constexpr int X = REGEN ? 0 : 1;
    const int nb = (int)gridDim.x - X, b = (int)blockIdx.x - X;
    const PlaneThread th = plane_thread(a.pp);
    if (REGEN) pdl_wait();
    const int j = REGEN ? k0 : pass1_begin(ctl, k0, k0 == 0);
    PlaneM<T> em{reinterpret_cast<V*>(a.vt), REGEN ? 0 : *(volatile int*)&ctl->done, 0.0};
    if (!REGEN && b < 0) {
        if (em.done || j == 1) return;
        PartSum::start(a.part + nb, nb, nullptr, nullptr, nullptr);
        const double s = PartSum::total(nb);
        if (threadIdx.x == 0) {
            const double beta = sqrt(s);
            a.h.beta[j] = beta;
            a.h.invbeta[j] = 1.0 / beta;
        }
        return;
    }
    plane_phase_M<T, IMASS>(a, th, b, nb, em, ring(a, j));
    if (REGEN || em.done) return;
    __shared__ double sh[32];
    const double loc = block_sum_any(em.loc, sh);
    if (threadIdx.x == 0) a.part[b] = loc;
}

// Block 0 is the scalar step of iteration j (alpha~_j, the pole recurrences,
// the stopping test).  The step, two L2 round trips and two dependent
// divisions, ends long before the workers do, and the next M sees its stop
// flag.  (As phases of one cooperative kernel with grid barriers the two
// kernels were slower: a barrier and the sum after it take 1.9 us at 144
// blocks and 3.8 us at 577, a kernel boundary about 1 us.)
template <class T, int IMASS, bool WALLS, bool REGEN>
__global__ void __maxnreg__(kPlaneRegs) k_lz1_Md(LzArgsT<T> a, int k0) {
    typedef typename unit_of<T>::type V;
    LzCtl* ctl = a.ctl;
    constexpr int X = REGEN ? 0 : 1;
    const int nb = (int)gridDim.x - X, b = (int)blockIdx.x - X;
    const PlaneThread th = plane_thread(a.pp);
    if (REGEN) pdl_wait();
    const int j = REGEN ? k0 : pass1_begin(ctl, k0, false);
    // M(j) ran if the solve had not stopped before iteration j: m is set with
    // done, by the scalar block of M^dagger(m)
    const int m = REGEN ? j : *(volatile int*)&ctl->m;
    // invbeta[0] is 0, so c2 is 0 for j = 1
    if (!REGEN)
        PartSum::start(a.part, nb, a.h.beta + j, a.h.invbeta + j, a.h.invbeta + j - 1);
    PlaneMd<T, WALLS> ed{a, reinterpret_cast<const V*>(ring(a, j)),
                         reinterpret_cast<const V*>(ring(a, j - 1)),
                         reinterpret_cast<V*>(ring(a, j + 1)), nb, j, m != 0 && m < j, false, 0.0};
    if (!REGEN && b < 0) {
        if (ed.done) return;
        const int k = threadIdx.x;
        double d = 0.0, rho = 0.0;
        if (k < kMaxPoles) {
            d = ctl->d[k];
            rho = ctl->rho[k];
        }
        const PoleConst pc = pole_const(ctl);
        const double s = PartSum::total(nb);
        if (k < 32) {
            pole_step(a, pc, j, alpha_of(s, lz_smem[nb + 1]), lz_smem[nb], d, rho);
            if (k < pc.npole) {
                ctl->d[k] = d;
                ctl->rho[k] = rho;
            }
        }
        return;
    }
    if (REGEN)
        ed.scalars(a.h.alphat[j], a.h.beta[j], a.h.invbeta[j], j > 1 ? a.h.invbeta[j - 1] : 0.0);
    plane_phase_Md<T, IMASS, WALLS>(a, th, b, nb, ed);
    if (REGEN || ed.done) return;
    __shared__ double sh[32];
    const double loc = block_sum_any(ed.loc, sh);
    if (threadIdx.x == 0) a.part[nb + b] = loc;
}

// Regenerating pass 2, iflag 1: x_k += y_kj q_j on the two wall slices of every
// pole's x_k, from r_j in planes.
template <class T>
__global__ void __launch_bounds__(kThreads) k_lzp_acc_walls(LzArgsT<T> a, int j) {
    typedef typename real_of<T>::type Real;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t cs2 = 2 * (int64_t)a.g.kvol, kf2 = 8 * cs2;
    if (t >= kf2) return;
    const Real ib = (Real)a.h.invbeta[j];
    const int c = (int)(t / cs2);
    const int64_t r = t - c * cs2;
    const double2 q =
        widen(zscal(ib, vget(a, ring(a, j), c, (r & 1) ? a.g.Ls - 1 : 0, r >> 1)));
    const int64_t H = kMaxIter + 2;
    for (int k = 0; k < a.npole; k++) {
        const double y = a.h.y[k * H + j];
        double2 xv = a.xw[k * kf2 + t];
        xv.x += y * q.x;
        xv.y += y * q.y;
        a.xw[k * kf2 + t] = xv;
    }
}

// ---- pass 1 on staged rows ---------------------------------------------------
// The same two kernels with the stencil's input rows staged in shared memory
// (row_stage.cuh): a persistent grid of the blocks that fit on all SMs at
// once, each walking a contiguous range of output rows of one flavour at a
// time.  Per element the operation sequence is that of k_lz1_M / k_lz1_Md,
// so the vectors are the same bits and the regenerating pass 2 reproduces
// them.  A copy that does not arrive within the bounded wait stops the solve
// with done = 4 (reported as a CUDA error).
__device__ __forceinline__ void row_fail(LzCtl* ctl, int* hflag) {
    ctl->done = 4;
    ctl->m = ctl->it_m;
    if (hflag) {
        *(volatile int*)hflag = 4;
        __threadfence_system();
    }
}

// PPT adjacent elements of a global vector
template <class T, int PPT> struct LzLd;
template <class T> struct LzLd<T, 1> {
    __device__ __forceinline__ static void get(const T* p, T* v) { v[0] = *p; }
    __device__ __forceinline__ static void put(T* p, const T* v) { *p = v[0]; }
};

template <class T, int IMASS, int PPT>
struct LzRowsM {
    typedef typename real_of<T>::type Real;
    const LzArgsT<T>& a;
    const T* rj;
    Real ib;
    double loc;
    RowWall<T, PPT> rw;
    __device__ __forceinline__ void pre(int f, int t, int y, int x, int s) {
        row_wall_prefetch<false, PPT>(rw, rj, a.g, f, t, y, x, s, a.chif);
    }
    __device__ __forceinline__ void compute(const T* c, const T* yp, const T* ym, const T* tps,
                                            const T* tms, int f, int t, int y, int x, int s,
                                            int i, int ixp, int ixm) {
        const Geom& g = a.g;
        const int site = x + g.L * (y + g.L * t);
        T acc[PPT][4];
        dwf_apply_rows<false, IMASS, PPT>(acc, c, yp, ym, tps, tms, a.rp.Lrow, i, ixp, ixm, s,
                                          site, t, rw, g, f, a.diag, a.hpin, a.apbc != 0);
        const int64_t p0 = s + (int64_t)g.Ls * site;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            T v[PPT];
#pragma unroll
            for (int p = 0; p < PPT; p++) {
                v[p] = zscal(ib, acc[p][d]);
                const double2 w = widen(v[p]);
                loc += w.x * w.x + w.y * w.y;
            }
            LzLd<T, PPT>::put(a.vt + p0 + g.cs * (d + 4 * f), v);
        }
    }
};

template <class T, int IMASS, int PPT>
__global__ void __maxnreg__(kRowRegs) k_lz1_M_rows(LzArgsT<T> a) {
    extern __shared__ __align__(128) unsigned char row_smem[];
    LzCtl* ctl = a.ctl;
    if (block_stopped(ctl)) return;
    const int j = ctl->it_m;
    const int nb = gridDim.x;
    const double bj = j == 1 ? a.h.beta[1] : sqrt(sum_partials_any(a.part + nb, nb));
    const double ibj = j == 1 ? a.h.invbeta[1] : 1.0 / bj;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->it_md = j;
        if (j > 1) {
            a.h.beta[j] = bj;
            a.h.invbeta[j] = ibj;
        }
    }
    LzRowsM<T, IMASS, PPT> body{a, ring(a, j), (typename real_of<T>::type)ibj, 0.0};
    const bool ok = row_sweep<T, PPT>(a.g, a.rp, row_smem, body.rj, body);
    __shared__ double sh[32];
    const double loc = block_sum_any(body.loc, sh);
    if (threadIdx.x == 0) {
        a.part[blockIdx.x] = loc;
        if (!ok) row_fail(ctl, a.hflag);
    }
}

template <class T, int IMASS, bool WALLS, int PPT>
struct LzRowsMd {
    typedef typename real_of<T>::type Real;
    const LzArgsT<T>& a;
    const T* rj;
    const T* rjm;
    T* rn;
    int j;
    Real ib, at, bj, ibm;
    double loc;
    T cj[4][PPT], cm[4][PPT];
    RowWall<T, PPT> rw;
    // q_j and q_{j-1} at the thread's points (streamed, not staged) and the
    // wall operands
    __device__ __forceinline__ void pre(int f, int t, int y, int x, int s) {
        const Geom& g = a.g;
        const int64_t e0 = (int64_t)x * g.Ls + s + (int64_t)g.L * g.Ls * (y + (int64_t)g.L * t);
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int64_t po = g.cs * (d + 4 * f);
            LzLd<T, PPT>::get(rj + e0 + po, cj[d]);
            if (j > 1) LzLd<T, PPT>::get(rjm + e0 + po, cm[d]);
        }
        row_wall_prefetch<true, PPT>(rw, a.vt, g, f, t, y, x, s, a.chif);
    }
    __device__ __forceinline__ void compute(const T* c, const T* yp, const T* ym, const T* tps,
                                            const T* tms, int f, int t, int y, int x, int s,
                                            int i, int ixp, int ixm) {
        const Geom& g = a.g;
        const int site = x + g.L * (y + g.L * t);
        T acc[PPT][4];
        dwf_apply_rows<true, IMASS, PPT>(acc, c, yp, ym, tps, tms, a.rp.Lrow, i, ixp, ixm, s,
                                         site, t, rw, g, f, a.diag, a.hpin, a.apbc != 0);
        const int64_t p0 = s + (int64_t)g.Ls * site;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            T v[PPT];
#pragma unroll
            for (int p = 0; p < PPT; p++) {
                // r_{j+1} = x3 - alpha~ q_j - beta_j q_{j-1}, as three_term (:655)
                const T qj = zscal(ib, cj[d][p]);
                v[p] = zsub(acc[p][d], zscal(at, qj));
                if (j > 1) v[p] = zsub(v[p], zscal(bj, zscal(ibm, cm[d][p])));
                if (WALLS) wall_put(a, j + 1, s + p, site, d + 4 * f, v[p]);
                const double2 w = widen(v[p]);
                loc += w.x * w.x + w.y * w.y;
            }
            LzLd<T, PPT>::put(rn + p0 + g.cs * (d + 4 * f), v);
        }
    }
};

template <class T, int IMASS, bool WALLS, int PPT>
__global__ void __maxnreg__(kRowRegs) k_lz1_Md_rows(LzArgsT<T> a) {
    typedef typename real_of<T>::type Real;
    extern __shared__ __align__(128) unsigned char row_smem[];
    LzCtl* ctl = a.ctl;
    if (block_stopped(ctl)) return;
    const int j = ctl->it_md;
    const int nb = gridDim.x;
    const double at = sum_partials_any(a.part, nb);
    LzRowsMd<T, IMASS, WALLS, PPT> body{a, ring(a, j), ring(a, j - 1), ring(a, j + 1), j,
                                        (Real)a.h.invbeta[j], (Real)at, (Real)a.h.beta[j],
                                        (Real)(j > 1 ? a.h.invbeta[j - 1] : 0.0), 0.0};
    const bool ok = row_sweep<T, PPT>(a.g, a.rp, row_smem, a.vt, body);
    __shared__ double sh[32];
    const double loc = block_sum_any(body.loc, sh);
    if (threadIdx.x == 0) {
        a.part[nb + blockIdx.x] = loc;
        if (!ok) row_fail(ctl, a.hflag);
    }
}

// ---- pass 2 on the ABI's layout: regenerate q_j and accumulate ---------------
// (row-staged solves).  One pass per block; the solution update of one
// element of x (iflag 0) or of the wall fields (iflag 1).
template <class T, int IFLAG>
__device__ __forceinline__ void lz2_accumulate(const LzArgsT<T>& a, int j, const T* rj,
                                               typename real_of<T>::type ib, int64_t p,
                                               const PointIdx& q, int c0, int nc) {
    if (IFLAG == 0) {
        const double cj = a.h.c[j];
        for (int c = c0; c < c0 + nc; c++) {
            const int64_t e = p + a.g.cs * c;
            const double2 qj = widen(zscal(ib, rj[e]));
            double2 xv = a.x[e];
            xv.x += cj * qj.x;
            xv.y += cj * qj.y;
            a.x[e] = xv;
        }
    } else {
        const int Ls = a.g.Ls;
        if (q.s != 0 && q.s != Ls - 1) return;
        const int sw = (q.s == 0) ? 0 : 1;
        const int64_t cs2 = 2 * (int64_t)a.g.kvol, kf2 = 8 * cs2;
        const int64_t H = kMaxIter + 2;
        const int n = a.npole;
        double2 qv[8];
#pragma unroll
        for (int c = 0; c < 8; c++)
            if (c < nc) qv[c] = widen(zscal(ib, rj[p + a.g.cs * (c + c0)]));
        const int64_t base = sw + 2 * (int64_t)q.site + cs2 * c0;
        for (int k = 0; k < n; k++) {
            const double y = a.h.y[k * H + j];
            double2* xk = a.xw + k * kf2 + base;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                if (c >= nc) break;
                double2 xv = xk[cs2 * c];
                xv.x += y * qv[c].x;
                xv.y += y * qv[c].y;
                xk[cs2 * c] = xv;
            }
        }
    }
}

template <class T, int IMASS, int IFLAG>
__global__ void __launch_bounds__(kThreads, LzShape<T>::min_blocks)
    k_lz2_M(LzArgsT<T> a, int j, int apply) {
    typedef typename real_of<T>::type Real;
    typedef LzShape<T> S;
    constexpr int NF = S::split ? 1 : 2;
    int64_t p;
    int f0;
    lz_lane<T>((int64_t)blockIdx.x * S::unit, &p, &f0);
    if (p >= a.g.npts) return;
    const PointIdx q = point_of(a.g, p);
    const Real ib = (Real)a.h.invbeta[j];
    const T* rj = ring(a, j);
    if (apply) {
#pragma unroll
        for (int f = f0; f < f0 + NF; f++) {
            T acc[4];
            apply_scaled<false, IMASS>(acc, rj, ib, a, q, f);
#pragma unroll
            for (int d = 0; d < 4; d++) a.vt[p + a.g.cs * (d + 4 * f)] = acc[d];
        }
    }
    lz2_accumulate<T, IFLAG>(a, j, rj, ib, p, q, 4 * f0, 4 * NF);
}

template <class T, int IMASS>
__global__ void __launch_bounds__(kThreads, LzShape<T>::min_blocks)
    k_lz2_Md(LzArgsT<T> a, int j) {
    typedef LzShape<T> S;
    constexpr int NF = S::split ? 1 : 2;
    int64_t p;
    int f0;
    lz_lane<T>((int64_t)blockIdx.x * S::unit, &p, &f0);
    if (p >= a.g.npts) return;
    const PointIdx q = point_of(a.g, p);
    T* rn = ring(a, j + 1);
#pragma unroll
    for (int f = f0; f < f0 + NF; f++) {
        T acc[4];
        dwf_apply_flavour<true, IMASS>(acc, LdPlainT<T>{a.vt}, a.g, q, f, a.chif, a.diag, a.hpin,
                                       a.apbc != 0);
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int64_t e = p + a.g.cs * (d + 4 * f);
            rn[e] = three_term(a, acc[d], e, j, a.h.alphat[j]);
        }
    }
}

// ---- pass 2 from the stored basis ---------------------------------------
// x += sum_j c_j q_j, q_j = r_j / beta_j, j = 1..m, in j order per element
// (the same sequence of operations as the regenerating pass 2).  A thread
// takes one 16-byte unit of the vectors (planes: one FP64 or two FP32
// elements; the ABI's layout: one element), so the stored vectors, m of them
// against one read and write of x, stream coalesced.  RING: the vectors are in
// the residual ring (regenerating pass 2).
template <class T> struct AccUnit;
template <> struct AccUnit<double2> {
    static constexpr int N = 1;
    __device__ __forceinline__ static void get(const LzArgsT<double2>&, const double2* v,
                                               int64_t i, double2* q) {
        q[0] = __ldg(v + i);
    }
};
template <> struct AccUnit<float2> {
    static constexpr int N = 2;
    __device__ __forceinline__ static void get(const LzArgsT<float2>& a, const float2* v,
                                               int64_t i, float2* q) {
        if (a.pl) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(v) + i);
            const cpair p{make_float2(f.x, f.y), make_float2(f.z, f.w)};
            q[0] = cpair_pt(p, 0);
            q[1] = cpair_pt(p, 1);
        } else {
            q[0] = __ldg(v + i);
            q[1] = make_float2(0.0f, 0.0f);
        }
    }
};
// Units of a stored vector, and the x elements of unit i: the first one's
// index and the number of elements (x is in the ABI's layout, the elements
// of a unit adjacent).
template <class T>
__host__ __device__ __forceinline__ int64_t acc_units(const LzArgsT<T>& a) {
    return a.pl ? 8 * (int64_t)a.pp.U * a.g.kvol : a.g.kferm;
}
template <class T>
__device__ __forceinline__ int64_t acc_elem(const LzArgsT<T>& a, int64_t i, int* n) {
    constexpr int N = AccUnit<T>::N;
    *n = 1;
    if (!a.pl) return i;
    const int64_t cu = i / a.g.kvol, site = i - cu * a.g.kvol;
    const int c = (int)(cu / a.pp.U), u = (int)(cu - (int64_t)c * a.pp.U);
    if (N == 2 && 2 * u + 1 < a.g.Ls) *n = 2;
    return (int64_t)N * u + (int64_t)a.g.Ls * site + a.g.cs * c;
}

template <class T, bool RING>
__global__ void __launch_bounds__(kThreads) k_lz_accum_x(LzArgsT<T> a, int j0, int j1) {
    typedef typename real_of<T>::type Real;
    constexpr int N = AccUnit<T>::N;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= acc_units(a)) return;
    int n;
    const int64_t e = acc_elem(a, i, &n);
    double2 xv[N];
    xv[0] = a.x[e];
    if (N == 2) xv[N - 1] = n == 2 ? a.x[e + 1] : make_double2(0.0, 0.0);
#pragma unroll 4
    for (int j = j0; j <= j1; j++) {
        T q[N];
        AccUnit<T>::get(a, RING ? ring(a, j) : a.basis + j * a.vs, i, q);
        const Real ib = (Real)a.h.invbeta[j];
        const double cj = a.h.c[j];
#pragma unroll
        for (int k = 0; k < N; k++) {
            const double2 qj = widen(zscal(ib, q[k]));
            xv[k].x += cj * qj.x;
            xv[k].y += cj * qj.y;
        }
    }
    a.x[e] = xv[0];
    if (N == 2 && n == 2) a.x[e + 1] = xv[N - 1];
}

template <class T>
static unsigned lz_direct_blocks(int64_t npts) {
    return (unsigned)((npts + LzShape<T>::unit - 1) / LzShape<T>::unit);
}

// ---- between the passes: y_kj and c_j -------------------------------------
// The backward recurrence is sequential in i for each pole: the block stages
// rho and mu in shared memory a chunk of iterations at a time, so each pole's
// lane runs its chain from shared memory; c_j of the chunk follows in
// parallel, summed over the poles in order.
__global__ void __launch_bounds__(kThreads) k_lz_coeffs(LzCtl* ctl, LzHist h, int iflag) {
    constexpr int CH = 48;
    __shared__ double s_rho[kMaxPoles][CH], s_mu[kMaxPoles][CH], s_y[kMaxPoles][CH];
    __shared__ double s_anum[kMaxPoles];
    const int m = ctl->m, n = ctl->npole;
    const int64_t H = kMaxIter + 2;
    const int k = threadIdx.x;
    if (k < n) s_anum[k] = ctl->anum[k];
    double y = 0.0;
    for (int hi = m; hi >= 1; hi -= CH) {
        const int lo = hi - CH + 1 > 1 ? hi - CH + 1 : 1;
        const int len = hi - lo + 1;
        for (int t = threadIdx.x; t < n * len; t += blockDim.x) {
            const int kk = t / len, o = t - kk * len;
            s_rho[kk][o] = h.rho[kk * H + lo + o];
            s_mu[kk][o] = h.mu[kk * H + lo + o + 1];
        }
        __syncthreads();
        if (k < n) {
            for (int o = len - 1; o >= 0; o--) {
                const int i = lo + o;
                y = i == m ? s_rho[k][o] : __dsub_rn(s_rho[k][o], __dmul_rn(s_mu[k][o], y));
                s_y[k][o] = y;
                h.y[k * H + i] = y;
            }
        }
        __syncthreads();
        if (iflag == 0) {
            for (int o = threadIdx.x; o < len; o += blockDim.x) {
                double c = 0.0;
                for (int kk = 0; kk < n; kk++) c = __dadd_rn(c, __dmul_rn(s_anum[kk], s_y[kk][o]));
                h.c[lo + o] = c;
            }
        }
        __syncthreads();
    }
}

// r_1 = Phi in the vector precision and layout; partial sums of |r_1|^2.  In
// planes a thread takes one unit: its reads of Phi are Ls elements apart from
// its neighbours', once per solve.
template <class T>
__device__ __forceinline__ T narrow(double2 v) {
    return zmake<T>((typename real_of<T>::type)v.x, (typename real_of<T>::type)v.y);
}
template <class T>
__global__ void k_lz_source(LzArgsT<T> a, T* __restrict__ r1, const double2* __restrict__ phi,
                            double* __restrict__ part) {
    __shared__ double sh[kThreads / 32];
    constexpr bool F32 = std::is_same<T, float2>::value;
    double s = 0.0;
    const int64_t n = a.pl ? 8 * (int64_t)a.pp.U * a.g.kvol : a.g.kferm;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        if (!a.pl) {
            const T t = narrow<T>(phi[i]);
            r1[i] = t;
            const double2 w = widen(t);
            s += w.x * w.x + w.y * w.y;
            continue;
        }
        const int64_t cu = i / a.g.kvol, site = i - cu * a.g.kvol;
        const int c = (int)(cu / a.pp.U), u = (int)(cu - (int64_t)c * a.pp.U);
        const double2* src = phi + (int64_t)a.g.Ls * site + a.g.cs * c;
        if constexpr (F32) {
            const float2 z = make_float2(0.0f, 0.0f);
            const float2 p0 = narrow<T>(src[2 * u]);
            const float2 p1 = 2 * u + 1 < a.g.Ls ? narrow<T>(src[2 * u + 1]) : z;
            const cpair v{make_float2(p0.x, p1.x), make_float2(p0.y, p1.y)};
            st_unit(reinterpret_cast<cpair*>(r1) + i, v);
            s += unit_norm2(v);
        } else {
            const double2 v = src[u];
            r1[i] = v;
            s += v.x * v.x + v.y * v.y;
        }
    }
    s = block_sum<kThreads>(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void k_lz_init(LzCtl* ctl, LzHist h, const double* part, int nb) {
    __shared__ double sh[kThreads / 32];
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) s += part[i];
    s = block_sum<kThreads>(s, sh);
    if (threadIdx.x == 0) {
        const double b = sqrt(s);
        h.beta[1] = b;
        h.invbeta[1] = 1.0 / b;
        h.invbeta[0] = 0.0;
        ctl->phimod = b;
    }
}

// Pass 1 on planes.  Algorithmic bytes: M reads q, writes vt; M^dagger reads
// vt, r_j, r_{j-1} and writes r_{j+1}; both read chi as REAL*4.
// dep: programmatic dependent launch (see pass1_begin).
template <class... P, class... A>
static void launch_grid(bool dep, void (*k)(P...), unsigned grid, unsigned nt, size_t smem,
                        cudaStream_t st, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(nt);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = dep ? 1 : 0;
    cudaLaunchKernelEx(&c, k, P(args)...);
}
template <class... P, class... A>
static void launch_dep(bool dep, void (*k)(P...), unsigned nb, unsigned nt, cudaStream_t st,
                       A... args) {
    // nb workers and the scalar block
    launch_grid(dep, k, nb + 1, nt, sizeof(double) * (nb + 3), st, args...);
}
template <class T, int IMASS>
static void launch_pass1_planes(const LzArgsT<T>& a, unsigned nb, int k0, int chunk, cudaStream_t st,
                                KernelTimer* tm) {
    const double V = (double)a.g.kferm * sizeof(T), chi = 12.0 * a.g.kvol;
    const unsigned nt = (unsigned)a.pp.threads;
    const bool dep = !tm || !tm->enabled;   // events need the kernel's own start
    if (k0 == 0) k_lz_tick<<<1, 1, 0, st>>>(a.ctl, chunk);
    if (tm) tm->begin(timer_class<T>(0), st, 2 * V + chi);
    launch_dep(dep, k_lz1_M<T, IMASS, false>, nb, nt, st, a, k0);
    if (tm) tm->end(st);
    if (tm) tm->begin(timer_class<T>(1), st, 4 * V + chi);
    if (a.wcap > 0) launch_dep(dep, k_lz1_Md<T, IMASS, true, false>, nb, nt, st, a, k0);
    else launch_dep(dep, k_lz1_Md<T, IMASS, false, false>, nb, nt, st, a, k0);
    if (tm) tm->end(st);
}

// Worker blocks of pass 1: the blocks of both kernels that are resident at
// once (one fewer: the scalar block), at most one per work item.
template <class T, int IMASS>
static unsigned pass1_workers(const PlanePlan& pp, int nsm) {
    const void* k[3] = {(const void*)k_lz1_M<T, IMASS, false>,
                        (const void*)k_lz1_Md<T, IMASS, false, false>,
                        (const void*)k_lz1_Md<T, IMASS, true, false>};
    int64_t res = kMaxPartBlocks;
    for (const void* f : k) {
        int per_sm = 0;
        const int64_t most = (int64_t)(24 / (pp.threads / 32)) * nsm;   // by registers
        const size_t smem = sizeof(double) * (size_t)((most < res ? most : res) + 3);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, pp.threads, smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        const int64_t r = (int64_t)per_sm * nsm - 1;
        if (r < res) res = r;
    }
    return res < 1 ? 0 : (unsigned)(res < (int64_t)pp.nitem ? res : (int64_t)pp.nitem);
}

// Row-staged pass 1 (same protocol: M, the scalar step on the side stream,
// M^dagger).  Grid: the blocks that fit on all SMs at once.
template <class T, int IMASS, int PPT>
static void launch_pass1_rows_ppt(const LzArgsT<T>& a, unsigned nb, cudaStream_t st,
                                  const LzSide& side, KernelTimer* tm) {
    const double V = (double)a.g.kferm * sizeof(T), chi = 12.0 * a.g.kvol;
    const unsigned nt = (unsigned)a.rp.nthreads, sm = a.rp.smem;
    if (tm) tm->begin(timer_class<T>(0), st, 2 * V + chi);
    k_lz1_M_rows<T, IMASS, PPT><<<nb, nt, sm, st>>>(a);
    if (tm) tm->end(st);
    cudaEventRecord(side.fork, st);
    cudaStreamWaitEvent(side.stream, side.fork, 0);
    k_lz_pole<T><<<1, kThreads, 0, side.stream>>>(a, (int)nb);
    cudaEventRecord(side.join, side.stream);
    if (tm) tm->begin(timer_class<T>(1), st, 4 * V + chi);
    if (a.wcap > 0) k_lz1_Md_rows<T, IMASS, true, PPT><<<nb, nt, sm, st>>>(a);
    else k_lz1_Md_rows<T, IMASS, false, PPT><<<nb, nt, sm, st>>>(a);
    if (tm) tm->end(st);
    cudaStreamWaitEvent(st, side.join, 0);
}

// One point a thread: the FP64 solves and odd-Ls FP32 solves.
template <class T, int IMASS>
static void launch_pass1_rows(const LzArgsT<T>& a, unsigned nb, cudaStream_t st,
                              const LzSide& side, KernelTimer* tm) {
    launch_pass1_rows_ppt<T, IMASS, 1>(a, nb, st, side, tm);
}

// The six pass-1 row kernels of one precision and thread shape.
template <class T, int PPT>
static void lz_rows_kernels(const void* kern[6]) {
    kern[0] = (const void*)k_lz1_M_rows<T, 1, PPT>;
    kern[1] = (const void*)k_lz1_M_rows<T, 3, PPT>;
    kern[2] = (const void*)k_lz1_Md_rows<T, 1, false, PPT>;
    kern[3] = (const void*)k_lz1_Md_rows<T, 1, true, PPT>;
    kern[4] = (const void*)k_lz1_Md_rows<T, 3, false, PPT>;
    kern[5] = (const void*)k_lz1_Md_rows<T, 3, true, PPT>;
}

// Whether pass 1 runs on the row-staged kernels (CHDWF_STENCIL=rows, where
// they fit), and their plan and grid.
template <class T>
static bool lz_rows_setup(const Geom& g, RowPlan* rp, unsigned* nb) {
    if (stencil_mode() != 2) return false;
    if (!row_plan(g, sizeof(T), rp) || rp->ppt != 1) return false;
    const void* kern[6];
    lz_rows_kernels<T, 1>(kern);
    int dev = 0, nsm = 0, per_sm = 1 << 20;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    for (const void* k : kern) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rp->smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, rp->nthreads, rp->smem) !=
                cudaSuccess || b < 1) {
            cudaGetLastError();
            return false;
        }
        if (b < per_sm) per_sm = b;
    }
    int64_t n = (int64_t)nsm * per_sm;
    if (n > rp->nrows) n = rp->nrows;
    if (n < 1) return false;
    *nb = (unsigned)n;
    return true;
}

// L2 residency of vt = M q_j: k_lz1_M writes it and k_lz1_Md reads it right
// back, so its address range is marked persisting in L2 for the pass-1
// launches instead of taking a DRAM round trip.  The persisting carve-out is
// a limit of this process's context.  Returns the window (num_bytes 0 when
// the device offers none).
static constexpr bool kVtL2Window = true;

static cudaAccessPolicyWindow vt_window(const void* vt, size_t bytes) {
    cudaAccessPolicyWindow w{};
    if (!kVtL2Window) return w;
    int dev = 0, max_win = 0, max_persist = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_win, cudaDevAttrMaxAccessPolicyWindowSize, dev);
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, dev);
    if (max_win <= 0 || max_persist <= 0) return w;
    const size_t win = bytes < (size_t)max_win ? bytes : (size_t)max_win;
    size_t cur = 0;
    cudaDeviceGetLimit(&cur, cudaLimitPersistingL2CacheSize);
    const size_t want = win < (size_t)max_persist ? win : (size_t)max_persist;
    if (cur < want && cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want) == cudaSuccess)
        cur = want;
    cudaGetLastError();
    if (cur == 0) return w;
    w.base_ptr = const_cast<void*>(vt);
    w.num_bytes = win;
    w.hitRatio = cur >= win ? 1.0f : (float)((double)cur / (double)win);
    w.hitProp = cudaAccessPropertyPersisting;
    w.missProp = cudaAccessPropertyStreaming;
    return w;
}

static void set_stream_window(cudaStream_t st, const cudaAccessPolicyWindow& w) {
    cudaStreamAttrValue v{};
    v.accessPolicyWindow = w;
    cudaStreamSetAttribute(st, cudaStreamAttributeAccessPolicyWindow, &v);
    cudaGetLastError();
}

// Pass 1 is a sequence of identical launch pairs (the iteration index and the
// residual ring live in device memory), so a chunk of them is captured once
// as a CUDA graph and replayed; the graph is rebuilt when any argument
// changes.
template <class T>
static void launch_pass1_any(const LzArgsT<T>& a, unsigned nb, int k0, int chunk, cudaStream_t st,
                             const LzSide& side, KernelTimer* tm, int imass);

template <class T>
static cudaGraphExec_t pass1_graph(LzWork& w, const LzArgsT<T>& a_in, unsigned nb, int imass,
                                   int chunk, cudaStream_t st, const cudaAccessPolicyWindow& win) {
    // pass-1 kernels never touch the pass-2 fields: clear them so one graph
    // serves every solve of this precision (heatbath, hamilton, force)
    LzArgsT<T> a = a_in;
    a.x = nullptr;
    a.xw = nullptr;
    a.npole = 0;
    LzGraph& G = w.graph[sizeof(T) == sizeof(float2) ? 1 : 0][a.wcap > 0 ? 1 : 0];
    const unsigned char* key = reinterpret_cast<const unsigned char*>(&a);
    if (G.exec && G.nb == nb && G.imass == imass && G.chunk == chunk &&
        G.key.size() == sizeof(a) && memcmp(G.key.data(), key, sizeof(a)) == 0)
        return G.exec;
    if (G.exec) cudaGraphExecDestroy(G.exec);
    G.exec = nullptr;
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    for (int c = 0; c < chunk; c++) {
        launch_pass1_any<T>(a, nb, c, chunk, st, w.side, nullptr, imass);
    }
    if (cudaStreamEndCapture(st, &graph) != cudaSuccess || !graph) {
        cudaGetLastError();
        return nullptr;
    }
    if (win.num_bytes) {                 // the L2 window on every captured launch
        size_t nn = 0;
        cudaGraphGetNodes(graph, nullptr, &nn);
        std::vector<cudaGraphNode_t> nodes(nn);
        if (nn && cudaGraphGetNodes(graph, nodes.data(), &nn) == cudaSuccess) {
            cudaKernelNodeAttrValue v{};
            v.accessPolicyWindow = win;
            for (cudaGraphNode_t nd : nodes) {
                cudaGraphNodeType t;
                if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel)
                    cudaGraphKernelNodeSetAttribute(nd, cudaKernelNodeAttributeAccessPolicyWindow, &v);
            }
        }
        cudaGetLastError();
    }
    cudaGraphExec_t exec = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    G.exec = exec;
    G.nb = nb;
    G.imass = imass;
    G.chunk = chunk;
    G.key.assign(key, key + sizeof(a));
    return exec;
}

template <class T, int IMASS>
static void launch_pass2(const LzArgsT<T>& a, int j, int m, int iflag, cudaStream_t st,
                         KernelTimer& tm) {
    const int apply = j < m;
    const double V = (double)a.g.kferm * sizeof(T), chi = 12.0 * a.g.kvol;
    // On planes x takes in three vectors at a time, while r_{j-2}, r_{j-1} and r_j are
    // in the ring, in front of M^dagger(j), which writes over r_{j-2}.  x (FP64, the
    // ABI's layout: elements Ls apart for neighbouring threads) is read and written
    // once a triple, and the kernels are launched as pass 1's (launch_grid).  Solves to
    // 1e-9 without a store: 12^3x8 11.8 ms, 20^3x20 68.7; 14.4 and 71.4 without the
    // programmatic launches, 16.4 and 90 with x taken once a vector besides.
    const bool take = iflag == 0 && (!a.pl || j % 3 == 0 || j == m);
    const int j0 = j - (j - 1) % 3;
    const double acc =
        take ? 2.0 * a.g.kferm * sizeof(double2) + (a.pl ? j - j0 + 1 : 1) * V : 0.0;
    if (apply) tm.begin(timer_class<T>(3), st, 2 * V + chi + acc);
    if (a.pl) {
        auto blocks = [](int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); };
        if (iflag != 0)
            k_lzp_acc_walls<T><<<blocks(16 * (int64_t)a.g.kvol), kThreads, 0, st>>>(a, j);
        else if (take)
            k_lz_accum_x<T, true><<<blocks(acc_units(a)), kThreads, 0, st>>>(a, j0, j);
        if (apply)
            launch_grid(!tm.enabled, k_lz1_M<T, IMASS, true>, a.pp.nitem, a.pp.threads, 0, st, a, j);
        count_launches((iflag != 0 || take) + apply);
    } else {
        const unsigned nb = lz_direct_blocks<T>(a.g.npts);
        if (iflag == 0) k_lz2_M<T, IMASS, 0><<<nb, kThreads, 0, st>>>(a, j, apply);
        else k_lz2_M<T, IMASS, 1><<<nb, kThreads, 0, st>>>(a, j, apply);
        count_launches(1);
    }
    if (apply) {
        tm.end(st);
        tm.begin(timer_class<T>(3), st, 4 * V + chi);
        if (a.pl)
            launch_grid(!tm.enabled, k_lz1_Md<T, IMASS, false, true>, a.pp.nitem, a.pp.threads, 0, st,
                        a, j);
        else k_lz2_Md<T, IMASS><<<lz_direct_blocks<T>(a.g.npts), kThreads, 0, st>>>(a, j);
        tm.end(st);
        count_launches(1);
    }
}

template <class T>
static int pass1_shape(const LzArgsT<T>& a) {
    return a.rows ? kStencilRows : kStencilGather3;
}

template <class T>
static void launch_pass1_any(const LzArgsT<T>& a, unsigned nb, int k0, int chunk, cudaStream_t st,
                             const LzSide& side, KernelTimer* tm, int imass) {
    if (a.pl) {
        if (imass == 3) launch_pass1_planes<T, 3>(a, nb, k0, chunk, st, tm);
        else launch_pass1_planes<T, 1>(a, nb, k0, chunk, st, tm);
        return;
    }
    if (imass == 3) launch_pass1_rows<T, 3>(a, nb, st, side, tm);
    else launch_pass1_rows<T, 1>(a, nb, st, side, tm);
}

template <class T>
static void launch_pass2_any(const LzArgsT<T>& a, int j, int m, int iflag, cudaStream_t st,
                             KernelTimer& tm, int imass) {
    if (imass == 3) launch_pass2<T, 3>(a, j, m, iflag, st, tm);
    else launch_pass2<T, 1>(a, j, m, iflag, st, tm);
}

// ---- kernel timer ----------------------------------------------------------
void KernelTimer::enable() {
    if (enabled) return;
    for (int i = 0; i < 2 * kPool; i++) cudaEventCreate(&ev[i]);
    for (int i = 0; i < 2 * kChunkPool; i++) cudaEventCreate(&cev[i]);
    enabled = true;
    reset();
}

void KernelTimer::release() {
    if (!enabled) return;
    for (int i = 0; i < 2 * kPool; i++) cudaEventDestroy(ev[i]);
    for (int i = 0; i < 2 * kChunkPool; i++) cudaEventDestroy(cev[i]);
    enabled = false;
    chunks = false;
}

void KernelTimer::chunk_begin(cudaStream_t st, int first) {
    if (!enabled || cused >= kChunkPool) return;
    cfirst[cused] = first;
    cudaEventRecord(cev[2 * cused], st);
}

void KernelTimer::chunk_end(cudaStream_t st) {
    if (!enabled || cused >= kChunkPool) return;
    cudaEventRecord(cev[2 * cused + 1], st);
    cused++;
}

void KernelTimer::collect_chunks(int m, int chunk, int prec) {
    if (!enabled) return;
    for (int i = 0; i < cused; i++) {
        float ms = 0.0f;
        if (cfirst[i] + chunk - 1 <= m &&
            cudaEventElapsedTime(&ms, cev[2 * i], cev[2 * i + 1]) == cudaSuccess) {
            chunk_ms[prec] += ms;
            chunk_iters[prec] += chunk;
        }
    }
    cused = 0;
}

void KernelTimer::reset() {
    used = 0;
    for (int c = 0; c < kClasses; c++) {
        total_ms[c] = 0;
        total_bytes[c] = 0;
        count[c] = 0;
        launches[c] = 0;
    }
    cused = 0;
    chunk_ms[0] = chunk_ms[1] = 0.0;
    chunk_iters[0] = chunk_iters[1] = 0;
}

void KernelTimer::begin(int c, cudaStream_t st, double nbytes) {
    if (!enabled) return;
    launches[c]++;
    if (used >= kPool) return;          // pool full: the launch is counted, not timed
    cls[used] = c;
    bytes[used] = nbytes;
    cudaEventRecord(ev[2 * used], st);
}

void KernelTimer::end(cudaStream_t st) {
    if (!enabled || used >= kPool) return;
    cudaEventRecord(ev[2 * used + 1], st);
    used++;
}

void KernelTimer::collect() {
    if (!enabled) return;
    for (int i = 0; i < used; i++) {
        float ms = 0.0f;
        if (cudaEventElapsedTime(&ms, ev[2 * i], ev[2 * i + 1]) == cudaSuccess) {
            total_ms[cls[i]] += ms;
            total_bytes[cls[i]] += bytes[i];
            count[cls[i]]++;
        }
    }
    used = 0;
}

LzWork::~LzWork() {
    release();
    timer.release();
}

void LzWork::release() {
    for (auto& row : graph)
        for (LzGraph& gr : row) {
            if (gr.exec) cudaGraphExecDestroy(gr.exec);
            gr = LzGraph();
        }
    if (side.fork) cudaEventDestroy(side.fork);
    if (side.join) cudaEventDestroy(side.join);
    if (side.stream) cudaStreamDestroy(side.stream);
    side = LzSide();
    if (ctl) cudaFree(ctl);
    if (hist_mem) cudaFree(hist_mem);
    if (part) cudaFree(part);
    if (hflag_host) cudaFreeHost(hflag_host);
    for (int i = 0; i < 3; i++) {
        if (rb[i]) cudaFree(rb[i]);
        if (rb32[i]) cudaFree(rb32[i]);
    }
    if (vt) cudaFree(vt);
    if (vt32) cudaFree(vt32);
    if (basis) cudaFree(basis);
    if (basis32) cudaFree(basis32);
    if (wall) cudaFree(wall);
    if (wall32) cudaFree(wall32);
    basis = nullptr;
    basis32 = nullptr;
    wall = nullptr;
    wall32 = nullptr;
    hcap = hcap32 = 0;
    wcap = wcap32 = 0;
    if (xw) cudaFree(xw);
    if (x2w) cudaFree(x2w);
    ctl = nullptr; hist_mem = nullptr; part = nullptr; hflag_host = nullptr;
    rb[0] = rb[1] = rb[2] = vt = xw = x2w = nullptr;
    rb32[0] = rb32[1] = rb32[2] = vt32 = nullptr;
    xw_poles = 0;
}

cudaError_t LzWork::ensure(const Geom& g, int npole_max, int prec, bool walls) {
    cudaError_t e;
    const bool same = ctl && g.kferm == geom.kferm && g.L == geom.L && g.Lt == geom.Lt;
    if (!same) {
        release();
        geom = g;
        if ((e = cudaMalloc(&ctl, sizeof(LzCtl)))) return e;
        const int64_t H = kMaxIter + 2;
        const size_t nh = 4 * H + 3 * (size_t)kMaxPoles * H;
        if ((e = cudaMalloc(&hist_mem, nh * sizeof(double)))) return e;
        hist.alphat = hist_mem;
        hist.beta = hist_mem + H;
        hist.invbeta = hist_mem + 2 * H;
        hist.c = hist_mem + 3 * H;
        hist.rho = hist_mem + 4 * H;
        hist.mu = hist.rho + kMaxPoles * H;
        hist.y = hist.mu + kMaxPoles * H;
        // block partials of the two pass-1 phases (at most kMaxPartBlocks
        // resident blocks), or the source norm's block partials
        if ((e = cudaMalloc(&part, sizeof(double) * 2 * kMaxPartBlocks))) return e;
        if ((e = cudaHostAlloc(&hflag_host, sizeof(int), cudaHostAllocMapped))) return e;
        if ((e = cudaStreamCreateWithFlags(&side.stream, cudaStreamNonBlocking))) return e;
        if ((e = cudaEventCreateWithFlags(&side.fork, cudaEventDisableTiming))) return e;
        if ((e = cudaEventCreateWithFlags(&side.join, cudaEventDisableTiming))) return e;
        if ((e = cudaHostGetDevicePointer((void**)&hflag_dev, hflag_host, 0))) return e;
    }
    if (prec == kPrecF64 && !rb[0]) {
        for (int i = 0; i < 3; i++)
            if ((e = cudaMalloc(&rb[i], sizeof(double2) * g.kferm))) return e;
        if ((e = cudaMalloc(&vt, sizeof(double2) * g.kferm))) return e;
    }
    if (prec == kPrecF32 && !rb32[0]) {
        for (int i = 0; i < 3; i++)
            if ((e = cudaMalloc(&rb32[i], sizeof(float2) * plane_elems<float2>(g)))) return e;
        if ((e = cudaMalloc(&vt32, sizeof(float2) * plane_elems<float2>(g)))) return e;
    }
    // Basis store: up to kMaxIter+2 vectors, at most 40% of the free HBM per
    // precision.  Solves longer than the store regenerate their vectors.
    if (basis_enabled && ((prec == kPrecF64 && !basis) || (prec == kPrecF32 && !basis32))) {
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        const size_t vb = prec == kPrecF64 ? sizeof(double2) * (size_t)g.kferm
                                           : sizeof(float2) * (size_t)plane_elems<float2>(g);
        // an explicit budget names the FP64 store; the FP32 store keeps the
        // same number of vectors in half the bytes
        const double budget = basis_max_bytes >= 0.0
                                  ? basis_max_bytes * (prec == kPrecF64 ? 1.0 : 0.5)
                                  : 0.4 * (double)fr;
        int64_t cap = (int64_t)(budget / (double)vb);
        if (cap > kMaxIter + 2) cap = kMaxIter + 2;
        if (cap >= 8) {
            void* ptr = nullptr;
            if (cudaMalloc(&ptr, vb * (size_t)cap) == cudaSuccess) {
                if (prec == kPrecF64) { basis = (double2*)ptr; hcap = (int)cap; }
                else { basis32 = (float2*)ptr; hcap32 = (int)cap; }
            } else {
                cudaGetLastError();   // not enough memory: regenerate instead
            }
        }
    }
    // Wall store: up to kMaxIter+2 two-slice vectors within 15% of the free
    // HBM; force solves that outgrow it regenerate their vectors.
    if (walls && basis_enabled && ((prec == kPrecF64 && !wall) || (prec == kPrecF32 && !wall32))) {
        size_t fr = 0, tot = 0;
        cudaMemGetInfo(&fr, &tot);
        const size_t vb = (prec == kPrecF64 ? sizeof(double2) : sizeof(float2)) * 16 * (size_t)g.kvol;
        int64_t cap = (int64_t)(0.15 * (double)fr / (double)vb);
        if (cap > kMaxIter + 2) cap = kMaxIter + 2;
        if (cap >= 8) {
            void* ptr = nullptr;
            if (cudaMalloc(&ptr, vb * (size_t)cap) == cudaSuccess) {
                if (prec == kPrecF64) { wall = (double2*)ptr; wcap = (int)cap; }
                else { wall32 = (float2*)ptr; wcap32 = (int)cap; }
            } else {
                cudaGetLastError();
            }
        }
    }
    if (npole_max > xw_poles) {
        if (xw) cudaFree(xw);
        if (x2w) cudaFree(x2w);
        xw_poles = npole_max;
        const size_t nw = (size_t)xw_poles * 16 * g.kvol;
        if ((e = cudaMalloc(&xw, sizeof(double2) * nw))) return e;
        if ((e = cudaMalloc(&x2w, sizeof(double2) * nw))) return e;
    }
    return cudaSuccess;
}

template <class T>
static void set_ring(LzArgsT<T>& a, LzWork& w);
template <>
void set_ring<double2>(LzArgsT<double2>& a, LzWork& w) {
    a.rb0 = w.rb[0]; a.rb1 = w.rb[1]; a.rb2 = w.rb[2]; a.vt = w.vt;
    a.basis = w.basis_enabled ? w.basis : nullptr;
    a.hcap = a.basis ? w.hcap : 0;
}
template <>
void set_ring<float2>(LzArgsT<float2>& a, LzWork& w) {
    a.rb0 = w.rb32[0]; a.rb1 = w.rb32[1]; a.rb2 = w.rb32[2]; a.vt = w.vt32;
    a.basis = w.basis_enabled ? w.basis32 : nullptr;
    a.hcap = a.basis ? w.hcap32 : 0;
}

// Force solves with a wall store keep only the ring and the wall slices.
template <class T>
static void set_walls(LzArgsT<T>& a, LzWork& w) {
    T* ws;
    int cap;
    if constexpr (std::is_same<T, double2>::value) { ws = w.wall; cap = w.wcap; }
    else { ws = w.wall32; cap = w.wcap32; }
    if (!w.basis_enabled || !ws) return;
    a.wbasis = ws;
    a.wcap = cap;
    a.basis = nullptr;
    a.hcap = 0;
}

// The two wall slices of r (s = 1 and s = Ls) into wall-store vector j, laid
// out as the wall fields: element (slice sw, component c, site) at
// sw + 2 site + 2 kvol c.
template <class T>
__global__ void __launch_bounds__(kThreads) k_lz_walls_of(LzArgsT<T> a, const T* __restrict__ r,
                                                         int j) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t cs2 = 2 * (int64_t)a.g.kvol;
    if (t >= 8 * cs2) return;
    const int c = (int)(t / cs2);
    const int64_t rr = t - c * cs2;
    const int sw = (int)(rr & 1);
    const int64_t site = rr >> 1;
    a.wbasis[(int64_t)j * 8 * cs2 + t] =
        vget(a, r, c, sw ? a.g.Ls - 1 : 0, site);
}

// q_j's wall slices (j = 1..m) into every pole's two-slice x_k: the same
// sums, in the same order, as from the full stored vectors.  One thread per
// wall element (slice, component, site) and NC poles per pass (one pass for
// up to 24 poles), so the store is read once or twice; the pass's y_kj and 1/beta_j
// are staged in shared memory kYChunk iterations at a time.  STORE: the q_j
// come from the wall store (coalesced), else from the stored basis.
constexpr int kYChunk = 32;
template <class T, int NC, bool STORE>
__global__ void __launch_bounds__(kThreads, 2) k_lz_accum_walls(LzArgsT<T> a, int m, int k0) {
    typedef typename real_of<T>::type Real;
    __shared__ double ys[NC][kYChunk];
    __shared__ Real ibs[kYChunk];
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t cs2 = 2 * (int64_t)a.g.kvol, kf2 = 8 * cs2;
    const bool act = t < kf2;
    // from the basis: component, wall and site of the element
    const int c = act ? (int)(t / cs2) : 0;
    const int64_t r = act ? t - c * cs2 : 0;
    const int s = (r & 1) ? a.g.Ls - 1 : 0;
    auto load = [&](int j) {
        return STORE ? __ldg(a.wbasis + j * kf2 + t) : vget(a, a.basis + j * a.vs, c, s, r >> 1);
    };
    const int64_t H = kMaxIter + 2;
    const int n = a.npole;
    double2 acc[NC];
#pragma unroll
    for (int k = 0; k < NC; k++) acc[k] = make_double2(0.0, 0.0);
    for (int j0 = 1; j0 <= m; j0 += kYChunk) {
        const int jn = m - j0 + 1 < kYChunk ? m - j0 + 1 : kYChunk;
        __syncthreads();
        for (int i = threadIdx.x; i < NC * kYChunk; i += blockDim.x) {
            const int k = i / kYChunk, jj = i - k * kYChunk;
            ys[k][jj] = (k0 + k < n && jj < jn) ? a.h.y[(k0 + k) * H + j0 + jj] : 0.0;
        }
        for (int i = threadIdx.x; i < kYChunk; i += blockDim.x)
            ibs[i] = i < jn ? (Real)a.h.invbeta[j0 + i] : (Real)0;
        __syncthreads();
        if (act) {
            // q_{j+1} is loaded while q_j is accumulated
            T qn = load(j0);
#pragma unroll 1
            for (int jj = 0; jj < jn; jj++) {
                const T q = qn;
                if (jj + 1 < jn) qn = load(j0 + jj + 1);
                const double2 qj = widen(zscal(ibs[jj], q));
#pragma unroll
                for (int k = 0; k < NC; k++) {
                    const double y = ys[k][jj];
                    acc[k].x += y * qj.x;
                    acc[k].y += y * qj.y;
                }
            }
        }
    }
    if (!act) return;
#pragma unroll
    for (int k = 0; k < NC; k++)
        if (k0 + k < n) a.xw[(k0 + k) * kf2 + t] = acc[k];
}

template <class T, bool STORE>
static void launch_accum_walls(const LzArgsT<T>& a, int m, int n, int64_t kvol, cudaStream_t st) {
    const unsigned nb = (unsigned)((16 * kvol + kThreads - 1) / kThreads);
    for (int k0 = 0; k0 < n; k0 += 24) {
        const int left = n - k0;
        if (left <= 8) k_lz_accum_walls<T, 8, STORE><<<nb, kThreads, 0, st>>>(a, m, k0);
        else if (left <= 16) k_lz_accum_walls<T, 16, STORE><<<nb, kThreads, 0, st>>>(a, m, k0);
        else k_lz_accum_walls<T, 24, STORE><<<nb, kThreads, 0, st>>>(a, m, k0);
        count_launches(1);
    }
}

static constexpr int kAccumChunk = 64;

// Per-shift solutions (iflag 2): x_k = sum_j y_kj q_j for poles k0..k0+7,
// every element summing j = 1..m in order; xk[k] are device pointers.
template <class T>
__global__ void __launch_bounds__(kThreads) k_lz_accum_poles(LzArgsT<T> a, int m, int k0,
                                                             double2* const* xk) {
    typedef typename real_of<T>::type Real;
    constexpr int N = AccUnit<T>::N;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= acc_units(a)) return;
    int ne;
    const int64_t e = acc_elem(a, i, &ne);
    const int64_t H = kMaxIter + 2;
    const int n = a.npole;
    double2 acc[8][N];
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
        for (int p = 0; p < N; p++) acc[k][p] = make_double2(0.0, 0.0);
    for (int j = 1; j <= m; j++) {
        T q[N];
        AccUnit<T>::get(a, a.basis + j * a.vs, i, q);
        const Real ib = (Real)a.h.invbeta[j];
        double2 qj[N];
#pragma unroll
        for (int p = 0; p < N; p++) qj[p] = widen(zscal(ib, q[p]));
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k0 + k < n) {
                const double y = a.h.y[(k0 + k) * H + j];
#pragma unroll
                for (int p = 0; p < N; p++) {
                    acc[k][p].x += y * qj[p].x;
                    acc[k][p].y += y * qj[p].y;
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (k0 + k < n) {
            xk[k0 + k][e] = acc[k][0];
            if (N == 2 && ne == 2) xk[k0 + k][e + 1] = acc[k][N - 1];
        }
}

template <class T>
static cudaError_t lz_solve_t(LzWork& w, const Geom& g, const double2* phi, float res, int ndiag,
                              const double* anum, const double* aden, int iflag,
                              const float* chif, float am3, float hpin, int imass, int ibound,
                              double2* x, float* dSdchi, int* itercg, int* status,
                              LzStats* stats, cudaStream_t st) {
    typedef typename real_of<T>::type Real;
    cudaError_t e;
    LzCtl hc;
    memset(&hc, 0, sizeof(hc));
    hc.it_m = 1;
    hc.npole = ndiag;
    hc.niter_cap = kMaxIter;
    const float resid = sqrtf((float)g.kferm * res * res);   // :621
    const float arelax = 2.0f;                                // :711
    hc.thresh = (double)(arelax * resid);
    for (int k = 0; k < ndiag; k++) {
        hc.sigma[k] = aden[k];
        hc.anum[k] = anum[k + 1];
    }
    if ((e = cudaMemcpyAsync(w.ctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, st))) return e;
    *w.hflag_host = 0;

    LzArgsT<T> a;
    memset(&a, 0, sizeof(a));
    a.g = g;
    set_ring(a, w);
    if (iflag == 1) set_walls(a, w);
    a.chif = chif;
    a.diag = (Real)(2.0f * ((3.0f - am3) + 1.0f));
    a.hpin = (Real)hpin;
    a.apbc = ibound == -1;
    a.ctl = w.ctl;
    a.h = w.hist;
    a.part = w.part;
    a.hflag = w.hflag_dev;
    a.x = x;
    a.xw = w.xw;
    a.npole = ndiag;
    unsigned nb = 0;
    a.rows = lz_rows_setup<T>(g, &a.rp, &nb) ? 1 : 0;
    a.pl = !a.rows;
    a.vs = a.pl ? plane_elems<T>(g) : g.kferm;
    if (a.pl) {
        if (!plane_ok(g)) return cudaErrorInvalidValue;
        int dev = 0, nsm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        a.pp = plane_plan(g, std::is_same<T, float2>::value, nsm);
        nb = imass == 3 ? pass1_workers<T, 3>(a.pp, nsm) : pass1_workers<T, 1>(a.pp, nsm);
        if (nb < 1) return cudaErrorLaunchOutOfResources;
    }
    const int nbr = reduce_blocks(g.kferm);
    // r_1 lives where ring(a, 1) looks for it: the basis store when present
    T* r1 = a.hcap > 1 ? a.basis + a.vs : a.rb1;

    // r_1 = Phi, beta_1 = |r_1|
    k_lz_source<T><<<nbr, kThreads, 0, st>>>(a, r1, phi, w.part);
    k_lz_init<<<1, kThreads, 0, st>>>(w.ctl, w.hist, w.part, nbr);
    count_launches(2);
    if (a.wcap > 1) {                    // r_1's wall slices (pass 1 adds r_2, r_3, ...)
        k_lz_walls_of<T><<<(unsigned)((16 * (int64_t)g.kvol + kThreads - 1) / kThreads), kThreads,
                           0, st>>>(a, r1, 1);
        count_launches(1);
    }

    // pass 1: launch chunks of iterations and poll the mapped flag with
    // kAhead chunks queued beyond the one being checked, so a host thread
    // that wakes late still finds the GPU busy
    const int chunk = 16;
    constexpr int kAhead = 2;
    cudaEvent_t ev[kAhead + 1];
    for (cudaEvent_t& e : ev) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    int launched = 0, nchunk = 0;
    const cudaAccessPolicyWindow win = vt_window(a.vt, sizeof(T) * (size_t)a.vs);
    if (win.num_bytes) set_stream_window(st, win);
    // per-launch timing issues pass 1 launch by launch; chunk timing keeps
    // the graph replays and brackets each one
    const bool chunked = w.timer.enabled && w.timer.chunks;
    const int per_it = a.pl ? 2 : 3;      // kernels an iteration
    cudaGraphExec_t gexec = w.timer.enabled && !chunked
                                ? nullptr
                                : pass1_graph<T>(w, a, nb, imass, chunk, st, win);
    while (launched < kMaxIter) {
        if (gexec) {
            if (chunked) w.timer.chunk_begin(st, launched + 1);
            cudaGraphLaunch(gexec, st);
            if (chunked) w.timer.chunk_end(st);
        } else {
            for (int c = 0; c < chunk; c++)
                launch_pass1_any<T>(a, nb, c, chunk, st, w.side, &w.timer, imass);
        }
        launched += chunk;
        count_launches(per_it * chunk + a.pl);
        note_stencil(pass1_shape(a), 2 * chunk);
        cudaEventRecord(ev[nchunk % (kAhead + 1)], st);
        if (nchunk >= kAhead) {
            cudaEventSynchronize(ev[(nchunk - kAhead) % (kAhead + 1)]);
            if (*(volatile int*)w.hflag_host) break;
        }
        nchunk++;
    }
    if (chunked) {
        cudaStreamSynchronize(st);
        LzCtl hm;
        cudaMemcpy(&hm, w.ctl, sizeof(hm), cudaMemcpyDeviceToHost);
        w.timer.collect_chunks(hm.m, chunk, std::is_same<T, float2>::value ? 1 : 0);
    } else if (w.timer.enabled) {
        // launches after convergence returned at once: drop them
        cudaStreamSynchronize(st);
        LzCtl hm;
        cudaMemcpy(&hm, w.ctl, sizeof(hm), cudaMemcpyDeviceToHost);
        int keep = 0;
        for (int i = 0, it = 0; i < w.timer.used; i++) {
            if (w.timer.cls[i] == timer_class<T>(0)) it++;
            const bool real = it <= hm.m;      // M^dagger(m) completes too
            if (real) {
                w.timer.cls[keep] = w.timer.cls[i];
                w.timer.bytes[keep] = w.timer.bytes[i];
                std::swap(w.timer.ev[2 * keep], w.timer.ev[2 * i]);
                std::swap(w.timer.ev[2 * keep + 1], w.timer.ev[2 * i + 1]);
                keep++;
            }
        }
        w.timer.launches[timer_class<T>(0)] -= launched - hm.m;
        w.timer.launches[timer_class<T>(1)] -= launched - hm.m;
        w.timer.used = keep;
        w.timer.collect();
    }
    for (cudaEvent_t& e : ev) cudaEventDestroy(e);   // the stream sync below covers them
    if (win.num_bytes) set_stream_window(st, cudaAccessPolicyWindow{});
    if ((e = cudaGetLastError())) return e;
    LzCtl hr;
    if ((e = cudaMemcpyAsync(&hr, w.ctl, sizeof(hr), cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    const int m = hr.m;
    *itercg = m;
    if (hr.done == 4) return cudaErrorLaunchTimeout;   // a bounded wait ran out
    *status = hr.done == 1 ? 0 : (hr.done == 2 ? 1 : 2);
    if (stats) { stats->iters = m; stats->pass1_launches = 2 * launched; }
    if (m < 1) return cudaErrorUnknown;

    // coefficients, then pass 2 over the regenerated vectors
    k_lz_coeffs<<<1, kThreads, 0, st>>>(w.ctl, w.hist, iflag);
    k_lz_source<T><<<nbr, kThreads, 0, st>>>(a, r1, phi, w.part);
    count_launches(2);
    if (iflag == 2) {
        // every x_k from the stored basis, poles in chunks of 8 (one pass over
        // the basis per chunk); needs the whole basis in HBM
        if (!(m < a.hcap) || !w.pole_out) return cudaErrorInvalidValue;
        const unsigned nbx = (unsigned)((acc_units(a) + kThreads - 1) / kThreads);
        for (int k0 = 0; k0 < ndiag; k0 += 8) {
            k_lz_accum_poles<T><<<nbx, kThreads, 0, st>>>(a, m, k0, w.pole_out);
            count_launches(1);
        }
        return cudaGetLastError();
    }
    launch_scale(x, phi, anum[0], g.kferm, st);                       // x = a0 Phi (:628)
    if (iflag == 1) cudaMemsetAsync(w.xw, 0, sizeof(double2) * (size_t)ndiag * 16 * g.kvol, st);
    if (a.wcap > 0 ? m < a.wcap : m < a.hcap) {
        // every q_j (or, for the force, its wall slices) is still in HBM:
        // one streaming pass over the store reads the m stored vectors and
        // the solution once
        const double vb = (double)sizeof(T);
        const double nbytes = iflag == 0
            ? (double)m * g.kferm * vb + 2.0 * g.kferm * sizeof(double2)
            : (double)m * 16.0 * g.kvol * vb + (double)ndiag * 16.0 * g.kvol * sizeof(double2);
        w.timer.begin(timer_class<T>(2), st, nbytes);
        if (iflag == 0) {
            // a chunk of stored vectors per launch: x (FP64) is carried in
            // memory between chunks, so each element still sums j = 1..m in
            // order, and the pages a launch touches stay few
            const unsigned nbx = (unsigned)((acc_units(a) + kThreads - 1) / kThreads);
            for (int j0 = 1; j0 <= m; j0 += kAccumChunk) {
                const int j1 = j0 + kAccumChunk - 1 < m ? j0 + kAccumChunk - 1 : m;
                k_lz_accum_x<T, false><<<nbx, kThreads, 0, st>>>(a, j0, j1);
                count_launches(1);
            }
        } else if (a.wcap > 0) {
            launch_accum_walls<T, true>(a, m, ndiag, g.kvol, st);
        } else {
            launch_accum_walls<T, false>(a, m, ndiag, g.kvol, st);
        }
        w.timer.end(st);
    } else {
        for (int j = 1; j <= m; j++) {
            launch_pass2_any<T>(a, j, m, iflag, st, w.timer, imass);
            if (w.timer.enabled && w.timer.used >= KernelTimer::kPool - 2) {
                cudaStreamSynchronize(st);
                w.timer.collect();
            }
        }
    }
    if (w.timer.enabled) {
        cudaStreamSynchronize(st);
        w.timer.collect();
    }
    if (iflag == 1) {
        // X2 = M x_k on the walls, then derivs pole by pole (:733-740)
        launch_wall_dslash64(ndiag, w.x2w, w.xw, chif, g, am3, hpin, ibound, imass, st);
        const double* anum_dev = reinterpret_cast<const double*>(
            reinterpret_cast<const char*>(w.ctl) + offsetof(LzCtl, anum));
        launch_derivs_walls(ndiag, w.xw, w.x2w, anum_dev, imass, dSdchi, g, st);
    }
    return cudaGetLastError();
}

// Multi-shift solve.  anum[0..n], aden[0..n-1] as in the reference.
// iflag 0: x = a0 Phi + sum_k a_k x_k.  iflag 1: x = a0 Phi and the force
// contribution of every pole is accumulated into dSdchi (device, REAL*4).
cudaError_t lz_solve(LzWork& w, const Geom& g, const double2* phi, float res, int ndiag,
                     const double* anum, const double* aden, int iflag, const float* chif,
                     float am3, float hpin, int imass, int ibound, double2* x, float* dSdchi,
                     int* itercg, int* status, LzStats* stats, cudaStream_t st, int prec) {
    if (ndiag < 1 || ndiag > kMaxPoles) return cudaErrorInvalidValue;
    cudaError_t e = w.ensure(g, iflag == 1 ? ndiag : 1, prec, iflag == 1);
    if (e) return e;
    if (prec == kPrecF32)
        return lz_solve_t<float2>(w, g, phi, res, ndiag, anum, aden, iflag, chif, am3, hpin,
                                  imass, ibound, x, dSdchi, itercg, status, stats, st);
    return lz_solve_t<double2>(w, g, phi, res, ndiag, anum, aden, iflag, chif, am3, hpin, imass,
                               ibound, x, dSdchi, itercg, status, stats, st);
}

}  // namespace chdwf
