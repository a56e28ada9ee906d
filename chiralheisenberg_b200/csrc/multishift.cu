// multishift.cu -- per-shift solutions of (M^dag M + sigma_k) x_k = Phi with
// their true residuals (no reference routine returns them: qmrherm keeps
// x1(ndiag,kferm) internally, rhmc/cheisdwf.f:614,:689-695, and testinv,
// :854-890, checks each pole's true residual), in FP64 or with FP32 Krylov
// vectors and FP64 defect correction.
//
// FP64: the two-pass Lanczos solve (lanczos.cu) with every x_k formed from
// the stored basis, stopping by the reference's rule at res.
// FP32: the same solve with FP32 vectors stopped at max(res, 1e-6), x_k
// accumulated in FP64; then, per shift, while the FP64 true residual
// |Phi - (M^dag M + sigma_k) x_k| / |Phi| exceeds res: an FP32 CG on the
// shifted system with the FP64 residual as right-hand side, and its solution
// added to x_k in FP64 -- defect correction, each round recomputing the true
// residual in FP64.  The result meets the same true-residual target as FP64.
//
// The corrections of several shifts run as one batch (plane_cg.cuh): their
// scalars stay on the device and each iteration is three launches for all of
// them: 20 shifts at 16^3x16 to 1e-10 take 92 to 99 ms.  One shift at a time, with
// the scalars on the host (two round trips an iteration), they took 560 to 700 ms.
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/chdwf.h"
#include "ctx.h"
#include "lanczos.h"
#include "plane_cg.cuh"

using namespace chdwf;

namespace chdwf {
namespace {

unsigned nb_of(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// r = Phi - t - sigma x (FP64); partial sums of |r|^2 per block
__global__ void k_ms_resid(double2* __restrict__ r, const double2* __restrict__ phi,
                           const double2* __restrict__ t, const double2* __restrict__ x,
                           double sigma, int64_t n, double* __restrict__ part) {
    __shared__ double sh[kThreads / 32];
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = make_double2(phi[i].x - t[i].x - sigma * x[i].x,
                                       phi[i].y - t[i].y - sigma * x[i].y);
        r[i] = v;
        s += v.x * v.x + v.y * v.y;
    }
    s = block_sum<kThreads>(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// r (FP64, ABI layout) times scale into planes: the inner solve's r and p, e
// = 0, and the blocks' partials of |p|^2 (k_pcg3's blocks)
__global__ void __launch_bounds__(kPcgThreads) k_ms_planes(cpair* p, cpair* rp, cpair* x,
                                                           double* part, Geom g, int U,
                                                           const double2* __restrict__ r,
                                                           double scale) {
    constexpr int kN = pcg_units_thread<float2>();
    const int64_t nu = 8 * (int64_t)U * g.kvol;
    const int64_t i0 = (int64_t)blockIdx.x * (kPcgThreads * kN) + threadIdx.x;
    double loc = 0.0;
    for (int q = 0; q < kN; q++) {
        const int64_t i = i0 + q * kPcgThreads;
        if (i >= nu) break;
        const PlaneUnit pu = plane_unit_of<float2>(g, U, i);
        const double2 a = r[pu.e], b = pu.n == 2 ? r[pu.e + 1] : make_double2(0.0, 0.0);
        const cpair v{make_float2((float)(a.x * scale), (float)(b.x * scale)),
                      make_float2((float)(a.y * scale), (float)(b.y * scale))};
        const cpair z{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        st_unit(p + i, v);
        st_unit(rp + i, v);
        st_unit(x + i, z);
        loc += unit_norm2(v);
    }
    __shared__ double sh[32];
    loc = block_sum_any(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = loc;
}
// x += scale * e (FP64, ABI layout; e in planes)
__global__ void k_ms_add(double2* __restrict__ x, const cpair* __restrict__ ev, Geom g, int U,
                         double scale) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= 8 * (int64_t)U * g.kvol) return;
    const PlaneUnit pu = plane_unit_of<float2>(g, U, i);
    const cpair e = ld_unit(ev + i);
    for (int k = 0; k < pu.n; k++) {
        const float2 v = cpair_pt(e, k);
        x[pu.e + k] = make_double2(x[pu.e + k].x + scale * v.x, x[pu.e + k].y + scale * v.y);
    }
}

struct MsWork {
    double2 *t = nullptr, *r = nullptr;   // r: one residual per system of a part
    double* part = nullptr;
    double2** xk_dev = nullptr;
    ~MsWork() {
        cudaFree(t); cudaFree(r); cudaFree(part); cudaFree(xk_dev);
    }
};

// Residual vector Phi - (M^dag M + sigma) x into r, block partials of its
// square into part (FP64)
void true_residual(Ctx* c, MsWork& w, const double* chi, const double2* phi, const double2* x,
                   double sigma, float hpin, int imass, double2* r, double* part) {
    const Geom& g = c->g;
    launch_dslash64(false, imass, w.t, x, {chi, c->chif}, g, c->am3, hpin, c->ibound, c->stream);
    launch_dslash64(true, imass, c->spin[3], w.t, {chi, c->chif}, g, c->am3, hpin, c->ibound, c->stream);
    k_ms_resid<<<reduce_blocks(g.kferm), kThreads, 0, c->stream>>>(r, phi, c->spin[3], x, sigma,
                                                                  g.kferm, part);
    count_launches(1);
}

// Sums of n consecutive runs of len partials.
cudaError_t run_sums(const double* part_dev, int n, int len, double* out, cudaStream_t st) {
    std::vector<double> h((size_t)n * len);
    cudaError_t e = cudaMemcpyAsync(h.data(), part_dev, sizeof(double) * h.size(),
                                    cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    for (int i = 0; i < n; i++) {
        out[i] = 0.0;
        for (int k = 0; k < len; k++) out[i] += h[(size_t)i * len + k];
    }
    return e;
}

constexpr double kMsBytes = 90e6;      // FP32 vectors of a part: they stay in L2
constexpr int kMsRounds = 20;          // corrections of one shift at most
constexpr double kMsInner = 1e-5;      // relative residual of an inner solve, least
constexpr double kMsOuter = 1e-4;      // and largest

// Defect correction of the shifts k0..k0+n-1 together, until each one's true
// residual is at most res or stops falling.
cudaError_t correct_part(Ctx* c, MsWork& w, PcgWork<float2>& P, const double* chi,
                         const double2* phi, double phin,
                         float res, float hpin, int imass, int k0, int n, const double* sigma,
                         void* const* x, double* true_res, int* iters) {
    const Geom& g = c->g;
    cudaStream_t st = c->stream;
    const int nb = reduce_blocks(g.kferm);
    const size_t ve = (size_t)plane_elems<float2>(g) / 2;     // units of a vector
    std::vector<int> run(n);           // the part's shifts still to be corrected
    for (int i = 0; i < n; i++) run[i] = i;
    std::vector<double> rel(n, HUGE_VAL), r2(n), rr(n);
    cudaError_t e;
    for (int round = 0; !run.empty(); round++) {
        for (size_t a = 0; a < run.size(); a++) {
            const int i = run[a];
            true_residual(c, w, chi, phi, (const double2*)x[k0 + i], sigma[k0 + i], hpin, imass,
                          w.r + g.kferm * (int64_t)a, w.part + (size_t)nb * a);
        }
        if ((e = run_sums(w.part, (int)run.size(), nb, r2.data(), st))) return e;
        std::vector<int> next, slot;
        for (size_t a = 0; a < run.size(); a++) {
            const int i = run[a];
            const double now = std::sqrt(r2[a]) / phin;
            const bool falls = now < rel[i];
            rel[i] = now;
            true_res[k0 + i] = now;
            if (falls && now > (double)res && round < kMsRounds) {
                next.push_back(i);
                slot.push_back((int)a);
            }
        }
        run = next;
        if (run.empty()) break;
        PcgBatch<float2> B;
        std::vector<PcgDyn<float2>> dyn;
        std::vector<PcgSlot> slots(run.size());
        for (size_t q = 0; q < run.size(); q++)
            if (!B.add(g, 2.0f * ((3.0f - c->am3) + 1.0f), hpin, c->ibound == -1, imass, 1, pcg_sms()))
                return cudaErrorInvalidValue;
        P.bind(B, c->chif);
        const int U = B.geo(0).pl.U, neblk = B.geo(0).neblk, nblk = B.geo(0).nblk;
        for (size_t a = 0; a < run.size(); a++) {
            cpair* p = P.vec + B.a.vec0[a];
            double* part3 = P.part + B.a.part0[a] + 2 * nblk;
            k_ms_planes<<<neblk, kPcgThreads, 0, st>>>(p, p + ve, p + 3 * ve, part3, g, U,
                                                       w.r + g.kferm * (int64_t)slot[a],
                                                       1.0 / std::sqrt(r2[slot[a]]));
            count_launches(1);
        }
        for (size_t a = 0; a < run.size(); a++) {
            if ((e = run_sums(P.part + B.a.part0[a] + 2 * nblk, 1, neblk, &rr[a], st))) return e;
            // one round to a tenth of res where FP32 can reach it, and never
            // less than four digits: x is then 1.5e-10 from 64 bits at res
            // 1e-10 (a quarter of res: 3.8e-10; a fixed 1e-4: 2.6e-10)
            double tol = 0.1 * (double)res / rel[run[a]];
            tol = tol < kMsInner ? kMsInner : (tol > kMsOuter ? kMsOuter : tol);
            memset(&slots[a], 0, sizeof(PcgSlot));
            slots[a].rr = rr[a];
            PcgDyn<float2> d;
            memset(&d, 0, sizeof(d));
            d.x = P.vec + B.a.vec0[a] + 3 * ve;
            d.sigma = (float)sigma[k0 + run[a]];
            d.rstop = tol * tol * rr[a];
            d.niterc = 4 * kMaxIter;
            dyn.push_back(d);
        }
        if ((e = P.solve(B, dyn, slots, st))) return e;
        for (size_t a = 0; a < run.size(); a++) {
            *iters += slots[a].iters;
            k_ms_add<<<nb_of((int64_t)ve), kThreads, 0, st>>>((double2*)x[k0 + run[a]], dyn[a].x, g, U,
                                                             std::sqrt(r2[slot[a]]));
            count_launches(1);
        }
    }
    return cudaGetLastError();
}

}  // namespace

void free_multishift(PcgWork<float2>* w) {
    if (w) {
        w->release();
        delete w;
    }
}
}  // namespace chdwf

extern "C" int chdwf_multishift_dev(chdwf_ctx* ctx, const void* Phi, float res, const void* chi,
                                    float hpin, int imass, int n, const double* sigma,
                                    void* const* x, double* true_res, int prec, int* iters,
                                    int* refine_iters) {
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    if (!c || !Phi || !chi || !sigma || !x || !true_res || !iters || !refine_iters) return CHDWF_BAD_ARG;
    if (n < 1 || n > kMaxPoles || (prec != CHDWF_PREC_F64 && prec != CHDWF_PREC_F32)) return CHDWF_BAD_ARG;
    cudaSetDevice(c->device);
    const Geom& g = c->g;
    cudaStream_t st = c->stream;
    launch_round_chi((const double*)chi, c->chif, g.kvol, st);
    MsWork w;
    cudaError_t e;
    // shifts that are corrected together: as many as keep their four FP32
    // vectors in L2
    const size_t ve = (size_t)plane_elems<float2>(g) / 2;
    int np = prec == CHDWF_PREC_F32 ? (int)(kMsBytes / (64.0 * (double)ve)) : 1;
    np = np < 1 ? 1 : (np > n ? n : np);
    if ((e = cudaMalloc(&w.t, sizeof(double2) * g.kferm)) ||
        (e = cudaMalloc(&w.r, sizeof(double2) * g.kferm * np)) ||
        (e = cudaMalloc(&w.part, sizeof(double) * 2048 * np)) ||
        (e = cudaMalloc(&w.xk_dev, sizeof(double2*) * n)))
        return c->status_of(e, "multishift");
    cudaMemcpyAsync(w.xk_dev, x, sizeof(double2*) * n, cudaMemcpyHostToDevice, st);
    std::vector<double> anum(n + 1, 1.0);
    anum[0] = 0.0;
    const float res1 = prec == CHDWF_PREC_F32 ? std::fmax(res, 1e-6f) : res;
    int st_code = 0;
    c->lz.pole_out = w.xk_dev;
    e = lz_solve(c->lz, g, (const double2*)Phi, res1, n, anum.data(), sigma, 2, c->chif, c->am3,
                 hpin, imass, c->ibound, nullptr, c->dS, iters, &st_code, &c->last_lz, st,
                 prec == CHDWF_PREC_F32 ? kPrecF32 : kPrecF64);
    c->lz.pole_out = nullptr;
    if (e) return c->status_of(e, "multishift (basis store too small for per-shift output?)");
    if (st_code == 1) { c->err = "multishift: iteration cap reached"; return CHDWF_ITER_CAP; }
    if (st_code == 2) { c->err = "multishift: non-finite value"; return CHDWF_NONFINITE; }
    double phi2 = 0.0;
    launch_norm2((const double2*)Phi, g.kferm, w.part, c->red, st);
    cudaMemcpyAsync(&phi2, c->red, sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    const double phin = std::sqrt(phi2);
    *refine_iters = 0;
    if (prec == CHDWF_PREC_F32) {
        if (!c->ms) c->ms = new PcgWork<float2>();
        PcgWork<float2>& P = *c->ms;
        PcgBatch<float2> B;                 // the largest part
        for (int i = 0; i < np; i++)
            if (!plane_ok(g) || !B.add(g, 0.0f, 0.0f, 0, imass, 1, pcg_sms()))
                return c->status_of(cudaErrorInvalidValue, "multishift: lattice");
        if ((e = P.reserve(B.units, 0, B.parts))) return c->status_of(e, "multishift: workspace");
        for (int k0 = 0; k0 < n; k0 += np) {
            const int m = n - k0 < np ? n - k0 : np;
            if ((e = correct_part(c, w, P, (const double*)chi, (const double2*)Phi, phin, res, hpin, imass, k0, m, sigma,
                                  x, true_res, refine_iters)))
                return c->status_of(e, "multishift refinement");
        }
        // kept for the next call while it is small beside what a solve holds
        if (64.0 * (double)ve > kMsBytes) P.release();
    } else {
        for (int k = 0; k < n; k++) {
            double r2 = 0.0;
            true_residual(c, w, (const double*)chi, (const double2*)Phi, (const double2*)x[k], sigma[k], hpin, imass, w.r,
                          w.part);
            if ((e = run_sums(w.part, 1, reduce_blocks(g.kferm), &r2, st)))
                return c->status_of(e, "multishift residual");
            true_res[k] = std::sqrt(r2) / phin;
        }
    }
    return c->status_of(cudaStreamSynchronize(st), "multishift");
}
