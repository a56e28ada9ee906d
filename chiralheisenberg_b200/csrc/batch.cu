// batch.cu -- many independent propagator solves in one set of launches.
//
// fermion() (rhmc/cheisdwf.f:897-1058) solves M^dagger M x = Phi with congrad
// (:1064-1157) once per source, one after the other.  On small lattices each
// iteration of one solve is a few microseconds of GPU work, so a sequence of
// solves is bound by kernel launches and host round trips.  Here nsys solves
// -- on lattices of different sizes, with their own chi, imass and hpin --
// advance together: one launch per CG stage covers the blocks of every
// still-running system, each system keeps its own REAL*4 scalars (the types of
// congrad) and stops on its own criterion (plane_cg.cuh).  Each system's
// arithmetic, block partition and reduction order are those of congrad on its
// own, so the results equal chdwf_congrad_dev's.
//
// Systems whose vectors together outgrow L2 would stream them from HBM every
// iteration, so systems advance together only as far as their vectors fit
// kBatchBytes and their mass terms agree (and up to 256 of them on 34 lattices); the
// parts run one after the other.  Heights, pinnings and the order of the list do not
// divide a batch: small solves are bound by latency, and 32 on eight lattices up to
// 8^3x8 took 15.7 ms in six parts instead of 4.4 together.
#include <algorithm>
#include <cstring>
#include <map>
#include <tuple>
#include <vector>

#include "../../include/chdwf.h"
#include "cg.h"
#include "ctx.h"
#include "plane_cg.cuh"

namespace chdwf {

// Batch workspace, kept in the context and reallocated when a larger batch
// arrives.
struct BatchWork {
    PcgWork<double2> w;
};

void free_batch(BatchWork* b) {
    if (b) {
        b->w.release();
        delete b;
    }
}

// p, r, x1 and x of the systems of one part.  32 solves on lattices up to
// 16^3x24 (one to 50 MB each): 60-90 MB 190-194 ms, one solve at a time 235,
// all at once 203.
constexpr double kBatchBytes = 90e6;

}  // namespace chdwf

using namespace chdwf;

extern "C" int chdwf_congrad_batch(chdwf_ctx* ctx, const chdwf_cg_system* in, int nsys, float res,
                                   int* itercg, int* status) {
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    if (!c || !in || nsys < 1 || !itercg || !status) return CHDWF_BAD_ARG;
    cudaSetDevice(c->device);
    for (int i = 0; i < nsys; i++) {
        const chdwf_cg_system& s = in[i];
        if (!geom_ok(s.ksize, s.ksizet, s.kthird) || !s.Phi || !s.x || !s.chi ||
            (s.imass != 1 && s.imass != 3))
            return CHDWF_BAD_ARG;
    }
    if (!c->batch) c->batch = new BatchWork();
    PcgWork<double2>& w = c->batch->w;
    cudaStream_t st = c->stream;
    const int nsm = pcg_sms();
    // the systems in the order in which they run (imass 1, then 3; those of a
    // lattice together, as a part holds few lattices), and the parts that advance
    // together (part p: from order[first[p]])
    std::map<std::tuple<int, int, int, int>, int> at;          // first of its kind
    std::vector<int> order(nsys), kind(nsys);
    for (int i = 0; i < nsys; i++) {
        const chdwf_cg_system& s = in[i];
        order[i] = i;
        kind[i] = at.emplace(std::make_tuple(s.imass, s.ksize, s.ksizet, s.kthird), i).first->second;
    }
    std::stable_sort(order.begin(), order.end(), [&](int i, int k) {
        return std::tie(in[i].imass, kind[i]) < std::tie(in[k].imass, kind[k]);
    });
    std::vector<PcgBatch<double2, kPcgSysBatch>> parts(1);
    std::vector<int> first(1, 0);
    std::vector<Geom> geo(nsys);
    double bytes = 0.0;
    int64_t units = 0;                                // of the largest part
    int chis = 0, nparts = 0;
    for (int o = 0; o < nsys; o++) {
        const int i = order[o];
        const chdwf_cg_system& s = in[i];
        const Geom g = geo[i] = make_geom(s.ksize, s.ksizet, s.kthird);
        if (!plane_ok(g)) return c->status_of(cudaErrorInvalidValue, "congrad_batch: lattice");
        const double b = 4.0 * sizeof(double2) * (double)g.kferm;
        auto add = [&] {
            return parts.back().add(g, (double)(2.0f * ((3.0f - s.am3) + 1.0f)), (double)s.hpin,
                                    s.ibound == -1, s.imass, 0, nsm);
        };
        if ((parts.back().a.nsys > 0 && bytes + b > kBatchBytes) || !add()) {
            parts.emplace_back();
            first.push_back(o);
            bytes = 0.0;
            if (!add()) return c->status_of(cudaErrorInvalidValue, "congrad_batch: lattice");
        }
        bytes += b;
        const PcgBatch<double2, kPcgSysBatch>& P = parts.back();
        if (P.units > units) units = P.units;
        if (P.chis > chis) chis = P.chis;
        if (P.parts > nparts) nparts = P.parts;
    }
    first.push_back(nsys);
    cudaError_t e = w.reserve(units, chis, nparts);
    if (e) return c->status_of(e, "congrad_batch: workspace");
    int worst = CHDWF_OK;
    for (size_t part = 0; part < parts.size(); part++) {
        std::vector<PcgDyn<double2>> dyn;
        for (int k = 0; k < parts[part].a.nsys; k++) {
            const int i = order[first[part] + k];
            dyn.push_back(pcg_congrad_dyn(geo[i], res, (double2*)in[i].x, (const double2*)in[i].Phi,
                                          (const double*)in[i].chi));
        }
        std::vector<PcgSlot> slots(dyn.size(), pcg_congrad_slot());
        auto run = [&](auto P) {
            w.bind(P);
            return pcg_congrad(w, P, dyn, slots, st);
        };
        e = parts[part].fits<kPcgSys>() ? run(parts[part].cut<kPcgSys>()) : run(parts[part]);
        if (e) return c->status_of(e, "congrad_batch");
        for (size_t k = 0; k < slots.size(); k++) {
            const int i = order[first[part] + k], s = pcg_status(slots[k]);
            itercg[i] = slots[k].iters;
            status[i] = s == 0 ? CHDWF_OK : (s == 1 ? CHDWF_ITER_CAP : CHDWF_NONFINITE);
            if (status[i] > worst) worst = status[i];
        }
    }
    if ((e = cudaStreamSynchronize(st))) return c->status_of(e, "congrad_batch");
    return worst;
}
