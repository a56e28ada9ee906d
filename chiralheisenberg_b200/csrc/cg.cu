// cg.cu -- congrad: CGNE on M^dagger M (rhmc/cheisdwf.f:1064-1157), one
// system.  The kernels and their arithmetic are those of the batched solver
// (plane_cg.cuh), with a system's own blocks and order of sums, so one solve
// gives the same bits alone and in a batch.
#include <cstdio>
#include <cstring>

#include "cg.h"
#include "plane_cg.cuh"

namespace chdwf {

CgWork::~CgWork() { release(); }

void CgWork::release() {
    if (w) {
        w->release();
        delete w;
    }
    w = nullptr;
}

static bool cg_batch(PcgBatch<double2, 1>& b, const Geom& g, float am3, float hpin, int imass,
                     int ibound) {
    return plane_ok(g) && b.add(g, (double)(2.0f * ((3.0f - am3) + 1.0f)), (double)hpin,
                                ibound == -1, imass, 0, pcg_sms());
}

cudaError_t cg_solve(CgWork& w, const Geom& g, const double2* phi, float res, const float* chif,
                     float am3, float hpin, int imass, int ibound, double2* x, int* itercg,
                     int* status, cudaStream_t st) {
    if (!w.w) w.w = new PcgWork<double2>();
    PcgWork<double2>& W = *w.w;
    PcgBatch<double2, 1> b;
    if (!cg_batch(b, g, am3, hpin, imass, ibound)) return cudaErrorInvalidValue;
    cudaError_t e = W.reserve(b.units, 0, b.parts);
    if (e) return e;
    W.bind(b, chif);
    std::vector<PcgDyn<double2>> dyn(1, pcg_congrad_dyn(g, res, x, phi));
    std::vector<PcgSlot> slots(1, pcg_congrad_slot());
    if ((e = pcg_congrad(W, b, dyn, slots, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    *itercg = slots[0].iters;
    *status = pcg_status(slots[0]);
    return cudaSuccess;
}

// ---- congrad without any allocation ---------------------------------------
// For callers that cannot allocate device memory: a host program whose device
// memory is owned by another runtime's pool or reserved in full up front, or
// code that must not allocate (a real-time or otherwise allocation-free
// section).  The solver's scratch -- the REAL*4 copy of chi, the CG vectors
// x1, p, r, the per-block partial sums and the control block (scalars and
// counters) -- lives in one file-scope device array sized for kferm <=
// kStaticMaxFerm.  The array is shared by every call: calls whose GPU work
// overlaps (other streams, other host threads) race on it.  Each call writes
// the control block before its first kernel.
constexpr int64_t kStaticMaxFerm = 262144;            // 8*kvol*kthird, e.g. 16^3 x 8
constexpr int64_t kStaticMaxKvol = kStaticMaxFerm / 16;   // kthird >= 2
struct StaticCtl {
    PcgDyn<double2> dyn;
    PcgSlot slot[2];
    PcgRun run;
};
constexpr size_t kStaticCtl = 1024;
// stencil blocks twice, element blocks (kferm units, rounded up), alpha
constexpr size_t kStaticParts =
    2 * (size_t)kPcgMaxBlocks +
    kStaticMaxFerm / (kPcgThreads * pcg_units_thread<double2>()) + 2;
static_assert(sizeof(StaticCtl) <= kStaticCtl, "the control block outgrew its place");
static_assert(kStaticParts * sizeof(double) <= 64 * 1024, "the partials outgrew their place");
constexpr size_t kStaticBytes = kStaticCtl + 64 * 1024 +    // control block, partials
                                3 * kStaticMaxKvol * sizeof(float) +
                                3 * kStaticMaxFerm * sizeof(double2);
static __device__ __align__(256) unsigned char g_cg_scratch[kStaticBytes];

namespace {
constexpr int kMaxDevices = 64;
// Device address of the array per device ordinal.  Two host threads making
// their first call on a device at the same time both look it up and store
// the same value: a benign race, since cudaGetSymbolAddress returns one
// address per device.
unsigned char* g_scratch_addr[kMaxDevices] = {};
}  // namespace

}  // namespace chdwf

extern "C" int chdwf_congrad_static(const void* Phi, void* x, const void* chi, int ksize,
                                    int ksizet, int kthird, float am3, int ibound, float res,
                                    float hpin, int imass, int* itercg, void* stream) {
    using namespace chdwf;
    if (!Phi || !x || !chi || !itercg) return 4;
    if (imass != 1 && imass != 3) return 4;
    // sizes in 64-bit arithmetic first: kvol = ksize^2*ksizet is a 32-bit
    // int in the geometry and must not wrap before the size check
    if (!geom_ok(ksize, ksizet, kthird)) return 4;
    if (8 * (int64_t)ksize * ksize * ksizet * kthird > kStaticMaxFerm) return 4;
    const Geom g = make_geom(ksize, ksizet, kthird);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 3;
    // once per device: the device address of the array (its host-side name
    // is only a stand-in and must never be passed to a kernel)
    if (!g_scratch_addr[dev]) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_cg_scratch) != cudaSuccess || !ptr) return 3;
        g_scratch_addr[dev] = (unsigned char*)ptr;
    }
    // a sticky error from earlier work on this device fails here; a stale
    // non-sticky one is cleared so that it is not reported as this call's
    if (cudaGetLastError() != cudaSuccess && cudaPeekAtLastError() != cudaSuccess) return 3;
    unsigned char* base = g_scratch_addr[dev];
    StaticCtl* ctl = reinterpret_cast<StaticCtl*>(base);
    double* part = reinterpret_cast<double*>(base + kStaticCtl);
    float* chif = reinterpret_cast<float*>(base + kStaticCtl + 64 * 1024);
    double2* vec = reinterpret_cast<double2*>(base + kStaticCtl + 64 * 1024 +
                                              3 * kStaticMaxKvol * sizeof(float));
    cudaStream_t st = (cudaStream_t)stream;
    PcgBatch<double2, 1> b;
    if (!cg_batch(b, g, am3, hpin, imass, ibound)) return 4;
    b.a.vec = vec;
    b.a.chif = b.a.chi_out = chif;
    b.a.part = part;
    b.a.dyn = &ctl->dyn;
    b.a.slot = ctl->slot;
    b.a.run = &ctl->run;
    StaticCtl hc;
    memset(&hc, 0, sizeof(hc));
    hc.dyn = pcg_congrad_dyn(g, res, (double2*)x, (const double2*)Phi, (const double*)chi);
    hc.slot[0] = hc.slot[1] = pcg_congrad_slot();
    hc.run.active = 1;
    if (cudaMemcpyAsync(ctl, &hc, sizeof(hc), cudaMemcpyHostToDevice, st) != cudaSuccess) return 3;
    pcg_congrad_enter(b.a, st);
    // chunks of 16 iterations; the scalars are copied into a host stack
    // variable after each chunk (launches after convergence return at once)
    const int64_t cap = hc.dyn.niterc;
    int64_t launched = 0;
    bool failed = false;
    PcgSlot hs[2];
    PcgSlot hr;
    memset(&hr, 0, sizeof(hr));
    while (launched < cap) {
        pcg_launch_chunk(b.a, imass, 16, st);
        launched += 16;
        count_launches(3 * 16 + 1);
        // a failed launch or copy ends the solve at once instead of launching
        // on until the iteration cap
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(hs, ctl->slot, sizeof(hs), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            failed = true;
            break;
        }
        hr = hs[0].done ? hs[0] : hs[1];
        if (hr.done) break;
    }
    pcg_congrad_leave(b.a, st);
    failed |= cudaGetLastError() != cudaSuccess;
    failed |= cudaStreamSynchronize(st) != cudaSuccess;
    if (failed) return 3;
    *itercg = hr.iters;
    if (hr.done == 2) {
        fprintf(stdout, " # iterations of congrad exceeds niterc\n");   // :1151-1153
        return 1;
    }
    if (hr.done == 3) return 2;
    return 0;
}
