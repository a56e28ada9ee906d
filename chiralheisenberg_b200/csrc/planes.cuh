// planes.cuh -- site-fastest vectors of the solvers and the stencil on them.
//
// The spinors of the C ABI have s innermost.  The solvers' own vectors
// (Krylov and CG vectors, which never cross the boundary) are kept in
// "planes" instead: 16-byte units with the site fastest,
//     unit(c, u, site) at (c*U + u)*kvol + site,      c = d + 4f,
// a unit being one FP64 complex number (u = s, U = Ls) or two FP32 ones (a
// cpair: s = 2u and 2u+1, U = ceil(Ls/2); for odd Ls the last unit's second
// half is kept zero).  A warp then covers 32 neighbouring sites of ONE s, so
//   * the wall coupling is a branch of the whole warp, taken by the first and
//     last unit only (with s innermost every warp holds wall points and runs
//     the wall code);
//   * a thread walks a run of units at its site, so the neighbours' offsets
//     are computed once per run;
//   * a block is a tile of nx*ny*nt sites, so the y and t neighbours of most
//     of its threads are in the block and come from L1.
// FP64 elements go through dwf_apply_flavour's operations in its order, so
// they have the same bits in either layout.
//
// What bounds the kernels (B200, 24^3x24, ncu): L1 wavefronts (28 16-byte
// loads a unit, 55-65% of the L1 rate) and the latency of the loads at 24
// warps an SM.  At 80 registers no value is carried from one unit of a run
// to the next: holding the unit and its s neighbours in registers saves 4
// of 32 loads but costs 40 registers, i.e. half of the warps, and the FP32
// iteration (M and M^dagger back to back) took 30 us instead of 25.  With s
// innermost (thread pairs of adjacent s) it took 38.
#pragma once
#include <type_traits>

#include "dwf_stencil.cuh"

namespace chdwf {

// Packed fused multiply-add and product.  f2_mulp's result must not feed a
// packed addition (it would be fused, see above): it is for products that
// are stored or that a fused multiply-add takes as its addend.
#ifdef CHDWF_F32X2
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 f2_mulp(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
#else
__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
    return make_float2(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y));
}
__device__ __forceinline__ float2 f2_mulp(float2 a, float2 b) {
    return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
}
#endif
// s*a with packed products (see f2_mulp), and s*a + b fused
__device__ __forceinline__ cpair zscal2(float s, cpair a) {
    const float2 ss = make_float2(s, s);
    return cpair{f2_mulp(ss, a.re), f2_mulp(ss, a.im)};
}
__device__ __forceinline__ cpair zaxpy(float s, cpair a, cpair b) {
    const float2 ss = make_float2(s, s);
    return cpair{f2_fma(ss, a.re, b.re), f2_fma(ss, a.im, b.im)};
}
__device__ __forceinline__ double2 zscal2(double s, double2 a) { return zscal(s, a); }
__device__ __forceinline__ double2 zaxpy(double s, double2 a, double2 b) {
    return make_double2(__fma_rn(s, a.x, b.x), __fma_rn(s, a.y, b.y));
}


// Launch plan of the plane kernels: work item = (site tile, flavour, run of
// units), each taken by one block pass.
struct PlanePlan {
    int L, Lt, Ls, U;
    uint32_t kvol;
    int nx, ny, nt;            // tile
    int tx, ty, tt;            // tiles along x, y, t
    int nrun;                  // runs of units: run k covers [k*U/nrun, (k+1)*U/nrun)
    int threads;               // nx*ny*nt rounded up to warps
    uint32_t ntile, nitem;     // nitem = ntile*2*nrun
    FastDiv dtile, dtx, dty;   // item decoding
};

inline int plane_units(int Ls, bool f32) { return f32 ? (Ls + 1) / 2 : Ls; }
// Elements of the complex type T in one vector.
template <class T> inline int64_t plane_elems(const Geom& g) {
    const bool f32 = std::is_same<T, float2>::value;
    return 8 * (int64_t)plane_units(g.Ls, f32) * g.kvol * (f32 ? 2 : 1);
}

// One block may fill an SM: 24 warps at 80 registers, 6 a scheduler.
constexpr int kPlaneRegs = 80;
constexpr int kPlaneMaxThreads = 768;
static_assert(kPlaneMaxThreads / 4 * kPlaneRegs <= 16384, "a block exceeds an SM's registers");

// Tile and runs for a lattice on nsm SMs.  A step (one unit of every warp
// resident on an SM) takes about 1500 cycles of load latency plus 220 cycles
// a warp, most of it L1 wavefronts.  Fitted to 60 plans each of nine lattices
// from 8^3x8 to 24^3x24, both precisions; the plan that the model picks is
// within 4% of the best one measured.  Examples, us an iteration (M and
// M^dagger): 24^3x24 FP32, tiles 24x8x2 in runs of 3 units (12 warps, 288
// blocks, 2 an SM) 29.8, tiles 24x6x2 in runs of 2 33.2, tiles 24x5x4 that
// leave a second wave nearly empty 53.9; 12^3x8 FP64, 288 blocks of 3 warps
// 10.0, 48 blocks of 18 13.7.  The plan minimises
//     waves * (units in a run + 0.3) * (1500 + 220 * warps an SM)
// over the tiles of whole x rows that fit a block and the runs.  Halo reads
// from L2 (2/ny + 2/nt of a site's) and the block barriers of large blocks
// weigh a few per cent of a step, and a block's partial 3 cycles.
//
// block > 0: the kernel's blocks have that many threads whatever the tile
// (several lattices in one launch, plane_cg.cuh); tiles then hold at most that.
inline PlanePlan plane_plan(const Geom& g, bool f32, int nsm, int block = 0) {
    const int most = block ? block : kPlaneMaxThreads;
    PlanePlan best{};
    double best_cost = 1e300;
    const int U = plane_units(g.Ls, f32);
    const int sx = (g.L + 63) / 64, nx = (g.L + sx - 1) / sx;
    for (int nt = 1; nt <= g.Lt && nx * nt <= most; nt++)
        for (int ny = 1; ny <= g.L && nx * ny * nt <= most; ny++) {
            const int warps = (nx * ny * nt + 31) / 32;
            const int tx = (g.L + nx - 1) / nx, ty = (g.L + ny - 1) / ny;
            const int tt = (g.Lt + nt - 1) / nt;
            const int64_t ntile = (int64_t)tx * ty * tt;
            const double halo = 1.0 + (ny < g.L ? 2.0 / ny : 0.0) + (nt < g.Lt ? 2.0 / nt : 0.0);
            const int occ = 4 * (16384 / (32 * kPlaneRegs)) / (block ? block / 32 : warps);
            for (int nrun = 1; nrun <= U; nrun++) {
                const int64_t nitem = ntile * 2 * nrun;
                if (nitem > 0x7fffffff) break;
                const int C = (U + nrun - 1) / nrun;
                const int64_t per_sm = (nitem + nsm - 1) / nsm;
                const int64_t full = per_sm / occ, rem = per_sm - full * occ;
                auto step = [&](double w) { return 1500.0 + 220.0 * w; };
                double cost = (double)full * step((double)occ * warps);
                if (rem) cost += step((double)rem * warps);
                cost *= (C + 0.3) * (1.0 + 0.02 * halo) * (1.0 + 0.005 * warps);
                cost += 3.0 * (double)(nitem < (int64_t)nsm * occ ? nitem : (int64_t)nsm * occ);
                if (cost < best_cost * 0.999) {
                    best_cost = cost;
                    best.nx = nx; best.ny = ny; best.nt = nt;
                    best.tx = tx; best.ty = ty; best.tt = tt;
                    best.nrun = nrun;
                    best.threads = warps * 32;
                    best.ntile = (uint32_t)ntile;
                    best.nitem = (uint32_t)nitem;
                }
            }
        }
    best.L = g.L; best.Lt = g.Lt; best.Ls = g.Ls; best.U = U;
    best.kvol = (uint32_t)g.kvol;
    best.dtile = make_fastdiv(best.ntile);
    best.dtx = make_fastdiv((uint32_t)best.tx);
    best.dty = make_fastdiv((uint32_t)best.ty);
    return best;
}

// Plane offsets are 32-bit bytes.
inline bool plane_ok(const Geom& g) { return (int64_t)g.kvol * 16 < (int64_t(1) << 32); }

template <class T> struct unit_of;                      // T: complex type of the vectors
template <> struct unit_of<double2> { typedef double2 type; };
template <> struct unit_of<float2> { typedef cpair type; };

// Plain (coherent) 16-byte loads: the persistent kernels read what other
// blocks wrote earlier in the same launch.
__device__ __forceinline__ double2 ld_unit(const double2* p) { return *p; }
// Unit at byte offset off (32 bits: a plane is below 4 GB) of a base that is
// the same for the whole block: the base stays in uniform registers and the
// neighbours' offsets serve every component and every unit of a run.
template <class V> __device__ __forceinline__ const V* unit_at(const V* base, uint32_t off) {
    return reinterpret_cast<const V*>(reinterpret_cast<const char*>(base) + off);
}
template <class V> __device__ __forceinline__ V* unit_at(V* base, uint32_t off) {
    return reinterpret_cast<V*>(reinterpret_cast<char*>(base) + off);
}
__device__ __forceinline__ cpair ld_unit(const cpair* p) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    return cpair{make_float2(q.x, q.y), make_float2(q.z, q.w)};
}
__device__ __forceinline__ void st_unit(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void st_unit(cpair* p, const cpair& v) {
    *reinterpret_cast<float4*>(p) = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
__device__ __forceinline__ double unit_norm2(double2 v) { return v.x * v.x + v.y * v.y; }
__device__ __forceinline__ double unit_norm2(const cpair& v) {
    const double a = v.re.x, b = v.im.x, c = v.re.y, d = v.im.y;
    double s = a * a + b * b;
    s += c * c + d * d;
    return s;
}

// s hop within a run: a -= the element one s up (UP) or down, which for a
// pair is the other half of the same unit and one half of the next.
template <bool UP>
__device__ __forceinline__ void plane_shop(double2& a, double2, double2 other, bool have) {
    if (have) a = zsub(a, other);
}
template <bool UP>
__device__ __forceinline__ void plane_shop(cpair& a, const cpair& self, const cpair& other,
                                           bool have) {
    if (UP) {
        a.re.x = __fsub_rn(a.re.x, self.re.y);
        a.im.x = __fsub_rn(a.im.x, self.im.y);
        if (have) {
            a.re.y = __fsub_rn(a.re.y, other.re.x);
            a.im.y = __fsub_rn(a.im.y, other.im.x);
        }
    } else {
        if (have) {
            a.re.x = __fsub_rn(a.re.x, other.re.y);
            a.im.x = __fsub_rn(a.im.x, other.im.y);
        }
        a.re.y = __fsub_rn(a.re.y, self.re.x);
        a.im.y = __fsub_rn(a.im.y, self.im.x);
    }
}

// Wall coupling of the Dirac pair D0, D0+1 of flavour f at one wall (SIDE 0:
// s = Ls, SIDE 1: s = 1) for the wall's half of the unit; o points at the
// other wall's units of this site (component stride cst), oh is its half.
template <bool DAG, int IMASS, int D0, int SIDE>
__device__ __forceinline__ void plane_wall(double2 acc[4], const double2* o, int64_t cst, int, int,
                                           int f, float c1, float c2, float c3, bool pin,
                                           double hpin) {
#pragma unroll
    for (int d = D0; d < D0 + 2; d++)
        wall_elem<DAG, IMASS, SIDE>(acc[d], ld_unit(o + cst * d), ld_unit(o + cst * (d + 4)), f,
                                    c1, c2, c3, pin, hpin);
}
template <bool DAG, int IMASS, int D0, int SIDE>
__device__ __forceinline__ void plane_wall(cpair acc[4], const cpair* o, int64_t cst, int h,
                                           int oh, int f, float c1, float c2, float c3, bool pin,
                                           float hpin) {
#pragma unroll
    for (int d = D0; d < D0 + 2; d++) {
        const cpair r1 = ld_unit(o + cst * d), r2 = ld_unit(o + cst * (d + 4));
        float2 a = cpair_pt(acc[d], h);
        wall_elem<DAG, IMASS, SIDE>(a, cpair_pt(r1, oh), cpair_pt(r2, oh), f, c1, c2, c3, pin,
                                    hpin);
        if (h) {
            acc[d].re.y = a.x;
            acc[d].im.y = a.y;
        } else {
            acc[d].re.x = a.x;
            acc[d].im.x = a.y;
        }
    }
}

__device__ __forceinline__ void plane_prefetch(const void* p) {
#ifdef __CUDA_ARCH__
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
#endif
}
__device__ __forceinline__ void plane_clear_pad(double2*, bool) {}
__device__ __forceinline__ void plane_clear_pad(cpair* acc, bool pad) {
    if (pad) {
#pragma unroll
        for (int d = 0; d < 4; d++) acc[d].re.y = acc[d].im.y = 0.0f;
    }
}

// Diagonal term and hops.  FP64 keeps the reference's order of operations
// element by element (diag*R, six hops, times 1/2), so the operator has the
// oracle's bits.  FP32 pairs sum the six hops first and form
// (diag/2) R - (1/2) sum with one packed fused multiply-add: the products
// are not rounded separately, which is no less exact, and costs 16 packed
// instructions a unit less.  The fused operations are explicit, so every kernel
// that evaluates the operator on pairs produces the same bits.
template <int SF>
__device__ __forceinline__ void plane_first_hop(double2*, const double2*) {}
template <int MU, int SIG>
__device__ __forceinline__ void plane_hop(double2 acc[4], const double2 r[4]) {
    hop<MU, SIG, false>(acc, r);
}
__device__ __forceinline__ void plane_kappa(double2 acc[4], const double2*, double) {
#pragma unroll
    for (int d = 0; d < 4; d++) acc[d] = zscal(0.5, acc[d]);
}
template <int SF>
__device__ __forceinline__ void plane_first_hop(cpair acc[4], const cpair r[4]) {
    // minus the hop terms of direction x: (a, b, -+ i b, -+ i a)
    const cpair a = zcomb(r[0], r[3], true, SF), b = zcomb(r[1], r[2], true, SF);
    const cpair z{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
    acc[0] = a;
    acc[1] = b;
    acc[2] = zcomb(z, b, true, -SF);
    acc[3] = zcomb(z, a, true, -SF);
}
template <int MU, int SIG>
__device__ __forceinline__ void plane_hop(cpair acc[4], const cpair r[4]) {
    hop<MU, SIG, true>(acc, r);
}
__device__ __forceinline__ void plane_kappa(cpair acc[4], const cpair cur[4], float diag) {
    const float hd = 0.5f * diag;
#pragma unroll
    for (int d = 0; d < 4; d++) acc[d] = zaxpy(-0.5f, acc[d], zscal2(hd, cur[d]));
}

struct PlaneThread { int x, y, t; };   // the thread's place in its tile
__device__ __forceinline__ PlaneThread plane_thread(const PlanePlan& pl, int tid) {
    const int r = tid / pl.nx, t = r / pl.ny;
    return PlaneThread{tid - r * pl.nx, r - t * pl.ny, t};
}
__device__ __forceinline__ PlaneThread plane_thread(const PlanePlan& pl) {
    return plane_thread(pl, (int)threadIdx.x);
}
// Where a work item puts the thread: flavour, run of units, site, and the byte
// offsets in a plane of the site and its neighbours.  Threads without a site
// (act false) stand at the tile's corner; with SKIP `none` says that no thread
// of the warp has one.
struct PlanePlace {
    int f, u0, u1, t;
    bool act, none;
    uint32_t site, o_0, o_xp, o_xm, o_yp, o_ym, o_tp, o_tm;
};
template <bool SKIP, uint32_t W>
__device__ __forceinline__ PlanePlace plane_place(const PlanePlan& pl, const PlaneThread& th,
                                                  uint32_t item) {
    PlanePlace p;
    const int L = pl.L, Lt = pl.Lt, U = pl.U;
    // item -> (run, flavour, tile); tile -> corner
    const uint32_t rf = fdiv(item, pl.dtile), tile = item - rf * pl.ntile;
    const int run = (int)(rf >> 1);
    p.f = (int)(rf & 1);
    const uint32_t tyt = fdiv(tile, pl.dtx), tix = tile - tyt * (uint32_t)pl.tx;
    const uint32_t tit = fdiv(tyt, pl.dty), tiy = tyt - tit * (uint32_t)pl.ty;
    p.u0 = run * U / pl.nrun;
    p.u1 = (run + 1) * U / pl.nrun;
    int x = (int)tix * pl.nx + th.x, y = (int)tiy * pl.ny + th.y, t = (int)tit * pl.nt + th.t;
    p.act = th.t < pl.nt && x < L && y < L && t < Lt;
    // whole warps only: behind a branch of single threads nothing is kept in
    // uniform registers
    p.none = SKIP && !__any_sync(0xffffffffu, p.act);
    if (!p.act) { x = (int)tix * pl.nx; y = (int)tiy * pl.ny; t = (int)tit * pl.nt; }
    p.t = t;
    const uint32_t uL = (uint32_t)L, LL = uL * uL;
    p.site = (uint32_t)x + uL * ((uint32_t)y + uL * (uint32_t)t);
    const uint32_t o_0 = p.o_0 = p.site * W;
    p.o_xp = x + 1 == L ? o_0 - (uL - 1) * W : o_0 + W;
    p.o_xm = x == 0 ? o_0 + (uL - 1) * W : o_0 - W;
    p.o_yp = y + 1 == L ? o_0 - uL * (uL - 1) * W : o_0 + uL * W;
    p.o_ym = y == 0 ? o_0 + uL * (uL - 1) * W : o_0 - uL * W;
    p.o_tp = t + 1 == Lt ? o_0 - LL * (uint32_t)(Lt - 1) * W : o_0 + LL * W;
    p.o_tm = t == 0 ? o_0 + LL * (uint32_t)(Lt - 1) * W : o_0 - LL * W;
    return p;
}

// One work item: the thread's site, flavour and run of units.  For every
// unit of the run epi(acc, off) is called by every thread of the block with
// the four Dirac components of M R or M^dagger R: component d belongs at unit
// e + d*cst of an output vector, byte offset o0 (the thread's site) from
// there; act tells whether the thread holds a site, u is the unit.  It
// returns whether to go on (the same for the whole block).
// SKIP: warps without a site return at once (no block barrier in epi).
// S_LATE: the units above and below are loaded behind the diagonal term, which
// suits kernels that would spill otherwise (CG in FP64 207 -> 193 ms for 32
// solves; the multi-shift kernels with imass 1 are 3% faster with it off).
template <bool DAG, int IMASS, bool SKIP = false, bool S_LATE = IMASS == 3, class V, class Real,
          class Epi>
__device__ __forceinline__ void plane_item(const V* in, const PlanePlan& pl, const PlaneThread& th,
                                           uint32_t item, const float* chif, Real diag, Real hpin, bool apbc,
                                           Epi& epi) {
    constexpr int SF = DAG ? -1 : 1;
    constexpr int UP = DAG ? 0 : 2, DN = DAG ? 2 : 0;
    const int U = pl.U, Lt = pl.Lt;
    const PlanePlace w0 = plane_place<SKIP, sizeof(V)>(pl, th, item);
    if (SKIP && w0.none) return;
    const bool act = w0.act;
    const int f = w0.f, u0 = w0.u0, u1 = w0.u1, t = w0.t;
    const uint32_t kv = pl.kvol, site = w0.site, o_0 = w0.o_0, o_xp = w0.o_xp, o_xm = w0.o_xm,
                   o_yp = w0.o_yp, o_ym = w0.o_ym, o_tp = w0.o_tp, o_tm = w0.o_tm;
    const int64_t cst = (int64_t)U * kv;             // component stride
    const int64_t e0 = 4 * f * cst + (int64_t)u0 * kv;
    const V *p0 = in + e0, *p1 = p0 + cst, *p2 = p1 + cst, *p3 = p2 + cst;
    int64_t e = e0;
#pragma unroll 1
    for (int u = u0; u < u1; u++) {
        V acc[4], r[4];
        const bool has_next = u + 1 < U;
        if (u == 0 || u == U - 1) {          // the wall operands, used last
            const V* w = in + (u == 0 ? (int64_t)(U - 1) * kv : 0);
            plane_prefetch(unit_at(w + (u == 0 ? DN : UP) * cst, o_0));
            plane_prefetch(unit_at(w + (u == 0 ? DN + 1 : UP + 1) * cst, o_0));
            plane_prefetch(unit_at(w + (u == 0 ? DN + 4 : UP + 4) * cst, o_0));
            plane_prefetch(unit_at(w + (u == 0 ? DN + 5 : UP + 5) * cst, o_0));
            plane_prefetch(chif + site);
            plane_prefetch(chif + kv + site);
            plane_prefetch(chif + 2 * kv + site);
        }
#define CHDWF_PLANE_LD(N)                \
    {                                    \
        r[0] = ld_unit(unit_at(p0, N));  \
        r[1] = ld_unit(unit_at(p1, N));  \
        r[2] = ld_unit(unit_at(p2, N));  \
        r[3] = ld_unit(unit_at(p3, N));  \
    }
        if (std::is_same<V, double2>::value) {
            CHDWF_PLANE_LD(o_0)
#pragma unroll
            for (int d = 0; d < 4; d++) acc[d] = zscal(diag, r[d]);      // :2651-2667
            CHDWF_PLANE_LD(o_xp)
            plane_hop<0, SF>(acc, r);
        } else {
            CHDWF_PLANE_LD(o_xp)
            plane_first_hop<SF>(acc, r);
        }
        CHDWF_PLANE_LD(o_xm) plane_hop<0, -SF>(acc, r);
        CHDWF_PLANE_LD(o_yp) plane_hop<1, SF>(acc, r);
        CHDWF_PLANE_LD(o_ym) plane_hop<1, -SF>(acc, r);
        CHDWF_PLANE_LD(o_tp) plane_hop<2, SF>(acc, r);
        CHDWF_PLANE_LD(o_tm) plane_hop<2, -SF>(acc, r);
        V cur[4], nx[2], pv[2];
        cur[0] = ld_unit(unit_at(p0, o_0)); cur[1] = ld_unit(unit_at(p1, o_0));
        cur[2] = ld_unit(unit_at(p2, o_0)); cur[3] = ld_unit(unit_at(p3, o_0));
        nx[0] = nx[1] = pv[0] = pv[1] = V{};
        auto load_s = [&] {                  // the units above and below
            if (has_next) {
                nx[0] = ld_unit(unit_at((DAG ? p0 : p2) + kv, o_0));
                nx[1] = ld_unit(unit_at((DAG ? p1 : p3) + kv, o_0));
            }
            if (u > 0) {
                pv[0] = ld_unit(unit_at((DAG ? p2 : p0) - kv, o_0));
                pv[1] = ld_unit(unit_at((DAG ? p3 : p1) - kv, o_0));
            }
        };
        if (!S_LATE) load_s();
        plane_kappa(acc, cur, diag);                                     // :2815-2829
        if (apbc) {                                                      // :2831-2876
            if (t == Lt - 1) { CHDWF_PLANE_LD(o_tp) hop<2, SF, true>(acc, r); }
            if (t == 0) { CHDWF_PLANE_LD(o_tm) hop<2, -SF, true>(acc, r); }
        }
#undef CHDWF_PLANE_LD
        // s hops (:2879-2908; M^dagger :3313-3342)
        if (S_LATE) load_s();
#pragma unroll
        for (int d = 0; d < 2; d++) plane_shop<true>(acc[UP + d], cur[UP + d], nx[d], has_next);
#pragma unroll
        for (int d = 0; d < 2; d++) plane_shop<false>(acc[DN + d], cur[DN + d], pv[d], u > 0);
        // wall coupling: the pair at s=Ls reads s=1, the pair at s=1 reads s=Ls
        if (u == 0 || u == U - 1) {
            const float c1 = chif[site], c2 = chif[kv + site], c3 = chif[2 * kv + site];
            const bool pin = site == 0;
            // half of the last unit that holds s = Ls
            const int hL = std::is_same<V, cpair>::value ? ((pl.Ls & 1) ? 0 : 1) : 0;
            if (u == U - 1)
                plane_wall<DAG, IMASS, UP, 0>(acc, in + site, cst, hL, 0, f, c1, c2, c3, pin, hpin);
            if (u == 0)
                plane_wall<DAG, IMASS, DN, 1>(acc, in + (int64_t)(U - 1) * kv + site, cst, 0, hL, f,
                                              c1, c2, c3, pin, hpin);
            plane_clear_pad(acc, u == U - 1 && (pl.Ls & 1));
        }
        if (!epi(acc, e, cst, o_0, act, u, site)) return;
        p0 += kv; p1 += kv; p2 += kv; p3 += kv;
        e += kv;
    }
}

// ---- between the ABI's layout and planes ---------------------------------------
// Units are visited in plane order: coalesced on that side, Ls elements apart
// on the other.  Once or twice a solve.
struct PlaneUnit { int64_t e; int n; };   // first element in the ABI's layout, elements
template <class T>
__device__ __forceinline__ PlaneUnit plane_unit_of(const Geom& g, int U, int64_t i) {
    constexpr int N = std::is_same<T, float2>::value ? 2 : 1;
    const int64_t cu = i / g.kvol, site = i - cu * g.kvol;
    const int c = (int)(cu / U), u = (int)(cu - (int64_t)c * U);
    return PlaneUnit{(int64_t)N * u + (int64_t)g.Ls * site + g.cs * c,
                     N == 2 && N * u + 1 < g.Ls ? 2 : 1};
}

}  // namespace chdwf
