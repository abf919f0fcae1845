// WCSPH pair loops: Riemann continuity, Riemann momentum and Shepard density
// re-initialisation (the SPH->DEM coupling force, a sum per solid, is in dem.cu).
//
// Physics restated from core/integrate.cu:3-330 (reference) with the Wendland
// C2 kernel of core/SPHKernelDEMContactModel.h:5-32.  Algebraic forms used
// here (equal to the reference's expressions, with fewer operations and no
// cancellation of the Riemann averages):
//   grad W(r, h)   = -G r,  G = 5 sigma t^3 / h^2,  t = 1 - |r| / (2h),
//                    sigma = 21 / (16 pi h^3)        (zero for |r| >= 2h)
//   continuity, fluid partner j (integrate.cu:75-103):
//     dRho/dt += -2 rho_i V_j G / (rho_i + rho_j)
//                * [rho_j (v_i - v_j).r + (P_i - P_j) |r| / c_ij]
//   continuity, solid partner a (integrate.cu:139-158), with the mirrored
//   velocity 2 v_a - v_i and the hydrostatic wall pressure P_a:
//     dRho/dt += -2 rho_i V_a G / (rho_i + rho_a)
//                * [2 rho_a (v_i - v_a).r + (P_i - P_a) |r| / c_i]
//   momentum, fluid partner (integrate.cu:185-213):
//     dv/dt += 2 V_i V_j G / m_i [P* r - gamma_ij (v_i - v_j)]
//   momentum, solid partner (integrate.cu:251-277) and the per-pair coupling
//   force (integrate.cu:282-329, = m_i times the same term):
//     dv/dt += 2 V_i V_a G / m_i [P* r - 2 gamma_i (v_i - v_a)]
// Sums are Kahan-compensated FP32; positions and velocities are integrated
// in double-float.  The continuity pass reads every partner's density as of
// the pass start (dRho is double-buffered).
#include "sph_common.cuh"

namespace demsph {

namespace {

constexpr int T = 128;
using namespace sph;

// The offsets of the 27 walk cells (code = (dz+1) 9 + (dy+1) 3 + dx+1), one
// array per axis in a block's shared memory (filled before the block's first
// early return): three 4-byte reads of 27 words each take a wavefront of the
// L1 apiece, one 16-byte read took four to ten.
struct WalkTable {
    float o[3][32];
};
__device__ __forceinline__ void fillWalkTable(WalkTable& tab, float3 cs)
{
    const int code = threadIdx.x;
    if (code < 27) {
        tab.o[0][code] = (float)(code % 3 - 1) * cs.x;
        tab.o[1][code] = (float)(code / 3 % 3 - 1) * cs.y;
        tab.o[2][code] = (float)(code / 9 - 1) * cs.z;
    }
    __syncthreads();
}

// Relative position of fluid partner entry e of slot i (the products of the
// table are exact, so it changes no bit).
__device__ __forceinline__ float3 fluidRel(const DeviceState& d, const WalkTable& tab, int4 ci, float4 pi, unsigned e,
                                           int j, float4 pj)
{
    if (ffRegular(e)) {
        const int t = entryWalk(e);
        return make_float3((pi.x - pj.x) - tab.o[0][t], (pi.y - pj.y) - tab.o[1][t], (pi.z - pj.z) - tab.o[2][t]);
    }
    return relF(ci, pi, d.fcell[j], pj, d.grid);
}

// ---- batched partner loops ----
// Partners whose state is gathered before any of them is used: B gathers per
// lane are in flight instead of one (depths 1 and 4 are slower; 4 spills).
// Blocks per SM: what the registers of the loop need without spills in it.  A
// pass over 410k particles with 8 / 7 / 6 continuity blocks takes 135 / 124 / 128
// us, with 8 / 7 / 6 momentum blocks 148 / 140 / 142; over 19k with parameters
// of their own the momentum takes 19.9 / 17.9 / 20.0.
#ifndef DEMSPH_PAIR_BATCH
#define DEMSPH_PAIR_BATCH 2
#endif
#ifndef DEMSPH_CONTINUITY_BLOCKS
#define DEMSPH_CONTINUITY_BLOCKS 7  // resident blocks of T per SM the registers allow
#endif
#ifndef DEMSPH_MOMENTUM_BLOCKS
#define DEMSPH_MOMENTUM_BLOCKS 7
#endif
constexpr int BATCH = DEMSPH_PAIR_BATCH;

// E consecutive list entries in one load (streamed: the list is read once a pass).
template <int E>
__device__ __forceinline__ void loadEntries(const unsigned* __restrict__ p, unsigned* e)
{
    if constexpr (E == 8) {
        asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3]), "=r"(e[4]), "=r"(e[5]), "=r"(e[6]), "=r"(e[7])
            : "l"(p));
    } else if constexpr (E == 4) {
        const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p));
        e[0] = v.x, e[1] = v.y, e[2] = v.z, e[3] = v.w;
    } else if constexpr (E == 2) {
        const uint2 v = __ldcs(reinterpret_cast<const uint2*>(p));
        e[0] = v.x, e[1] = v.y;
    } else {
        e[0] = __ldcs(p);
    }
}

// The loop over the m entries of particle i's list by one of its L lanes.  A
// sector of eight entries (listAt) is shared by the lanes, 8 / L consecutive
// entries each in one load; the next sector is read while this one is used.
// gather(e) reads a partner's state, use(e, state, ok) takes B of them at a time
// without a branch on the entry (ok false: past the list's end, where the entry
// is the particle itself), so that the B terms' chains interleave.
template <int L, int B, class Gather, class Use>
__device__ __forceinline__ void forFluidPartners(const unsigned* __restrict__ ff, int n, int i, int lane, int m,
                                                 Gather gather, Use use)
{
    constexpr int E = 8 / L, S = E < B ? B / E : 1, N = E * S;  // entries of a lane per sector, sectors and entries per round
    const size_t stride = (size_t)n * 8;
    const unsigned* p = ff + (size_t)i * 8 + lane * E;
    const int sectors = (m + 7) >> 3;
    const unsigned none = ffEntry(i, 13, true);
    unsigned next[N];
#pragma unroll
    for (int u = 0; u < S; ++u, p += stride)
        if (u < sectors) loadEntries<E>(p, next + u * E);
    for (int s = 0; s < sectors; s += S) {
        unsigned e[N];
        bool ok[N];
#pragma unroll
        for (int c = 0; c < N; ++c) {
            ok[c] = (s + c / E) * 8 + lane * E + c % E < m;
            e[c] = ok[c] ? next[c] : none;
        }
#pragma unroll
        for (int c = 0; c < N; c += B) {
            decltype(gather(0u)) g[B];
#pragma unroll
            for (int u = 0; u < B; ++u) g[u] = gather(e[c + u]);
            if (c == (N / B / 2) * B) {
#pragma unroll
                for (int u = 0; u < S; ++u, p += stride)
                    if (s + S + u < sectors) loadEntries<E>(p, next + u * E);
            }
            use(e + c, g, ok + c);
        }
    }
}

// A fluid partner's state read by the continuity and momentum terms of scenes
// whose fluids differ (the buffers a pass reads are not written by it:
// read-only loads).
struct FluidPartner {
    float4 p, v, par;
    float dr;
};
__device__ __forceinline__ FluidPartner gatherFluid(const DeviceState& d, int j, const float4* __restrict__ ph,
                                                    const float4* __restrict__ vh, const float* __restrict__ dr)
{
    return FluidPartner{__ldg(ph + j), __ldg(vh + j), __ldg(d.fpar + j), __ldg(dr + j)};
}

// A partner of a uniform fluid: the pass's record, one sector in one 32-byte load.
__device__ __forceinline__ FluidRec loadRecord(const FluidRec* __restrict__ p)
{
    FluidRec r;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(r.pc.x), "=f"(r.pc.y), "=f"(r.pc.z), "=f"(r.pc.w), "=f"(r.vd.x), "=f"(r.vd.y), "=f"(r.vd.z), "=f"(r.vd.w)
        : "l"(p));
    return r;
}

// The loop over the partners of a uniform fluid: term(r, record, ok), r the
// relative position.  Entries whose walk cell does not give their offset (lists
// made by the walk) are mended out of line.
template <int L, int B, class Term>
__device__ __forceinline__ void forFluidRecords(const DeviceState& d, const WalkTable& tab, const FluidRec* __restrict__ rec,
                                                int i, int lane, int m, float4 pi, Term term)
{
    forFluidPartners<L, B>(
        d.ff, d.nf, i, lane, m, [&](unsigned e) { return loadRecord(rec + ffPartner(e)); },
        [&](const unsigned* e, const FluidRec* q, const bool* ok) {
            float3 r[B];
            unsigned all = e[0];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int t = entryWalk(e[u]);
                r[u] = make_float3((pi.x - q[u].pc.x) - tab.o[0][t], (pi.y - q[u].pc.y) - tab.o[1][t],
                                   (pi.z - q[u].pc.z) - tab.o[2][t]);
                all &= e[u];
            }
            if (!ffRegular(all)) {
#pragma unroll
                for (int u = 0; u < B; ++u)
                    if (!ffRegular(e[u])) r[u] = relF(d.fcell[i], pi, d.fcell[ffPartner(e[u])], q[u].pc, d.grid);
            }
#pragma unroll
            for (int u = 0; u < B; ++u) term(r[u], q[u], ok[u]);
        });
}

// Approximate reciprocal and square root of the pair terms.  Two particles may
// come so close that their squared distance is a subnormal float, which the root
// takes (its result is normal) at no cost; a reciprocal that takes them too made
// a pass of 410k particles 5 % slower, and none is asked for: distances after the
// root are normal, and so are the densities' products of a uniform fluid.
__device__ __forceinline__ float fastRcp(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float fastSqrt(float x)
{
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// term(e, state) for the entries inside the list, one by one.
template <class Term>
struct EachOf {
    Term term;
    template <class State, int B>
    __device__ __forceinline__ void operator()(const unsigned* e, const State (&q)[B], const bool* ok) const
    {
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (ok[u]) term(e[u], q[u]);
    }
};
template <class Term>
__device__ __forceinline__ EachOf<Term> eachOf(Term term)
{
    return EachOf<Term>{term};
}

// ---- lane groups ----
// A fluid particle's neighbour loop is split over a group of L lanes (L a
// power of two <= 32, chosen per scene so that small scenes still fill the
// GPU); the lanes' compensated partial sums are added in a fixed tree, so the
// result does not depend on timing.  Kernels return early only for whole
// warps: the shuffles take every lane.
// ---- continuity (+ optional drift) ----
// What bounds the pair loops: in large scenes L1 wavefronts, one for nearly every
// sector gathered (90 % of their peak at 410k particles, spills in the loop a
// fifteenth of them), in small ones latency of the gathers.  A partner is one
// 32-byte record in one load, the terms of a round run without branches, two
// lanes share a list sector, and a uniform fluid's own state is its position,
// velocity and density (its parameters are kernel constants, and what its solid
// partners need is read again where it has any): 400k particles 131 to 124 us
// with the last (160 with four reads a partner; momentum 202, 140), 1.0M 306 to
// 286 (327 to 321).
struct ContinuityArgs {
    int ps, vs, ds, dd;  // position / velocity / density source, density destination
    int rec;             // partner records read (uniform fluids): position ps, velocity vs, density ds
    int recOut;          // -1: none; else frec[recOut] receives the drifted position, the velocity and density dd
    int driftTo;         // -1: no drift; else position buffer receiving x + v * drift
    int velCopyTo;       // -1: none; else velocity buffer receiving a copy of this particle's velocity
    int countStep;       // 1: the pass ends the step (nothing after it can raise a status): count it
    float dt;
    dfl drift;
};

template <int L, bool U>
__global__ void __launch_bounds__(T, DEMSPH_CONTINUITY_BLOCKS) kContinuity(DeviceState d, ContinuityArgs a)
{
    stepKernelBegin();
    __shared__ WalkTable walkTab;
    fillWalkTable(walkTab, d.grid.cs);
    if (a.countStep && blockIdx.x == 0 && threadIdx.x == 0 && *d.status == 0) atomicAdd(d.stepsDone, 1);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= d.nf * L || *d.status) return;
    const int i = t / L, lane = t % L;
    const bool live = i < d.nf;
    KahanF acc;
    if (live) {
        const int n = d.nf;
        const int nff = min(d.ffc[i], d.kff), nfs = min(d.fsc[i], d.kfs);
        int next = 0;  // solid partner, read ahead (the first beside the fluids in groups of four lanes and more)
        if (L >= 4 && lane < nfs) next = d.fs[listAt(lane, i, n)];
        if constexpr (U) {
            // every fluid particle has the same rest density, sound speed,
            // viscosity, mass and smoothing length: the kernel's constants come
            // from the kernel parameters, P_i - P_j = c^2 (dRho_i - dRho_j)
            const float4 pI = d.fph[a.ps][i];
            const float3 vI = xyz(d.fvh[a.vs][i]);
            const float drhoI = d.fdrho[a.ds][i], rhoI = d.fparU.x + drhoI;
            const float scale = -2.f * rhoI * d.fparU.w * d.fconstU.z;
            forFluidRecords<L, BATCH>(
                d, walkTab, d.frec[a.rec], i, lane, nff, pI, [&](float3 r, const FluidRec& q, bool ok) {
                    const float r2 = ok ? dot3(r, r) : d.fconstU.x;
                    const float rhoj = d.fparU.x + q.vd.w;
                    const float rr = fastSqrt(r2);
                    const float tt = 1.f - rr * d.fconstU.y;
                    const float3 vij = vI - xyz(q.vd);
                    const float flux = rhoj * dot3(vij, r) + (drhoI - q.vd.w) * d.fparU.y * rr;
                    const float term = scale * (tt * tt * tt) * fastRcp(rhoj * (rhoI + rhoj)) * flux;
                    acc.add(r2 >= d.fconstU.x ? 0.f : term);
                });
        } else {
            const Self o = loadSelf(d, i, a.ps, a.vs, a.ds);
            const float4* __restrict__ ph = d.fph[a.ps];
            const float4* __restrict__ vh = d.fvh[a.vs];
            const float* __restrict__ drh = d.fdrho[a.ds];
            forFluidPartners<L, BATCH>(
                d.ff, n, i, lane, nff, [&](unsigned e) { return gatherFluid(d, ffPartner(e), ph, vh, drh); },
                eachOf([&](unsigned e, const FluidPartner& q) {
                    const float3 r = fluidRel(d, walkTab, o.c, o.p, e, ffPartner(e), q.p);
                    const float r2 = dot3(r, r);
                    const float h = 0.5f * (o.h + q.p.w);
                    if (r2 >= 4.f * h * h) return;
                    const float rhoj = q.par.x + q.dr;
                    const float Pj = q.dr * q.par.y * q.par.y;
                    const float Vj = q.par.w / rhoj;
                    const float rr = sqrtf(r2);
                    const float tt = 1.f - 0.5f * rr / h;
                    const float h2 = h * h;
                    const float G = KG * tt * tt * tt / (h2 * h2 * h);
                    const float c = 0.5f * (o.cs + q.par.y);
                    const float3 vij = o.v - xyz(q.v);
                    acc.add(-2.f * o.rho * Vj * G / (o.rho + rhoj) * (rhoj * dot3(vij, r) + (o.P - Pj) * rr / c));
                }));
        }
        if (L < 4 && lane < nfs) next = d.fs[listAt(lane, i, n)];
        if (lane < nfs) {  // near a wall: the particle's state again, not kept through the fluid loop
            const Self o = loadSelf<U>(d, i, a.ps, a.vs, a.ds);
            const float ci2 = o.cs * o.cs;
            for (int k = lane; k < nfs; k += L) {
                const int sa = fsPartner(next);
                if (k + L < nfs) next = d.fs[listAt(k + L, i, n)];
                const SolidPartner sp = solidPartner(d, o.c, o.p, o.h, o.P, o.rho, o.rho0, ci2, sa);
                if (!sp.inside) continue;
                acc.add(-2.f * o.rho * sp.Va * sp.G / (o.rho + sp.rhoa) *
                        (2.f * sp.rhoa * dot3(o.v - sp.v, sp.r) + (o.P - sp.Pa) * sp.rr / o.cs));
            }
        }
    }
    const float sum = groupSum<L>(acc);
    if (!live) return;
    const float drho = d.fdrho[a.ds][i] + a.dt * sum;
    if (lane == 0) d.fdrho[a.dd][i] = drho;
    if (a.driftTo >= 0) {
        if constexpr (L >= 4) {
            const int x = axisOf<L>(lane);
            const float v = component(d.fvh[a.vs], i, x);
            const dfl p = df_add(df_make(component(d.fph[a.ps], i, x), component(d.fpl[a.ps], i, x)),
                                 df_mul(df_make(v, component(d.fvl[a.vs], i, x)), a.drift));
            if (axisLead<L>(lane)) {
                component(d.fph[a.driftTo], i, x) = p.hi;
                component(d.fpl[a.driftTo], i, x) = p.lo;
                if (x == 2) d.fph[a.driftTo][i].w = U ? d.fhmax : d.fph[a.ps][i].w;
                if (U && a.recOut >= 0) {
                    FluidRec& rec = d.frec[a.recOut][i];
                    component(&rec.pc, 0, x) = p.hi;
                    component(&rec.vd, 0, x) = v;
                    if (x == 2) rec.vd.w = drho;
                }
            }
        } else if (lane == 0) {
            float4 xh = d.fph[a.ps][i], xl = d.fpl[a.ps][i];
            const float4 v = d.fvh[a.vs][i];
            dfAxpy(xh, xl, v, d.fvl[a.vs][i], a.drift);
            d.fph[a.driftTo][i] = xh;
            d.fpl[a.driftTo][i] = xl;
            if (U && a.recOut >= 0)
                d.frec[a.recOut][i] = FluidRec{make_float4(xh.x, xh.y, xh.z, 0.f), make_float4(v.x, v.y, v.z, drho)};
        }
    }
    if (a.velCopyTo >= 0) {
        if (lane == 0) d.fvh[a.velCopyTo][i] = d.fvh[a.vs][i];
        if (lane == (L > 1 ? 1 : 0)) d.fvl[a.velCopyTo][i] = d.fvl[a.vs][i];
    }
}

// ---- momentum + kick (dt_f) + drift (dt_f / 2) ----
// Reads position [1], velocity [0], density [1]; writes acc, velocity [1] and
// position [0] (the buffers no other thread reads in this pass).
// Groups of four lanes and more close it axis by axis (groupSumAxes): with one
// lane for all three, 48k particles took 30.9 us, here 29.0 (both with the 2 us
// of a timed stage).
template <int L, bool U>
__global__ void __launch_bounds__(T, DEMSPH_MOMENTUM_BLOCKS) kMomentum(DeviceState d, dfl dtf, dfl halfDtf)
{
    stepKernelBegin();
    __shared__ WalkTable walkTab;
    fillWalkTable(walkTab, d.grid.cs);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= d.nf * L || *d.status) return;
    const int i = t / L, lane = t % L;
    const bool live = i < d.nf;
    KahanF3 acc;
    if (live) {
        const int n = d.nf;
        const int nff = min(d.ffc[i], d.kff), nfs = min(d.fsc[i], d.kfs);
        int next = 0;  // solid partner, read ahead (the first beside the fluids in groups of four lanes and more)
        if (L >= 4 && lane < nfs) next = d.fs[listAt(lane, i, n)];
        if constexpr (U) {  // see kContinuity
            const float4 pI = d.fph[1][i];
            const float3 vI = xyz(d.fvh[0][i]);
            const float drhoI = d.fdrho[1][i], rhoI = d.fparU.x + drhoI;
            const float c2 = d.fparU.y * d.fparU.y, PI = drhoI * d.fparU.y * d.fparU.y;
            const float twoNuRhoI = 2.f * d.fparU.z * rhoI, scale = 2.f * (d.fparU.w / rhoI) * d.fconstU.z;
            forFluidRecords<L, BATCH>(
                d, walkTab, d.frec[1], i, lane, nff, pI, [&](float3 r, const FluidRec& q, bool ok) {
                    const float r2 = ok ? dot3(r, r) : d.fconstU.x;
                    const float rhoj = d.fparU.x + q.vd.w;
                    const float Pj = q.vd.w * c2;
                    const float rr = fastSqrt(r2);
                    const float tt = 1.f - rr * d.fconstU.y;
                    const float3 vij = vI - xyz(q.vd);
                    const float dU = -dot3(vij, r) * fastRcp(rr);  // U_L - U_R
                    const float beta = fminf(3.f * fmaxf(dU, 0.f), d.fparU.y);
                    const float invSum = fastRcp(rhoI + rhoj);
                    const float Ps = (rhoI * Pj + rhoj * PI + rhoI * rhoj * beta * dU) * invSum;
                    const float gbar = twoNuRhoI * rhoj * invSum;  // 2 g_i g_j / (g_i + g_j), g = nu rho
                    // 2 V_i V_j G / m, V_j = m / rho_j
                    const float w = scale * (tt * tt * tt) * fastRcp(rhoj);
                    const float3 term = (r * Ps - vij * gbar) * w;
                    acc.add(r2 >= d.fconstU.x ? make_float3(0.f, 0.f, 0.f) : term);
                });
        } else {
            const Self o = loadSelf(d, i, 1, 0, 1);
            forFluidPartners<L, BATCH>(
                d.ff, n, i, lane, nff,
                [&](unsigned e) { return gatherFluid(d, ffPartner(e), d.fph[1], d.fvh[0], d.fdrho[1]); },
                eachOf([&](unsigned e, const FluidPartner& q) {
                    const float3 r = fluidRel(d, walkTab, o.c, o.p, e, ffPartner(e), q.p);
                    const float r2 = dot3(r, r);
                    const float h = 0.5f * (o.h + q.p.w);
                    if (r2 >= 4.f * h * h) return;
                    const float rhoj = q.par.x + q.dr;
                    const float Pj = q.dr * q.par.y * q.par.y;
                    const float Vj = q.par.w / rhoj;
                    const float gj = q.par.z * rhoj;
                    const float rr = sqrtf(r2);
                    const float tt = 1.f - 0.5f * rr / h;
                    const float h2 = h * h;
                    const float G = KG * tt * tt * tt / (h2 * h2 * h);
                    const float c = 0.5f * (o.cs + q.par.y);
                    const float3 vij = o.v - xyz(q.v);
                    const float dU = -dot3(vij, r) / rr;  // U_L - U_R
                    const float beta = fminf(3.f * fmaxf(dU, 0.f), c);
                    const float Ps = (o.rho * Pj + rhoj * o.P + o.rho * rhoj * beta * dU) / (o.rho + rhoj);
                    const float gbar = 2.f * o.gam * gj / (o.gam + gj);
                    const float w = 2.f * o.V * Vj * G / o.m;
                    acc.add((r * Ps - vij * gbar) * w);
                }));
        }
        if (L < 4 && lane < nfs) next = d.fs[listAt(lane, i, n)];
        if (lane < nfs) {
            const Self o = loadSelf<U>(d, i, 1, 0, 1);
            const float ci2 = o.cs * o.cs;
            for (int k = lane; k < nfs; k += L) {
                const int sa = fsPartner(next);
                if (k + L < nfs) next = d.fs[listAt(k + L, i, n)];
                const SolidPartner sp = solidPartner(d, o.c, o.p, o.h, o.P, o.rho, o.rho0, ci2, sa);
                if (!sp.inside) continue;
                const float3 via = o.v - sp.v;
                const float dU = -2.f * dot3(via, xyz(d.snormal[sa]));
                const float beta = fminf(3.f * fmaxf(dU, 0.f), o.cs);
                const float Ps = (o.rho * sp.Pa + sp.rhoa * o.P + o.rho * sp.rhoa * beta * dU) / (o.rho + sp.rhoa);
                const float w = 2.f * o.V * sp.Va * sp.G / o.m;
                acc.add((sp.r * Ps - via * (2.f * o.gam)) * w);
            }
        }
    }
    float dx, dy, dz;  // moved since the candidates were listed
    if constexpr (L >= 4) {
        const int x = axisOf<L>(lane), j = live ? i : 0;
        const float vh0 = component(d.fvh[0], j, x), vl0 = component(d.fvl[0], j, x), xh = component(d.fph[1], j, x),
                    xl = component(d.fpl[1], j, x), p0 = component(d.fvref, j, x);
        const int c = ((const int*)(d.fcell + j))[x];
        const float acl = groupSumAxes<L>(acc) + component(d.g, x);
        const dfl v = df_add(df_make(vh0, vl0), df_mul_f(dtf, acl));       // kick: v += a dt_f
        const dfl p = df_add(df_make(xh, xl), df_mul(v, halfDtf));         // drift: x += v dt_f / 2
        if (live && axisLead<L>(lane)) {
            component(d.facc, i, x) = acl;
            component(d.fvh[1], i, x) = v.hi;
            component(d.fvl[1], i, x) = v.lo;
            component(d.fph[0], i, x) = p.hi;
            component(d.fpl[0], i, x) = p.lo;
            if (U) {  // the second continuity pass's partners
                FluidRec& rec = d.frec[2][i];
                component(&rec.pc, 0, x) = p.hi;
                component(&rec.vd, 0, x) = v.hi;
                if (x == 2) rec.vd.w = d.fdrho[1][i];
            }
        }
        const float moved = (float)c * component(d.grid.cs, x) + p.hi - p0;
        dx = __shfl_sync(0xffffffffu, moved, 0, L);
        dy = __shfl_sync(0xffffffffu, moved, L / 4, L);
        dz = __shfl_sync(0xffffffffu, moved, L / 2, L);
        if (!live || lane != 0) return;
    } else {
        const float3 sum = make_float3(groupSum<L>(acc.x), groupSum<L>(acc.y), groupSum<L>(acc.z));
        if (!live || lane != 0) return;
        const float3 acl = sum + d.g;
        d.facc[i] = f4(acl);
        // kick: v += a dt_f
        const float4 vh0 = d.fvh[0][i], vl0 = d.fvl[0][i];
        const dfl vx = df_add(df_make(vh0.x, vl0.x), df_mul_f(dtf, acl.x));
        const dfl vy = df_add(df_make(vh0.y, vl0.y), df_mul_f(dtf, acl.y));
        const dfl vz = df_add(df_make(vh0.z, vl0.z), df_mul_f(dtf, acl.z));
        const float4 vh = make_float4(vx.hi, vy.hi, vz.hi, 0.f), vl = make_float4(vx.lo, vy.lo, vz.lo, 0.f);
        d.fvh[1][i] = vh;
        d.fvl[1][i] = vl;
        // drift: x += v dt_f / 2
        float4 xh = d.fph[1][i], xl = d.fpl[1][i];
        dfAxpy(xh, xl, vh, vl, halfDtf);
        d.fph[0][i] = xh;
        d.fpl[0][i] = xl;
        if (U)  // the second continuity pass's partners
            d.frec[2][i] = FluidRec{make_float4(xh.x, xh.y, xh.z, 0.f), make_float4(vh.x, vh.y, vh.z, d.fdrho[1][i])};
        const int4 c = d.fcell[i];
        const float4 p0 = d.fvref[i];
        dx = (float)c.x * d.grid.cs.x + xh.x - p0.x;
        dy = (float)c.y * d.grid.cs.y + xh.y - p0.y;
        dz = (float)c.z * d.grid.cs.z + xh.z - p0.z;
    }
    // the fluid candidates go stale once a particle has moved half the margin
    const float half = 0.5f * d.fskin;
    if (!(dx * dx + dy * dy + dz * dz <= half * half)) *(volatile int*)d.frebuild = 1;
}

// The first continuity pass's partner records from the state.
__global__ void kFluidRecords(DeviceState d)
{
    stepKernelBegin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nf || *d.status) return;
    const float4 x = d.fph[0][i], v = d.fvh[0][i];
    d.frec[0][i] = FluidRec{make_float4(x.x, x.y, x.z, packCell(d.fcell[i])), make_float4(v.x, v.y, v.z, d.fdrho[0][i])};
}

// The walk cells' offsets in double-float (exact: the code's -1, 0 or 1 times
// the cell size).
struct WalkTableDF {
    float hi[3][32], lo[3][32];
};
__device__ __forceinline__ void fillWalkTableDF(WalkTableDF& tab, const GridDev& g)
{
    const int code = threadIdx.x;
    if (code < 27) {
        const float x = (float)(code % 3 - 1), y = (float)(code / 3 % 3 - 1), z = (float)(code / 9 - 1);
        tab.hi[0][code] = x * g.csx.hi;
        tab.lo[0][code] = x * g.csx.lo;
        tab.hi[1][code] = y * g.csy.hi;
        tab.lo[1][code] = y * g.csy.lo;
        tab.hi[2][code] = z * g.csz.hi;
        tab.lo[2][code] = z * g.csz.lo;
    }
    __syncthreads();
}
// One axis of x_i - x_j: the differences of the leading parts and of the trailing
// ones with their rounding errors (34 operations to the 44 of two double-float
// additions).
__device__ __forceinline__ dfl relTable(float hi, float lo, float hj, float lj, float oh, float ol)
{
    const dfl a = df_two_sum(hi, -hj), b = df_two_sum(a.hi, -oh);
    const dfl l = df_two_sum(lo, -lj), m = df_two_sum(l.hi, -ol);
    const dfl r = df_fast_two_sum(b.hi, __fadd_rn(m.hi, __fadd_rn(a.lo, b.lo)));
    return df_fast_two_sum(r.hi, __fadd_rn(r.lo, __fadd_rn(l.lo, m.lo)));
}
// A sum of double-floats: leading parts error-free into two words, what those
// leave and the trailing parts into a third (14 operations a term to df_add's
// 20, and fewer roundings).
struct DFSum {
    float a, b, c;
    __device__ __forceinline__ void add(float hi, float lo)
    {
        const dfl s = df_two_sum(a, hi), t = df_two_sum(b, s.lo);
        a = s.hi;
        b = t.hi;
        c = __fadd_rn(c, __fadd_rn(t.lo, lo));
    }
    __device__ __forceinline__ dfl value() const
    {
        const dfl s = df_two_sum(a, b);
        return df_fast_two_sum(s.hi, __fadd_rn(s.lo, c));
    }
};
// S += f(|x| / h), f(q) = (1 - q/2)^4 (1 + 2q) (shepardTerm): every product and
// sum of leading parts with its rounding error, the trailing products fused and
// each result normalised; no branch.  With t = 1 - q/2 the second factor is
// 5 - 4t, and both leading terms are known to be the larger ones.  Beyond the
// support (f is 1e-28 within the rounding of q at its edge) and for entries past
// the list (ok false) nothing is added.
// Bound by these operations: the re-initialisation of 48k particles (30 partners)
// takes 47.6 us, with double-float arithmetic throughout 62, of 410k 255.  Against
// 64 bits (a host emulation, distances and cells at random, h from 1e-4 to 150,
// root and reciprocal off by up to one unit): a term 1.24e-15 rms and 1.8e-14 at
// most, with double-float throughout 1.25e-15 and 1.9e-14 (42 us, but 1.64e-15 and
// 2.6e-14, with the trailing parts summed in plain float); sums of 64 terms
// 1.4e-14 and 3.2e-14 rms.
__device__ __forceinline__ void addShepardTerm(DFSum& S, dfl x, dfl y, dfl z, dfl invh, bool ok)
{
    const dfl xx = df_two_prod(x.hi, x.hi), yy = df_two_prod(y.hi, y.hi), zz = df_two_prod(z.hi, z.hi);
    const dfl s1 = df_two_sum(xx.hi, yy.hi), s2 = df_two_sum(s1.hi, zz.hi);
    const float lx = __fmaf_rn(2.f * x.hi, x.lo, xx.lo), ly = __fmaf_rn(2.f * y.hi, y.lo, yy.lo),
                lz = __fmaf_rn(2.f * z.hi, z.lo, zz.lo);
    const dfl s = df_fast_two_sum(s2.hi, ((lx + ly) + s1.lo) + (lz + s2.lo));
    // the root: one correction of the approximate float root and of the
    // reciprocal, then the residual's share
    const float r0 = fastSqrt(s.hi), w0 = 0.5f * fastRcp(r0);
    const float r = r0 > 0.f ? __fmaf_rn(__fmaf_rn(-r0, r0, s.hi), w0, r0) : r0;
    const float w1 = __fmaf_rn(w0, __fmaf_rn(-2.f * r, w0, 1.f), w0);
    const float rl = r0 > 0.f ? (__fmaf_rn(-r, r, s.hi) + s.lo) * w1 : 0.f;
    const dfl q = df_two_prod(r, invh.hi);
    const float ql = __fmaf_rn(rl, invh.hi, __fmaf_rn(r, invh.lo, q.lo));
    const dfl u = df_fast_two_sum(1.f, -0.5f * q.hi), t = df_fast_two_sum(u.hi, __fmaf_rn(-0.5f, ql, u.lo));  // 1 - q/2
    const auto square = [](dfl v) {
        const dfl p = df_two_prod(v.hi, v.hi);
        return df_fast_two_sum(p.hi, __fmaf_rn(2.f * v.hi, v.lo, p.lo));
    };
    const dfl t4 = square(square(t)), v = df_fast_two_sum(5.f, -4.f * t.hi),
              w = df_fast_two_sum(v.hi, __fmaf_rn(-4.f, t.lo, v.lo));  // 1 + 2q = 5 - 4 (1 - q/2)
    dfl f = df_two_prod(t4.hi, w.hi);
    f.lo = __fmaf_rn(t4.lo, w.hi, __fmaf_rn(t4.hi, w.lo, f.lo));
    const bool in = ok && !(t.hi <= 0.f);
    S.add(in ? f.hi : 0.f, in ? f.lo : 0.f);
}

template <int L>
__global__ void __launch_bounds__(T) kDensityReinit(DeviceState d, int storeReference)
{
    stepKernelBegin();
    __shared__ WalkTableDF tab;
    fillWalkTableDF(tab, d.grid);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= d.nf * L || *d.status) return;
    const int i = t / L, lane = t % L;
    const bool live = i < d.nf;
    dfl S = df_make(lane == 0 ? 1.f : 0.f);
    if (live) {
        const int4 ci = d.fcell[i];
        const float4 pi = d.fph[0][i], li = d.fpl[0][i];
        const dfl h = df_make(pi.w, li.w);
        const dfl invh = df_div(df_make(1.f), h);
        const dfl twoH = df_add(h, h);
        const int n = d.nf;
        const int nff = min(d.ffc[i], d.kff);
        struct PartnerPosition {
            float4 h, l;
        };
        DFSum fluid = {0.f, 0.f, 0.f};
        forFluidPartners<L, BATCH>(
            d.ff, n, i, lane, nff,
            [&](unsigned e) {
                const int j = ffPartner(e);
                return PartnerPosition{__ldg(d.fph[0] + j), __ldg(d.fpl[0] + j)};
            },
            [&](const unsigned* e, const PartnerPosition* q, const bool* ok) {
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int t = entryWalk(e[u]);
                    dfl x = relTable(pi.x, li.x, q[u].h.x, q[u].l.x, tab.hi[0][t], tab.lo[0][t]);
                    dfl y = relTable(pi.y, li.y, q[u].h.y, q[u].l.y, tab.hi[1][t], tab.lo[1][t]);
                    dfl z = relTable(pi.z, li.z, q[u].h.z, q[u].l.z, tab.hi[2][t], tab.lo[2][t]);
                    if (!ffRegular(e[u])) {
                        const DF3 w = relDF(ci, pi, li, d.fcell[ffPartner(e[u])], q[u].h, q[u].l, d.grid);
                        x = w.x, y = w.y, z = w.z;
                    }
                    addShepardTerm(fluid, x, y, z, invh, ok[u]);
                }
            });
        S = df_add(S, fluid.value());
        // V0_a / V0_i = (2 r_a / (h_i / 1.3))^3 = (2.6 r_a / h_i)^3
        const dfl k26 = df_from_double(2.6);
        const int nfs = min(d.fsc[i], d.kfs);
        for (int k = lane; k < nfs; k += L) {
            const int a = fsPartner(d.fs[listAt(k, i, n)]);
            const dfl r = dfNorm(relDF(ci, pi, li, d.scell[a], d.sph[a], d.spl[a], d.grid));
            if (df_ge0(df_sub(r, twoH))) continue;
            const float4 ra = d.srad[a];
            const dfl x = df_mul(df_mul(k26, df_make(ra.x, ra.y)), invh);
            const dfl vr = df_mul(df_mul(x, x), x);
            S = df_add(S, df_mul(shepardTerm(r, invh), vr));
        }
    }
    S = groupSum<L>(S);
    if (!live || lane != 0) return;
    if (storeReference) {
        d.fsumW0[i] = make_float2(S.hi, S.lo);
    } else {
        const float2 s0 = d.fsumW0[i];
        const dfl diff = df_sub(S, df_make(s0.x, s0.y));
        const float rho0 = d.fpar[i].x;
        // max(rho*, rho0 S / S0) - rho0 = max(dRho, rho0 (S - S0) / S0)
        const float cand = rho0 * ((diff.hi + diff.lo) / s0.x);
        const float drho = fmaxf(d.fdrho[0][i], cand);
        d.fdrho[0][i] = drho;
        if (d.uniformFluid) d.frec[0][i].vd.w = drho;
    }
}

}  // namespace

void launchDensityReinit(const DeviceState& d, int iStep, cudaStream_t s)
{
    if (d.nf <= 0) return;
    if (d.fluidTiles) return launchTileShepard(d, iStep, s);
    LAUNCH_LANES(kDensityReinit, d.lanes, d.nf, T, s, d, iStep == 1 ? 1 : 0);
}

int fluidLanes(int nf)
{
    int L = 2;
    while (L < 8 && (long long)nf * L < 152LL * 2048) L *= 2;
    return L;
}

void launchContinuityPass(const DeviceState& d, int which, double dtf, cudaStream_t s, bool countStep)
{
    if (d.nf <= 0) return;
    if (d.fluidTiles) return launchTileContinuity(d, which, dtf, s, countStep);
    ContinuityArgs a;
    a.countStep = countStep ? 1 : 0;
    a.dt = (float)(0.5 * dtf);
    a.drift = df_from_double(0.5 * dtf);
    if (which == 0) {  // first half step: densities 0 -> 1, drift positions 0 -> 1
        a.ps = 0; a.vs = 0; a.ds = 0; a.dd = 1; a.driftTo = 1; a.velCopyTo = -1; a.rec = 0; a.recOut = 1;
    } else {           // second half step: densities 1 -> 0, velocity 1 -> 0
        a.ps = 0; a.vs = 1; a.ds = 1; a.dd = 0; a.driftTo = -1; a.velCopyTo = 0; a.rec = 2; a.recOut = -1;
    }
    if (d.uniformFluid) LAUNCH_LANES_U(kContinuity, true, d.lanes, d.nf, T, s, d, a);
    else LAUNCH_LANES_U(kContinuity, false, d.lanes, d.nf, T, s, d, a);
}

void launchFluidRecords(const DeviceState& d, cudaStream_t s)
{
    if (d.nf <= 0 || !d.uniformFluid) return;
    launchStep(kFluidRecords, blocksFor(d.nf, 256), 256, s, d);
}

void launchMomentumPass(const DeviceState& d, double dtf, cudaStream_t s)
{
    if (d.nf <= 0) return;
    if (d.fluidTiles) return launchTileMomentum(d, dtf, s);
    if (d.uniformFluid) LAUNCH_LANES_U(kMomentum, true, d.lanes, d.nf, T, s, d, df_from_double(dtf), df_from_double(0.5 * dtf));
    else LAUNCH_LANES_U(kMomentum, false, d.lanes, d.nf, T, s, d, df_from_double(dtf), df_from_double(0.5 * dtf));
}

}  // namespace demsph
