// Pair terms of the WCSPH loops shared by the list kernels (sph.cu) and the
// cell-tile kernels (sph_tiles.cu): the solid partner quantities, a fluid
// particle's own state, the double-float drift and the Shepard term.  The
// physics and its algebraic forms are described at the top of sph.cu.
#pragma once
#include "kernels.cuh"

namespace demsph {
namespace sph {

constexpr float KG = 5.f * 21.f / (16.f * 3.14159265358979323846f);  // G = KG t^3 / h^5
constexpr float SIG = 21.f / (16.f * 3.14159265358979323846f);       // sigma h^3

struct SolidPartner {
    float3 r;      // x_i - x_a
    float3 v;      // v_a
    float Pa, rhoa, Va, G, rr;
    bool inside;
};

// Wall/solid partner quantities shared by continuity, momentum and coupling.
__device__ __forceinline__ SolidPartner solidPartner(const DeviceState& d, int4 ci, float4 pi, float hi, float Pi,
                                                     float rhoi, float rho0i, float ci2, int a)
{
    SolidPartner s;
    const float4 pa = d.sph[a];
    s.r = relF(ci, pi, d.scell[a], pa, d.grid);
    const float ra = d.srad[a].x;
    const float h = 0.5f * (hi + 2.6f * ra);
    const float r2 = dot3(s.r, s.r);
    s.inside = r2 < 4.f * h * h;
    if (!s.inside) return s;
    s.rr = sqrtf(r2);
    const float t = 1.f - 0.5f * s.rr / h;
    const float h2 = h * h;
    s.G = KG * t * t * t / (h2 * h2 * h);
    s.v = xyz(d.svh[a]);
    const float3 na = xyz(d.snormal[a]);
    const float3 aa = xyz(d.sacc[a]);
    s.Pa = Pi + rhoi * fmaxf(0.f, dot3(d.g - aa, na)) * dot3(s.r, na);
    s.rhoa = s.Pa / ci2 + rho0i;
    s.Va = 8.f * ra * ra * ra;
    return s;
}

struct Self {
    int4 c;
    float4 p;
    float3 v;
    float h, rho0, cs, nu, m, rho, P, V, gam;
};

// U: every fluid particle has the parameters fparU and the smoothing length
// fhmax, kernel constants that take no registers through the loop.
template <bool U = false>
__device__ __forceinline__ Self loadSelf(const DeviceState& d, int i, int ps, int vs, int ds)
{
    Self o;
    o.c = d.fcell[i];
    o.p = d.fph[ps][i];
    o.v = xyz(d.fvh[vs][i]);
    const float dr = d.fdrho[ds][i];
    const float4 par = U ? d.fparU : d.fpar[i];
    o.h = U ? d.fhmax : o.p.w;
    o.rho0 = par.x;
    o.cs = par.y;
    o.nu = par.z;
    o.m = par.w;
    o.rho = o.rho0 + dr;
    o.P = dr * o.cs * o.cs;
    o.V = o.m / o.rho;
    o.gam = o.nu * o.rho;
    return o;
}

// Position/velocity update in double-float: x += v dt.
__device__ __forceinline__ void dfAxpy(float4& xh, float4& xl, float4 vh, float4 vl, dfl dt)
{
    dfl x = df_add(df_make(xh.x, xl.x), df_mul(df_make(vh.x, vl.x), dt));
    dfl y = df_add(df_make(xh.y, xl.y), df_mul(df_make(vh.y, vl.y), dt));
    dfl z = df_add(df_make(xh.z, xl.z), df_mul(df_make(vh.z, vl.z), dt));
    xh.x = x.hi; xl.x = x.lo;
    xh.y = y.hi; xl.y = y.lo;
    xh.z = z.hi; xl.z = z.lo;
}


// ---- Shepard density re-initialisation (integrate.cu:3-53) ----
// sumW = sigma(h_i) S with S = 1 + sum_j f(q_j) + sum_a f(q_a) V0_a / V0_i,
// f(q) = (1 - q/2)^4 (1 + 2q).  The update rho0 S / S0 - rho0 is a difference
// of two nearly equal sums (1e-3 apart), so S is carried in double-float from
// double-float distances, and S - S0 is formed before dividing.
__device__ __forceinline__ dfl shepardTerm(dfl r, dfl invh)
{
    const dfl q = df_mul(r, invh);
    const dfl t = df_add_f(df_mul_f(q, -0.5f), 1.0f);
    const dfl t2 = df_mul(t, t);
    return df_mul(df_mul(t2, t2), df_add_f(df_mul_f(q, 2.0f), 1.0f));
}

// Sum over the L lanes of a group in double-float, in a fixed tree: every lane
// gets the same bits.
template <int L>
__device__ __forceinline__ dfl groupSum(dfl v)
{
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        const dfl u = df_make(__shfl_xor_sync(0xffffffffu, v.hi, o, L), __shfl_xor_sync(0xffffffffu, v.lo, o, L));
        v = (threadIdx.x & o) ? df_add(u, v) : df_add(v, u);
    }
    return v;
}
template <int L>
__device__ __forceinline__ float groupSum(const KahanF& k)
{
    if (L == 1) return k.value();
    const dfl v = groupSum<L>(df_two_sum(k.s, -k.c));
    return v.hi + v.lo;
}

// Groups of four lanes and more end a pass axis by axis: after groupSumAxes the
// first quarter of the lanes carries x, the second y, the others z, and the
// first lane of each (axisLead) moves and stores that component of the particle.
template <int L>
__device__ __forceinline__ int axisOf(int lane)
{
    return min(lane / (L / 4), 2);
}
template <int L>
__device__ __forceinline__ bool axisLead(int lane)
{
    return lane % (L / 4) == 0 && lane < 3 * (L / 4);
}
__device__ __forceinline__ float component(const float4* p, int i, int axis) { return ((const float*)(p + i))[axis]; }
__device__ __forceinline__ float& component(float4* p, int i, int axis) { return ((float*)(p + i))[axis]; }
__device__ __forceinline__ float component(float3 v, int axis) { return axis == 0 ? v.x : axis == 1 ? v.y : v.z; }
// groupSum of three sums at once, the lanes sharing them out as they go: the
// same trees with the same operands in the same order, but four double-float
// additions where three butterflies over eight lanes take nine.
template <int L>
__device__ __forceinline__ float groupSumAxes(const KahanF3& k)
{
    static_assert(L >= 4, "an axis per quarter");
    constexpr unsigned FULL = 0xffffffffu;
    const auto passed = [&](dfl v, int o) { return df_make(__shfl_xor_sync(FULL, v.hi, o, L), __shfl_xor_sync(FULL, v.lo, o, L)); };
    const auto ordered = [&](dfl own, dfl other, bool upper) { return upper ? df_add(other, own) : df_add(own, other); };
    dfl x = df_two_sum(k.x.s, -k.x.c), y = df_two_sum(k.y.s, -k.y.c);
    const dfl z = df_two_sum(k.z.s, -k.z.c);
    const bool half = threadIdx.x & (L / 2), quarter = threadIdx.x & (L / 4);
    {   // the lower half keeps x and y, the upper z (in x)
        const dfl otherX = passed(half ? x : z, L / 2), otherY = passed(y, L / 2);
        x = ordered(half ? z : x, otherX, half);
        y = df_add(y, otherY);
    }
    {   // the second quarter keeps y (in x)
        const dfl other = passed(half || quarter ? x : y, L / 4);
        x = ordered(quarter && !half ? y : x, other, quarter);
    }
#pragma unroll
    for (int o = L / 8; o > 0; o >>= 1) x = ordered(x, passed(x, o), threadIdx.x & o);
    return x.hi + x.lo;
}

}  // namespace sph
}  // namespace demsph
