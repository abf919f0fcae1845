// Neighbour and contact lists.
//
// Reference: setFluidInteractionsKernel (core/neighborSearch.cu:115-220) and
// setSolid2SolidInteractionsKernel (:222-312) walk the 27 cells around each
// particle in (z, y, x) order and, within a cell, in (index) order, and keep
// HALF lists (i < j) in CSR form, evaluated from both sides later through
// reverse spans.  Pair membership is decided once per rebuild, on the
// positions of that moment, with FP64 distances.
//
// Here the same walk, the same order and the same membership test (a FP32
// distance with a 1e-5 margin, and a double-float distance inside the margin,
// so decisions agree with the FP64 reference), but:
//   * fluid lists are FULL lists (both directions) per fluid slot, in sectors
//     of eight entries (listAt), and each entry carries the cell delta of the
//     pair so the SPH loops never load the partner's cell;
//   * solid contacts are a forward CSR (A < B, by original index - the
//     reference's list exactly) plus a per-particle reverse CSR of the lower
//     partners, both filled in walk order; spring history is remapped by
//     looking the pair (A, B) up in A's previous forward segment, which holds
//     the same springs the reference finds through B's reverse span.
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "contact_rows.cuh"

namespace demsph {

namespace {

constexpr int T = 128;


__device__ __forceinline__ dfl dfMax(dfl a, dfl b) { return (a.hi > b.hi || (a.hi == b.hi && a.lo >= b.lo)) ? a : b; }

// Stencil walk shared by all list builders: calls f(hash, regular, hx, hy, hz)
// for the 27 cells around the (truncated) cell of a point, in the reference's
// order, skipping hashes outside [0, num).  "regular" means the hash is an
// in-domain cell whose coordinates are (hx, hy, hz); otherwise (aliased rows,
// overflow bucket) members carry their own cells.
template <class F>
__device__ __forceinline__ void forStencil(int4 c, float4 h, float4 l, const GridDev& g, F&& f)
{
    const int sx = truncAxis(c.x, h.x, l.x), sy = truncAxis(c.y, h.y, l.y), sz = truncAxis(c.z, h.z, l.z);
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                const int hx = sx + dx, hy = sy + dy, hz = sz + dz;
                const int hash = hz * g.gy * g.gx + hy * g.gx + hx;
                if (hash < 0 || hash >= g.num) continue;
                f(hash, inDomain(hx, hy, hz, g), hx, hy, hz);
            }
}

// ---- fluid lists (full) ----
// One particle's 27-cell walk split over a group of L lanes: lane l takes the
// walk positions t = l, l + L, ...  The group advances in lockstep, one
// candidate per lane per round; the accepted entries of a round are written
// in lane order after the entries of earlier rounds (a warp ballot gives each
// its slot), so the list is complete and its order fixed, though not the
// walk order (exports restore that from the walk positions in the entries).
struct LaneWalk {
    int t, p, pe, hx, hy, hz, hash;
    bool regular;
};

// Next candidate in lane's share of the walk over the cell ranges `start`
// (fluid or solid cells); returns false when the share is exhausted.
template <int L>
__device__ __forceinline__ bool nextCandidate(LaneWalk& w, const int* __restrict__ start, int sx, int sy, int sz,
                                              const GridDev& g, int& idx)
{
    while (w.p >= w.pe) {
        w.t += L;
        if (w.t >= 27) return false;
        const int dx = w.t % 3 - 1, dy = (w.t / 3) % 3 - 1, dz = w.t / 9 - 1;
        w.hx = sx + dx;
        w.hy = sy + dy;
        w.hz = sz + dz;
        w.hash = w.hz * g.gy * g.gx + w.hy * g.gx + w.hx;
        if (w.hash < 0 || w.hash >= g.num) continue;
        w.regular = inDomain(w.hx, w.hy, w.hz, g);
        w.p = start[w.hash];
        w.pe = start[w.hash + 1];
    }
    idx = w.p++;
    return true;
}

// ---- candidate rebuild: rows of cells ----
// Lanes of a particle in the list kernels of small scenes (walk, candidate
// rebuild, filter), whatever the pair loops use: eight lanes read neighbouring
// members or one sector of candidates, and write whole sectors of their list.
constexpr int LIST_LANES = 8;

// Appends entries to the list of a particle (row layout listAt) from its
// LIST_LANES lanes: the lanes' entries are collected in shared memory and
// written a full 32-byte sector at a time.  Called by whole warps; `ring` holds
// two sectors per particle of the block.
struct ListRing {
    unsigned v[T / LIST_LANES][16];
};
struct ListWriter {
    unsigned* ring;
    unsigned* out;  // first sector of the particle's list
    size_t stride;  // from one of its sectors to the next
    int k, cap;
    __device__ __forceinline__ ListWriter(ListRing& r, unsigned* list, int i, int n, int capacity)
        : ring(r.v[threadIdx.x / LIST_LANES]), out(list + (size_t)i * 8), stride((size_t)n * 8), k(0), cap(capacity)
    {
    }
    __device__ __forceinline__ void add(bool take, unsigned value)
    {
        const int lane = threadIdx.x & (LIST_LANES - 1), shift = (threadIdx.x & 31) & ~(LIST_LANES - 1);
        const unsigned mine = (__ballot_sync(0xffffffffu, take) >> shift) & ((1u << LIST_LANES) - 1u);
        if (take) ring[(k + __popc(mine & ((1u << lane) - 1u))) & 15] = value;
        __syncwarp();
        const int next = k + __popc(mine);
        if ((next ^ k) & ~7) {  // a sector is full
            const int sector = k >> 3;
            if (sector * 8 < cap) out[sector * stride + lane] = ring[((sector & 1) << 3) + lane];
        }
        k = next;
        __syncwarp();
    }
    // the last sector, part full; returns the number of entries
    __device__ __forceinline__ int finish()
    {
        const int lane = threadIdx.x & (LIST_LANES - 1), sector = k >> 3;
        if (lane < (k & 7) && sector * 8 < cap) out[sector * stride + lane] = ring[((sector & 1) << 3) + lane];
        __syncwarp();
        return k;
    }
};

// The same for one lane per particle (large scenes): each thread collects its
// entries in two sectors of its own in shared memory.  flush() is called at
// least once per eight add().
struct LaneRing {
    unsigned v[16][T];
};
struct LaneWriter {
    LaneRing& ring;
    unsigned* out;
    size_t stride;
    int k, done, cap;  // entries, sectors written, capacity
    __device__ __forceinline__ LaneWriter(LaneRing& r, unsigned* list, int i, int n, int capacity)
        : ring(r), out(list + (size_t)i * 8), stride((size_t)n * 8), k(0), done(0), cap(capacity)
    {
    }
    // without a branch: an entry not taken is overwritten by the next
    __device__ __forceinline__ void add(bool take, unsigned value)
    {
        ring.v[k & 15][threadIdx.x] = value;
        k += take ? 1 : 0;
    }
    __device__ __forceinline__ void flush()
    {
        if ((k >> 3) != done) sector();
    }
    __device__ __forceinline__ void sector()
    {
        if (done * 8 < cap) {
            unsigned e[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) e[u] = ring.v[((done & 1) << 3) + u][threadIdx.x];
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out), "r"(e[0]), "r"(e[1]), "r"(e[2]),
                         "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7])
                         : "memory");
        }
        out += stride;
        ++done;
    }
    __device__ __forceinline__ int finish()
    {
        flush();
        if (k & 7) sector();  // the entries past the count are never read as partners
        return k;
    }
};

__device__ __forceinline__ float cellGap(int k, int c, float h, float cs)
{
    const float lo = (float)(k - c) * cs - h, hi = h - (float)(k - c + 1) * cs;
    return fmaxf(0.f, fmaxf(lo, hi));
}
// The cells from lo to hi (offsets from the corner of cell c), clamped to n.
__device__ __forceinline__ void cellRange(int c, float lo, float hi, float cs, int n, int& first, int& last)
{
    first = max(0, c + (int)floorf(lo / cs));
    last = min(n - 1, c + (int)floorf(hi / cs));
}

// Lists (id(m) in `to`, in sorted order) the members m = load(p) of the cells
// within `reach` of a particle (cell c, offset h) that pass test(m, y, z) (y, z:
// the particle's offset from the corner of the member's cell along those axes);
// returns their number.  The cells of one row along x are
// consecutive keys, so their members are ONE range of the sorted order; rows
// and row ends beyond the reach (the corners and edges of the box) are left
// out.  The eight lanes of the particle first take a row each and find its
// range, then read the rows' members eight at a time; the four particles of a
// warp go on together, each at its own row.  Called by whole warps.
template <class Load, class Test>
__device__ __forceinline__ int takeMembers(bool live, int4 c, float4 h, float reach, const int* __restrict__ start,
                                           const GridDev& g, ListWriter to, Load load, Test test)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int L = LIST_LANES;
    const int lane = threadIdx.x & (L - 1), groupShift = (threadIdx.x & 31) & ~(L - 1);
    const unsigned groupBits = (1u << L) - 1u;
    // widened past the slack of the candidate test (1e-4, squared) and the few
    // FP32 roundings of the cell gaps
    const float wide = reach * 1.001f + 1.e-5f * (g.cs.x + g.cs.y + g.cs.z);
    int y0, y1, z0, z1;
    cellRange(c.y, h.y - wide, h.y + wide, g.cs.y, g.gy, y0, y1);
    cellRange(c.z, h.z - wide, h.z + wide, g.cs.z, g.gz, z0, z1);
    const int ny = max(1, y1 - y0 + 1);
    const int rows = live && y0 <= y1 && z0 <= z1 ? ny * (z1 - z0 + 1) : 0;
    for (int base = 0; __any_sync(FULL, base < rows); base += L) {
        const int row = base + lane;
        int p = 0, e = 0;
        float ry = 0.f, rz = 0.f;
        if (row < rows) {
            const int dz = row / ny, z = z0 + dz, y = y0 + row - dz * ny;
            const float gy = cellGap(y, c.y, h.y, g.cs.y), gz = cellGap(z, c.z, h.z, g.cs.z);
            const float rest = wide * wide - gy * gy - gz * gz;
            if (rest >= 0.f) {
                const float rx = sqrtf(rest);
                int x0, x1;
                cellRange(c.x, h.x - rx, h.x + rx, g.cs.x, g.gx, x0, x1);
                if (x0 <= x1) {
                    const int first = (z * g.gy + y) * g.gx;
                    p = start[first + x0];
                    e = start[first + x1 + 1];
                }
            }
            ry = h.y + (float)(c.y - y) * g.cs.y;
            rz = h.z + (float)(c.z - z) * g.cs.z;
        }
        unsigned todo = (__ballot_sync(FULL, p < e) >> groupShift) & groupBits;  // the particle's rows not begun
        int q = 0, qe = 0;
        float y = 0.f, z = 0.f;
        while (true) {
            const bool next = q >= qe && todo != 0u;
            if (__any_sync(FULL, next)) {
                const int r = next ? __ffs(todo) - 1 : 0;
                const int np = __shfl_sync(FULL, p, r, L), ne = __shfl_sync(FULL, e, r, L);
                const float nyo = __shfl_sync(FULL, ry, r, L), nzo = __shfl_sync(FULL, rz, r, L);
                if (next) {
                    q = np;
                    qe = ne;
                    y = nyo;
                    z = nzo;
                    todo &= todo - 1u;
                }
            }
            if (!__any_sync(FULL, q < qe)) break;
            bool take = false;
            unsigned id = 0;
            if (q + lane < qe) {
                const auto m = load(q + lane);
                take = test(m, y, z);
                id = (unsigned)m.id;
            }
            to.add(take, id);
            q += L;
        }
    }
    return to.finish();
}

// The same by one lane: it takes row after row, and reads BATCH members ahead of
// their tests (the particles of a warp are neighbours in the sorted order, so
// their reads fall into the same few lines).
struct RowBox {
    int y, z, y0, y1, z1;  // the row taken last, and the box's bounds
    float gz2, ry, rz;     // squared gap to plane z; the particle's y and z from the row's cells' corner
};
__device__ __forceinline__ bool nextRow(RowBox& b, int4 c, float4 h, float wide, const int* __restrict__ start,
                                        const GridDev& g, int& p, int& e)
{
    while (true) {
        if (++b.y > b.y1) {
            if (++b.z > b.z1) return false;
            b.y = b.y0;
            if (b.y > b.y1) return false;
            const float gz = cellGap(b.z, c.z, h.z, g.cs.z);
            b.gz2 = gz * gz;
            b.rz = h.z + (float)(c.z - b.z) * g.cs.z;
        }
        const float gy = cellGap(b.y, c.y, h.y, g.cs.y);
        const float rest = wide * wide - gy * gy - b.gz2;
        if (rest < 0.f) continue;
        const float rx = sqrtf(rest);
        int x0, x1;
        cellRange(c.x, h.x - rx, h.x + rx, g.cs.x, g.gx, x0, x1);
        if (x0 > x1) continue;
        const int row = (b.z * g.gy + b.y) * g.gx;
        p = start[row + x0];
        e = start[row + x1 + 1];
        b.ry = h.y + (float)(c.y - b.y) * g.cs.y;
        if (p < e) return true;
    }
}
template <class Load, class Test>
__device__ __forceinline__ int takeMembers(bool live, int4 c, float4 h, float reach, const int* __restrict__ start,
                                           const GridDev& g, LaneWriter to, Load load, Test test)
{
    constexpr int BATCH = 4;
    const float wide = reach * 1.001f + 1.e-5f * (g.cs.x + g.cs.y + g.cs.z);
    RowBox b;
    int z0, p = 0, e = 0;
    cellRange(c.y, h.y - wide, h.y + wide, g.cs.y, g.gy, b.y0, b.y1);
    cellRange(c.z, h.z - wide, h.z + wide, g.cs.z, g.gz, z0, b.z1);
    b.y = b.y1;  // one advance reaches the first row
    b.z = z0 - 1;
    b.gz2 = b.ry = b.rz = 0.f;
    while (live && nextRow(b, c, h, wide, start, g, p, e)) {
        for (; p < e; p += BATCH) {
            decltype(load(0)) m[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) m[u] = load(min(p + u, e - 1));
#pragma unroll
            for (int u = 0; u < BATCH; ++u) to.add(test(m[u], b.ry, b.rz) && p + u < e, (unsigned)m[u].id);
            to.flush();
        }
    }
    return to.finish();
}

// Verlet candidates of the fluid lists, of particle i by its L lanes (1 or
// LIST_LANES; whole warps; live false past the last particle): every fluid within the
// largest cut + fskin and every solid within 2 h + fskin, in sorted order (all
// particles are inside the domain here: one outside it sends the lists back to
// the walk).  P (cellPack): a fluid partner's cell and offset are its partner
// record, one 16-byte read.
//
// What bounds it: instruction issue.  Walking the cells one by one (64 cells
// of a box, 8 members each, every lane at its own cell) took 836M warp
// instructions for 400k particles, 1017 us; over rows of cells 305M, 421 us.
template <int L, bool P, class Ring>
__device__ __forceinline__ void fluidCandidates(const DeviceState& d, Ring& ring, int i, bool live)
{
    using Writer = std::conditional_t<L == 1, LaneWriter, ListWriter>;
    const int n = d.nf;
    int4 ci = make_int4(0, 0, 0, 0);
    float4 hi = make_float4(0, 0, 0, 0);
    if (live) {
        ci = d.fcell[i];
        hi = d.fph[0][i];
    }
    const float skin = d.fskin;
    const FluidRec* __restrict__ rec = d.frec[0];
    struct Member {
        float4 h;
        int x, id;
    };
    // squared cut of a pair, widened past the rounding of the estimate below
    const auto cut2 = [&](float h) {
        const float c = 2.f * h + skin;
        return c * c * (1.f + 1.e-4f);
    };
    const float cut2U = cut2(hi.w);
    const auto within = [&](const Member& m, float dc, float y, float z, float c2) {
        const float rx = (hi.x - m.h.x) + dc * d.grid.cs.x, ry = y - m.h.y, rz = z - m.h.z;
        return rx * rx + ry * ry + rz * rz <= c2;
    };
    const int nff = takeMembers(
        live, ci, hi, 2.f * fmaxf(hi.w, d.fhmax) + skin, d.fcellStart, d.grid, Writer(ring, d.fvc, i, n, d.kvf),
        [&](int p) {
            Member m;
            m.id = p;
            if constexpr (P) {
                m.h = __ldg(&rec[p].pc);
                m.x = (int)__float_as_uint(m.h.w);
            } else {
                m.h = d.fph[0][p];
                m.x = d.fcell[p].x;
            }
            return m;
        },
        [&](const Member& m, float y, float z) {
            // a packed cell's x + 2^23 as a float: no integer conversion per member
            const float dc = P ? ((float)ci.x + 8388608.f) - __uint_as_float(0x4b000000u | ((unsigned)m.x & 2047u))
                               : (float)(ci.x - m.x);
            return within(m, dc, y, z, P ? cut2U : cut2(fmaxf(hi.w, m.h.w))) && m.id != i;
        });
    const int nfs = takeMembers(
        live, ci, hi, 2.f * hi.w + skin, d.scellStart, d.grid, Writer(ring, (unsigned*)d.fvsc, i, n, d.kvs),
        [&](int p) {
            Member m;
            m.id = d.ssorted[p];
            m.h = d.sph[m.id];
            m.x = d.scell[m.id].x;
            return m;
        },
        [&](const Member& m, float y, float z) { return within(m, (float)(ci.x - m.x), y, z, cut2U); });
    if (!live || (threadIdx.x & (L - 1)) != 0) return;
    d.fvcn[i] = nff;
    d.fvsn[i] = nfs;
    d.fvref[i] = make_float4((float)ci.x * d.grid.cs.x + hi.x, (float)ci.y * d.grid.cs.y + hi.y,
                             (float)ci.z * d.grid.cs.z + hi.z, 0.f);
    if (nff > d.kvf || nfs > d.kvs) {
        atomicOr(d.status, ST_FVERLET_OVERFLOW);
        atomicMax(&d.need[2], nff);
        atomicMax(&d.need[3], nfs);
    }
}

// The lists from the reference's 27-cell walk (every fluid step once a particle
// has left the domain, or at initialisation).
__device__ __forceinline__ void fluidWalk(const DeviceState& d, int i, bool live)
{
    constexpr int L = LIST_LANES;
    const int lane = threadIdx.x & (L - 1);
    const int groupShift = (threadIdx.x & 31) & ~(L - 1);
    const unsigned groupBits = L == 32 ? 0xffffffffu : ((1u << L) - 1u);
    const unsigned below = (1u << lane) - 1u;
    const int n = d.nf;
    int4 ci = make_int4(0, 0, 0, 0);
    float4 hi = make_float4(0, 0, 0, 0), li = hi;
    dfl hI = df_make(0.f), cutS = hI;
    int sx = 0, sy = 0, sz = 0;
    if (live) {
        ci = d.fcell[i];
        hi = d.fph[0][i];
        li = d.fpl[0][i];
        hI = df_make(hi.w, li.w);
        cutS = df_add(hI, hI);  // fluid-solid: 2 h_i
        sx = truncAxis(ci.x, hi.x, li.x);
        sy = truncAxis(ci.y, hi.y, li.y);
        sz = truncAxis(ci.z, hi.z, li.z);
    }
    // a walk position gives the partner's cell offset from the particle's own
    // cell only when the walk is centred on that cell
    const bool centred = sx == ci.x && sy == ci.y && sz == ci.z;
    // fluid partners
    int nff = 0;
    {
        LaneWalk w{lane - L, 0, 0, 0, 0, 0, 0, false};
        while (true) {
            int j = 0;
            const bool has = live && nextCandidate<L>(w, d.fcellStart, sx, sy, sz, d.grid, j);
            bool take = false;
            int4 cj = make_int4(0, 0, 0, 0);
            if (has && j != i) {
                cj = w.regular ? make_int4(w.hx, w.hy, w.hz, w.hash) : d.fcell[j];
                const float4 hj = d.fph[0][j];
                // FP32 decision away from the cut (most candidates); the exact
                // double-float test within 1e-5 of it
                const float3 r = relF(ci, hi, cj, hj, d.grid);
                const float c = 2.f * fmaxf(hi.w, hj.w);
                const float d2 = dot3(r, r), c2 = c * c;
                if (d2 < c2 * (1.f - 1.e-5f)) {
                    take = true;
                } else if (d2 <= c2 * (1.f + 1.e-5f)) {
                    const dfl hJ = df_make(hj.w, d.fpl[0][j].w);
                    const dfl rad = dfMax(hI, hJ);
                    take = withinCut(ci, hi, li, cj, hj, d.fpl[0], j, df_add(rad, rad), d.grid);
                }
            }
            const unsigned mine = (__ballot_sync(0xffffffffu, take) >> groupShift) & groupBits;
            if (take) {
                const int slot = nff + __popc(mine & below);
                if (slot < d.kff) d.ff[listAt(slot, i, n)] = ffEntry(j, w.t, w.regular && centred);
            }
            nff += __popc(mine);
            if (!__any_sync(0xffffffffu, has)) break;
        }
    }
    // solid partners
    int nfs = 0;
    {
        LaneWalk w{lane - L, 0, 0, 0, 0, 0, 0, false};
        while (true) {
            int p = 0;
            const bool has = live && nextCandidate<L>(w, d.scellStart, sx, sy, sz, d.grid, p);
            bool take = false;
            int a = 0;
            if (has) {
                a = d.ssorted[p];
                const int4 ca = w.regular ? make_int4(w.hx, w.hy, w.hz, w.hash) : d.scell[a];
                const float4 ha = d.sph[a];
                const float3 r = relF(ci, hi, ca, ha, d.grid);
                const float c = 2.f * hi.w;
                const float d2 = dot3(r, r), c2 = c * c;
                if (d2 < c2 * (1.f - 1.e-5f)) take = true;
                else if (d2 <= c2 * (1.f + 1.e-5f)) take = withinCut(ci, hi, li, ca, ha, d.spl, a, cutS, d.grid);
            }
            const unsigned mine = (__ballot_sync(0xffffffffu, take) >> groupShift) & groupBits;
            if (take) {
                const int slot = nfs + __popc(mine & below);
                if (slot < d.kfs) d.fs[listAt(slot, i, n)] = fsEntry(a, w.t);
            }
            nfs += __popc(mine);
            if (!__any_sync(0xffffffffu, has)) break;
        }
    }
    if (!live || lane != 0) return;
    d.ffc[i] = nff;
    d.fsc[i] = nfs;
    if (nff > d.kff) atomicOr(d.status, ST_FF_OVERFLOW);
    if (nfs > d.kfs) atomicOr(d.status, ST_FS_OVERFLOW);
}

// Walk position (0..26) of cell cj in the 27-cell walk centred on ci, or -1.
__device__ __forceinline__ int walkPosition(int4 ci, int4 cj)
{
    const int dx = cj.x - ci.x, dy = cj.y - ci.y, dz = cj.z - ci.z;
    if (dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1) return -1;
    return (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
}

// The lists of this fluid step from the candidates (setFluidInteractionsKernel,
// core/neighborSearch.cu:115-220, on positions the candidates cover): the
// reference's test on the current positions, for partners in the 27 cells
// around the particle's current cell (all particles are inside the domain
// here, so those are the cells the reference walks).  The rebuild flag is
// cleared: the last position update of the step raises it again.
//
// P (cellPack): a candidate's cell and offset are its partner record (one
// 16-byte read), the smoothing length is every particle's, and the test runs
// on the packed cells (packedWalk): no unpacking, no integer conversions.
//
// What bounds it: latency of the candidate stream and the records, then the
// list's bytes.  With one column per entry, every entry stored was a sector
// write of its own: of 199 us for 400k particles, 120 were those stores, 60 the
// candidate ids, 20 the records; in sectors it takes 140 us (1.0M: 350 to 316).

// Packed cells (x | y << 11 | z << 22) and their place in the 27-cell walk:
// with one added to each field (PACK_ONES), the difference of two neighbouring
// cells has fields dx + 1, dy + 1, dz + 1 in 0..2; any other difference has a
// field of 3 or bits outside the fields (a borrow sets all of them).
constexpr unsigned PACK_ONES = 1u | 1u << 11 | 1u << 22;
__device__ __forceinline__ bool packedNeighbour(unsigned diff)
{
    return ((diff & ~(3u * PACK_ONES)) | (diff & (diff >> 1) & PACK_ONES)) == 0u;
}
// (dx + 1) + 3 (dy + 1) + 9 (dz + 1): the product puts the three terms at bit
// 22, the smaller cross terms below it (they never carry) and the others past
// bit 31.
__device__ __forceinline__ unsigned packedWalk(unsigned diff) { return (diff * ((1u << 22) + (3u << 11) + 9u)) >> 22; }

#ifndef DEMSPH_FILTER_UNROLL
#define DEMSPH_FILTER_UNROLL 2  // sectors of candidates in flight
#endif

// The fluid part of the filter from the partner records; tab: the offsets of
// the 27 walk cells, one array per axis.  Returns the number of partners.
__device__ __forceinline__ int filterRecords(const DeviceState& d, const float (*tab)[32], ListWriter to, int i, int lane,
                                             int nc, int4 ci, float4 hi, float4 li)
{
    constexpr int U = DEMSPH_FILTER_UNROLL;
    const FluidRec* __restrict__ rec = d.frec[0];
    const size_t stride = (size_t)d.nf * 8;
    const unsigned* cand = d.fvc + (size_t)i * 8 + lane;
    const unsigned mine0 = __float_as_uint(packCell(ci)) - PACK_ONES;
    const float c = 2.f * hi.w, c2 = c * c, c2lo = c2 * (1.f - 1.e-5f), c2hi = c2 * (1.f + 1.e-5f);
    int jn[U];
#pragma unroll
    for (int u = 0; u < U; ++u, cand += stride) jn[u] = u * LIST_LANES + lane < nc ? (int)__ldcs(cand) : i;
    for (int k = lane; __any_sync(0xffffffffu, k - lane < nc); k += U * LIST_LANES) {
        int j[U];
        float4 r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            j[u] = jn[u];
            r[u] = __ldg(&rec[j[u]].pc);
        }
#pragma unroll
        for (int u = 0; u < U; ++u, cand += stride) jn[u] = k + (U + u) * LIST_LANES < nc ? (int)__ldcs(cand) : i;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned diff = __float_as_uint(r[u].w) - mine0;
            const unsigned t = packedWalk(diff) & 31u;  // some word of the table where it is no neighbour
            const float x = (hi.x - r[u].x) - tab[0][t], y = (hi.y - r[u].y) - tab[1][t], z = (hi.z - r[u].z) - tab[2][t];
            const float d2 = x * x + y * y + z * z;
            bool take = d2 <= c2hi && packedNeighbour(diff) && k + u * LIST_LANES < nc;
            if (take && d2 >= c2lo) {  // within the rounding of the cut: decided in double-float
                const dfl hI = df_make(hi.w, li.w);
                take = withinCut(ci, hi, li, unpackCell(r[u].w), r[u], d.fpl[0], j[u], df_add(hI, hI), d.grid);
            }
            to.add(take, ffEntry(j[u], (int)t, true));
        }
    }
    return to.finish();
}

// The same from cells and positions of their own (fluids whose parameters
// differ, grids too large for packed cells).
__device__ __forceinline__ int filterCells(const DeviceState& d, ListWriter to, int i, int lane, int nc, int4 ci, float4 hi,
                                           float4 li)
{
    const dfl hI = df_make(hi.w, li.w);
    const size_t stride = (size_t)d.nf * 8;
    const unsigned* cand = d.fvc + (size_t)i * 8 + lane;
    int jn = lane < nc ? (int)__ldcs(cand) : i;
    for (int k = lane; __any_sync(0xffffffffu, k - lane < nc); k += LIST_LANES) {
        const int j = jn;
        const int4 cj = d.fcell[j];
        const float4 hj = d.fph[0][j];
        cand += stride;
        jn = k + LIST_LANES < nc ? (int)__ldcs(cand) : i;
        const int t = walkPosition(ci, cj);
        const float3 r = relF(ci, hi, cj, hj, d.grid);
        const float c = 2.f * fmaxf(hi.w, hj.w);
        const float d2 = dot3(r, r), c2 = c * c;
        bool take = k < nc && t >= 0 && d2 <= c2 * (1.f + 1.e-5f);
        if (take && d2 >= c2 * (1.f - 1.e-5f)) {
            const dfl rad = dfMax(hI, df_make(hj.w, d.fpl[0][j].w));
            take = withinCut(ci, hi, li, cj, hj, d.fpl[0], j, df_add(rad, rad), d.grid);
        }
        to.add(take, ffEntry(j, t & 31, true));
    }
    return to.finish();
}

// The reference's test for solid a of a fluid particle; t: the walk position of
// its cell.
__device__ __forceinline__ bool solidPartnerOf(const DeviceState& d, int4 ci, float4 hi, float4 li, int a, int4 ca,
                                               float4 ha, int& t)
{
    t = walkPosition(ci, ca);
    const float3 r = relF(ci, hi, ca, ha, d.grid);
    const float d2 = dot3(r, r), c2 = 4.f * hi.w * hi.w;
    if (t < 0 || d2 > c2 * (1.f + 1.e-5f)) return false;
    if (d2 < c2 * (1.f - 1.e-5f)) return true;
    const dfl hI = df_make(hi.w, li.w);
    return withinCut(ci, hi, li, ca, ha, d.spl, a, df_add(hI, hI), d.grid);
}

// filterRecords by one lane per particle: a sector of candidates in one load,
// four records in flight.
__device__ __forceinline__ int filterRecordsLane(const DeviceState& d, const float (*tab)[32], LaneWriter to, int i, int nc,
                                                 int4 ci, float4 hi, float4 li)
{
    constexpr int B = 4;
    const FluidRec* __restrict__ rec = d.frec[0];
    const size_t stride = (size_t)d.nf * 8;
    const uint4* cand = reinterpret_cast<const uint4*>(d.fvc + (size_t)i * 8);
    const unsigned mine0 = __float_as_uint(packCell(ci)) - PACK_ONES;
    const float c = 2.f * hi.w, c2 = c * c, c2lo = c2 * (1.f - 1.e-5f), c2hi = c2 * (1.f + 1.e-5f);
    uint4 a = make_uint4(i, i, i, i);
    if (nc > 0) a = __ldcs(cand);
    for (int k = 0; k < nc; k += B) {
        const unsigned j[B] = {a.x, k + 1 < nc ? a.y : (unsigned)i, k + 2 < nc ? a.z : (unsigned)i,
                               k + 3 < nc ? a.w : (unsigned)i};
        float4 r[B];
#pragma unroll
        for (int u = 0; u < B; ++u) r[u] = __ldg(&rec[j[u]].pc);
        // candidates k + 4 .. k + 7: the sector's other half, or the next sector
        cand = (k & 4) ? reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned*>(cand) - 4 + stride) : cand + 1;
        if (k + B < nc) a = __ldcs(cand);
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const unsigned diff = __float_as_uint(r[u].w) - mine0;
            const unsigned t = packedWalk(diff) & 31u;
            const float x = (hi.x - r[u].x) - tab[0][t], y = (hi.y - r[u].y) - tab[1][t], z = (hi.z - r[u].z) - tab[2][t];
            const float d2 = x * x + y * y + z * z;
            bool take = d2 <= c2hi && packedNeighbour(diff) && k + u < nc;
            if (take && d2 >= c2lo) {
                const dfl hI = df_make(hi.w, li.w);
                take = withinCut(ci, hi, li, unpackCell(r[u].w), r[u], d.fpl[0], (int)j[u], df_add(hI, hI), d.grid);
            }
            to.add(take, ffEntry((int)j[u], (int)t, true));
        }
        to.flush();
    }
    return to.finish();
}

// One lane per particle (packed cells only).
__global__ void __launch_bounds__(T) kFluidFilterLane(DeviceState d)
{
    stepKernelBegin();
    __shared__ LaneRing ring;
    __shared__ float tab[3][32];
    if (threadIdx.x < 27) {
        tab[0][threadIdx.x] = (float)((int)(threadIdx.x % 3) - 1) * d.grid.cs.x;
        tab[1][threadIdx.x] = (float)((int)(threadIdx.x / 3 % 3) - 1) * d.grid.cs.y;
        tab[2][threadIdx.x] = (float)((int)(threadIdx.x / 9) - 1) * d.grid.cs.z;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nf || *d.status || *d.fslowMode || *d.slowMode) return;
    if (i == 0) *(volatile int*)d.frebuild = 0;
    const int n = d.nf;
    const int4 ci = d.fcell[i];
    const float4 hi = d.fph[0][i], li = d.fpl[0][i];
    const int nc = min(d.fvcn[i], d.kvf), ns = min(d.fvsn[i], d.kvs);
    const int nff = filterRecordsLane(d, tab, LaneWriter(ring, d.ff, i, n, d.kff), i, nc, ci, hi, li);
    // few particles have solid candidates, but those many (a wall): four in flight
    LaneWriter to(ring, (unsigned*)d.fs, i, n, d.kfs);
    for (int k = 0; k < ns; k += 4) {
        const int4 v = __ldcs(reinterpret_cast<const int4*>(d.fvsc + listAt(k, i, n)));
        const int a[4] = {v.x, k + 1 < ns ? v.y : v.x, k + 2 < ns ? v.z : v.x, k + 3 < ns ? v.w : v.x};
        int4 ca[4];
        float4 ha[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            ca[u] = d.scell[a[u]];
            ha[u] = d.sph[a[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            int t;
            const bool take = solidPartnerOf(d, ci, hi, li, a[u], ca[u], ha[u], t) && k + u < ns;
            to.add(take, (unsigned)fsEntry(a[u], t));
        }
        to.flush();
    }
    const int nfs = to.finish();
    d.ffc[i] = nff;
    d.fsc[i] = nfs;
    if (nff > d.kff) atomicOr(d.status, ST_FF_OVERFLOW);
    if (nfs > d.kfs) atomicOr(d.status, ST_FS_OVERFLOW);
}

// One particle by its LIST_LANES lanes.
template <bool P>
__global__ void __launch_bounds__(T) kFluidFilter(DeviceState d)
{
    stepKernelBegin();
    __shared__ ListRing ring;
    __shared__ float tab[3][32];
    if (P) {
        if (threadIdx.x < 27) {
            tab[0][threadIdx.x] = (float)((int)(threadIdx.x % 3) - 1) * d.grid.cs.x;
            tab[1][threadIdx.x] = (float)((int)(threadIdx.x / 3 % 3) - 1) * d.grid.cs.y;
            tab[2][threadIdx.x] = (float)((int)(threadIdx.x / 9) - 1) * d.grid.cs.z;
        }
        __syncthreads();
    }
    const long long th = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(th / LIST_LANES), lane = threadIdx.x & (LIST_LANES - 1);
    if ((th & ~31LL) >= (long long)d.nf * LIST_LANES || *d.status || *d.fslowMode || *d.slowMode) return;
    if (th == 0) *(volatile int*)d.frebuild = 0;
    const bool live = i < d.nf;
    const int n = d.nf, self = live ? i : 0;
    const int4 ci = d.fcell[self];
    const float4 hi = d.fph[0][self], li = d.fpl[0][self];
    const int nc = live ? min(d.fvcn[i], d.kvf) : 0, ns = live ? min(d.fvsn[i], d.kvs) : 0;
    int sn = lane < ns ? d.fvsc[listAt(lane, i, n)] : 0;  // the first solid candidate, read beside the fluids
    int nff;
    if constexpr (P) nff = filterRecords(d, tab, ListWriter(ring, d.ff, self, n, d.kff), self, lane, nc, ci, hi, li);
    else nff = filterCells(d, ListWriter(ring, d.ff, self, n, d.kff), self, lane, nc, ci, hi, li);
    ListWriter to(ring, (unsigned*)d.fs, self, n, d.kfs);
    for (int k = lane; __any_sync(0xffffffffu, k - lane < ns); k += LIST_LANES) {
        bool take = false;
        int t = 0;
        const int a = sn;
        if (k + LIST_LANES < ns) sn = d.fvsc[listAt(k + LIST_LANES, i, n)];
        if (k < ns) take = solidPartnerOf(d, ci, hi, li, a, d.scell[a], d.sph[a], t);
        to.add(take, (unsigned)fsEntry(a, t));
    }
    const int nfs = to.finish();
    if (!live || lane != 0) return;
    d.ffc[i] = nff;
    d.fsc[i] = nfs;
    if (nff > d.kff) atomicOr(d.status, ST_FF_OVERFLOW);
    if (nfs > d.kfs) atomicOr(d.status, ST_FS_OVERFLOW);
}

// ---- fluid partners of each massive solid (coupling force) ----
__global__ void kCoupCount(DeviceState d)
{
    stepKernelBegin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nf || *d.status) return;
    const int m = min(d.fsc[i], d.kfs);
    for (int k = 0; k < m; ++k) {
        const int a = fsPartner(d.fs[listAt(k, i, d.nf)]);
        if (d.sflags[a].w & F_HASMASS) atomicAdd(&d.coupCount[a], 1);
    }
}
__global__ void kCoupFill(DeviceState d)
{
    stepKernelBegin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nf || *d.status) return;
    if (d.coupStart[d.ns] > d.coupCap) {
        if (i == 0) atomicOr(d.status, ST_COUPLE_OVERFLOW);
        return;
    }
    const int m = min(d.fsc[i], d.kfs);
    for (int k = 0; k < m; ++k) {
        const int a = fsPartner(d.fs[listAt(k, i, d.nf)]);
        if (d.sflags[a].w & F_HASMASS) d.coupList[d.coupStart[a] + atomicAdd(&d.coupCount[a], 1)] = i;
    }
}
// atomics leave each solid's fluid partners in arbitrary order: sort them
__global__ void kCoupSort(DeviceState d)
{
    stepKernelBegin();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= d.ns || *d.status) return;
    const int s = d.coupStart[a], e = d.coupStart[a + 1];
    for (int p = s + 1; p < e; ++p) {
        const int v = d.coupList[p];
        int q = p - 1;
        while (q >= s && d.coupList[q] > v) {
            d.coupList[q + 1] = d.coupList[q];
            --q;
        }
        d.coupList[q + 1] = v;
    }
}

// ---- solid contact lists ----
// One row's contacts of this step (setSolid2SolidInteractionsKernel,
// core/neighborSearch.cu:222-312): the partners that pass the reference's
// test, either from the Verlet candidates or - for grids under 3 cells on an
// axis, or once a solid has left the domain - from the reference's own 27-cell
// walk.  Forward partners (B > A) and reverse partners (B < A) are kept in
// index order, whichever way they were found, so the forces - and their sums
// per solid - do not depend on the candidate margin; the reference's pair
// order (walk order) matters only to exports, which restore it.  Each forward
// pair then takes the springs of the same pair in the previous list (the exact
// history remap of the reference, from the springs the last contact phase
// left in the previous list's slots).  At initialisation (forceWalk) the list
// stays in walk order: bonds are numbered in it.
// The spring history of the forward pairs q = first, first + step, ... of row
// r from the previous list (the pair's springs there, or zeros).
__device__ __forceinline__ void remapSprings(const DeviceState& d, int par, int r, int nf, int first, int step,
                                             int fromPairs)
{
    const int prev = par ^ 1;
    const size_t nr = (size_t)d.nrow;
    if (fromPairs) {  // the springs are in the candidates' slots
        const int vf = d.pfirst[r], forward = min(d.vcnt[r], d.vcap) - vf;
        for (int q = first; q < nf; q += step) {
            const size_t slot = (size_t)q * nr + r;
            const int b = d.fwd[par][slot];
            float4 s0 = make_float4(0, 0, 0, 0), s1 = s0, s2 = s0;
            for (int k = 0; k < forward; ++k) {
                const size_t ps = (size_t)k * nr + r;
                if (d.vcand[ps + (size_t)vf * nr] != b) continue;
                if (d.pflag[ps] == PAIR_LIVE) {
                    s0 = d.pspring[0][ps];
                    if (d.pairSprings == 3) {
                        s1 = d.pspring[1][ps];
                        s2 = d.pspring[2][ps];
                    }
                }
                break;
            }
            d.springIn[0][slot] = s0;
            d.springIn[1][slot] = s1;
            d.springIn[2][slot] = s2;
        }
        return;
    }
    const int prevCnt = min(d.fcnt[prev][r], d.scap);
    for (int q = first; q < nf; q += step) {
        const size_t slot = (size_t)q * nr + r;
        const int b = d.fwd[par][slot];
        float4 s0 = make_float4(0, 0, 0, 0), s1 = s0, s2 = s0;
        for (int k = 0; k < prevCnt; ++k) {
            const size_t ps = (size_t)k * nr + r;
            if (d.fwd[prev][ps] == b) {
                s0 = d.springOut[prev][0][ps];
                s1 = d.springOut[prev][1][ps];
                s2 = d.springOut[prev][2][ps];
                break;
            }
        }
        d.springIn[0][slot] = s0;
        d.springIn[1][slot] = s1;
        d.springIn[2][slot] = s2;
    }
}

__device__ __forceinline__ void detectRow(const DeviceState& d, int par, int forceWalk, bool walk, int r, int fromPairs)
{
    // stale candidates are rebuilt first, row by row (the contact force
    // kernel clears the flag once every row has read it)
    if (!walk && d.rebuild[par]) verletBuildRow(d, r);
    const int a = solidOf(d, r);
    const int4 fa = d.sflags[a];
    const int C = d.scap;
    const size_t nr = (size_t)d.nrow;
    int nf = 0, nb = 0;
    auto emit = [&](int b) {
        if (b > a) {
            if (nf < C) d.fwd[par][(size_t)nf * nr + r] = b;
            ++nf;
        } else {
            if (nb < C) d.rev[(size_t)nb * nr + r] = b;
            ++nb;
        }
    };
    if (walk) {
        const int4 ca = d.scell[a];
        const float4 ha = d.sph[a], la = d.spl[a];
        forStencil(ca, ha, la, d.grid, [&](int hash, bool, int, int, int) {
            for (int p = d.scellStart[hash], pe = d.scellStart[hash + 1]; p < pe; ++p) {
                const int b = d.ssorted[p];
                if (solidPairCandidate(d, a, fa, b) && solidsTouch(d, a, b)) emit(b);
            }
        });
    } else {
        const int n = min(d.vcnt[r], d.vcap);
        for (int k = 0; k < n; ++k) {
            const int b = d.vcand[(size_t)k * nr + r];
            if (solidsTouch(d, a, b)) emit(b);
        }
    }
    d.fcnt[par][r] = nf;
    d.rcnt[r] = nb;
    if (nf > C || nb > C) {
        atomicOr(d.status, ST_SS_OVERFLOW);
        atomicMax(&d.need[0], max(nf, nb));
        return;
    }
    if (walk && !forceWalk) {
        sortSlots(d.fwd[par], r, d.nrow, nf);
        sortSlots(d.rev, r, d.nrow, nb);
    }
    for (int q = 0; q < nb; ++q) d.revF[(size_t)q * nr + r].w = 0.f;  // until a forward row's pair force writes it
    remapSprings(d, par, r, nf, 0, 1, fromPairs);
}


// L lanes per row (rows with many candidates): the lanes test the candidates
// in turn and a ballot keeps the lists in candidate order, exactly the lists
// of one lane per row; each lane then remaps the history of every L-th
// forward pair.  The reference's walk (at initialisation, or once a solid has
// left the domain) and stale candidates (their rebuild) run on the row's
// first lane.
template <int L>
__global__ void __launch_bounds__(T) kContactDetect(DeviceState d, int par, int forceWalk, int fromPairs)
{
    stepKernelBegin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if ((t & ~31) >= d.nrow * L || *d.status) return;  // whole warps: the ballots take every lane
    const int r = t / L, lane = t % L;
    const bool live = r < d.nrow;
    const bool walk = forceWalk || *d.slowMode;
    if (L == 1 || walk) {
        if (live && lane == 0) detectRow(d, par, forceWalk, walk, r, fromPairs);
        return;
    }
    // stale candidates are rebuilt first (the contact force kernel clears the
    // flag once every row has read it)
    if (live && lane == 0 && d.rebuild[par]) verletBuildRow(d, r);
    __syncwarp();  // the rebuilt candidates, for the row's other lanes
    const unsigned FULL = 0xffffffffu;
    const int groupShift = (threadIdx.x & 31) & ~(L - 1);
    const unsigned groupBits = (1u << L) - 1u;
    const unsigned below = (1u << lane) - 1u;
    const int C = d.scap;
    const size_t nr = (size_t)d.nrow;
    const int a = live ? solidOf(d, r) : 0;
    const int n = live ? min(d.vcnt[r], d.vcap) : 0;
    int nf = 0, nb = 0;
    for (int base = 0; __any_sync(FULL, base < n); base += L) {
        const int k = base + lane;
        int b = 0;
        bool tf = false, tb = false;
        if (k < n) {
            b = d.vcand[(size_t)k * nr + r];
            if (solidsTouch(d, a, b)) {
                tf = b > a;
                tb = !tf;
            }
        }
        const unsigned mf = (__ballot_sync(FULL, tf) >> groupShift) & groupBits;
        const unsigned mb = (__ballot_sync(FULL, tb) >> groupShift) & groupBits;
        if (tf) {
            const int q = nf + __popc(mf & below);
            if (q < C) d.fwd[par][(size_t)q * nr + r] = b;
        }
        if (tb) {
            const int q = nb + __popc(mb & below);
            if (q < C) {
                d.rev[(size_t)q * nr + r] = b;
                d.revF[(size_t)q * nr + r].w = 0.f;  // until the forward row's pair force writes it
            }
        }
        nf += __popc(mf);
        nb += __popc(mb);
    }
    __syncwarp();  // the list entries, for the lanes that remap them
    if (!live) return;
    if (lane == 0) {
        d.fcnt[par][r] = nf;
        d.rcnt[r] = nb;
    }
    if (nf > C || nb > C) {
        if (lane == 0) {
            atomicOr(d.status, ST_SS_OVERFLOW);
            atomicMax(&d.need[0], max(nf, nb));
        }
        return;
    }
    remapSprings(d, par, r, nf, lane, L, fromPairs);
}

// Contact items (forward and reverse contacts, bonds) per row over at most
// 4096 evenly spaced rows, one row per thread, summed into rowStats (zeroed by
// the caller): the host sizes the rows per warp of the contact force kernel
// from them.
constexpr int ROW_SAMPLES = 4096;
__global__ void kRowStats(DeviceState d, int par)
{
    stepKernelBegin();
    __shared__ int sums[2][8];
    const int stride = max(1, d.nrow / ROW_SAMPLES);
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) * stride;
    int items = 0, rows = 0;
    if (r < d.nrow) {
        const int a = solidOf(d, r);
        items = min(d.fcnt[par][r], d.scap) + min(d.rcnt[r], d.scap) + d.bondStart[a + 1] - d.bondStart[a];
        rows = 1;
    }
    items = __reduce_add_sync(0xffffffffu, items);
    rows = __reduce_add_sync(0xffffffffu, rows);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        sums[0][w] = items;
        sums[1][w] = rows;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        int t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += sums[threadIdx.x][k];
        atomicAdd(&d.rowStats[threadIdx.x], t);
    }
}

// ---- bonds at initialisation (addBondData, core/dataBase.cpp:270-308) ----
// Flags over (row, slot) in row-major order: rows ascend with the solid index
// and the initial list is in walk order, so the exclusive scan numbers the new
// bonds in the reference's list order.
__global__ void kBondFlags(DeviceState d, int par, int* flag)
{
    stepKernelBegin();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)d.nrow * d.scap) return;
    const int r = (int)(i / d.scap), k = (int)(i % d.scap);
    int ok = 0;
    if (k < min(d.fcnt[par][r], d.scap)) {
        const int a = solidOf(d, r), b = d.fwd[par][(size_t)k * d.nrow + r];
        const float4 ra = d.srad[a], rb = d.srad[b];
        const dfl dist = dfNorm(relDF(d.scell[a], d.sph[a], d.spl[a], d.scell[b], d.sph[b], d.spl[b], d.grid));
        // skip when r_a + r_b + 1e-10 <= |x_a - x_b|
        const dfl gap = df_sub(df_add_f(df_add(df_make(ra.x, ra.y), df_make(rb.x, rb.y)), 1.e-10f), dist);
        if (df_ge0(gap) && !(gap.hi == 0.f && gap.lo == 0.f)) {
            const int4 fa = d.sflags[a], fb = d.sflags[b];
            const int slot = tableSlot(d.tab, fa.x, fb.x);
            if (slot >= 0 && d.tab.bd[6 * slot + 1] > 1.e-10f && fa.y >= 0 && fa.y == fb.y) ok = 1;
        }
    }
    flag[i] = ok;
}
__global__ void kBondWrite(DeviceState d, int par, const int* flag, const int* pos)
{
    stepKernelBegin();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)d.nrow * d.scap || !flag[i]) return;
    const int r = (int)(i / d.scap), k = (int)(i % d.scap);
    const int b = pos[i];
    const int ii = solidOf(d, r), j = d.fwd[par][(size_t)k * d.nrow + r];
    const DF3 rr = relDF(d.scell[ii], d.sph[ii], d.spl[ii], d.scell[j], d.sph[j], d.spl[j], d.grid);
    const dfl dist = dfNorm(rr);
    const float dd = dist.hi;
    const float3 n = toF3(rr) / dd;
    const float4 ri = d.srad[ii], rj = d.srad[j];
    // contact point - x_i = -(d + r_i - r_j) / 2 * n
    const float lever = -0.5f * (dd + ri.x - rj.x);
    d.bab[b] = make_int2(ii, j);
    d.bon[b] = 1;
    d.bFnTt[b] = make_float4(0, 0, 0, 0);
    d.bFsH[b] = d.bFsL[b] = d.bTbH[b] = d.bTbL[b] = make_float4(0, 0, 0, 0);
    d.bN[b] = f4(n);
    d.bLever[b] = f4(n * lever);
}

// ---- solid normals at initialisation (setSolidNormal, core/dataBase.cpp:348-413) ----
// FP64, once per scene: inside a three-layer wall the kernel-gradient sum of
// the middle layer cancels exactly, and the reference's absolute 1e-10
// threshold then sees an FP64 residue (~1e-15: zero normal) where FP32 would
// leave ~1e-6 (a spurious unit normal).
__global__ void kSolidNormals(DeviceState d, double h)
{
    stepKernelBegin();
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= d.ns) return;
    const int4 ca = d.scell[a];
    const float4 ha = d.sph[a], la = d.spl[a];
    const int4 fa = d.sflags[a];
    const double3 pa = solidAbsPos(d, a);
    const double PI = 3.1415926535897931;
    const double sigma = 21.0 / (16.0 * PI * h * h * h);
    const double hf = h / 1.3;
    const double vFixed = hf * hf * hf;
    // FP32 pre-test: candidates clearly beyond 2h skip the FP64 arithmetic
    // (GB300's FP64 rate is a small fraction of its FP32 rate)
    const float far2 = (float)(4.0 * h * h) * (1.f + 1.e-4f);
    double tx = 0, ty = 0, tz = 0;
    forStencil(ca, ha, la, d.grid, [&](int hash, bool, int, int, int) {
        for (int p = d.scellStart[hash], pe = d.scellStart[hash + 1]; p < pe; ++p) {
            const int b = d.ssorted[p];
            const int4 fb = d.sflags[b];
            const bool fixedPair = !(fa.w & F_MASSIVE) && !(fb.w & F_MASSIVE);  // both inverse mass <= 1e-10
            const bool sameClump = fa.z >= 0 && fa.z == fb.z;
            if (!fixedPair && !sameClump) continue;
            const float3 r32 = relF(ca, ha, d.scell[b], d.sph[b], d.grid);
            if (dot3(r32, r32) > far2) continue;
            const double3 pb = solidAbsPos(d, b);
            const double rx = pa.x - pb.x, ry = pa.y - pb.y, rz = pa.z - pb.z;
            const double rr = sqrt(rx * rx + ry * ry + rz * rz);
            if (rr > 2 * h) continue;
            double vol;
            if (fixedPair) {
                vol = vFixed;
            } else {
                const double s2 = 2.0 * (double)d.srad[b].x + 2.0 * (double)d.srad[b].y;
                vol = s2 * s2 * s2;
            }
            if (rr < 1.e-10 || rr >= 2.0 * h) continue;  // gradient of W is zero
            const double q = rr / h, t = 1.0 - 0.5 * q;
            const double t3 = t * t * t;
            const double dWdq = -2.0 * t3 * (1.0 + 2.0 * q) + 2.0 * t3 * t;
            const double f = sigma * dWdq / h / rr;
            tx -= vol * f * rx;
            ty -= vol * f * ry;
            tz -= vol * f * rz;
        }
    });
    const double l = sqrt(tx * tx + ty * ty + tz * tz);
    d.snormal[a] = l > 1.e-10 ? make_float4((float)(tx / l), (float)(ty / l), (float)(tz / l), 0.f)
                              : make_float4(0, 0, 0, 0);
}

}  // namespace

// The fluid walk of a fluid step in one launch: the reference's walk (at
// initialisation, and every fluid step once a fluid or a solid has left the
// domain), else the Verlet candidates when they are stale - with the contact
// rows' positions at the rebuild (a solid moving half the fluid margin since
// then makes the candidates stale) - else nothing.
template <int L, bool P>
__global__ void __launch_bounds__(T) kFluidWalk(DeviceState d, RunIf lists, RunIf cands)
{
    stepKernelBegin();
    __shared__ std::conditional_t<L == 1, LaneRing, ListRing> ring;
    if (*d.status) return;
    const bool walk = lists.active();
    if (!walk && !cands.active()) return;
    // whole warps: a warp takes 32 / lanes particles at a time
    const int lanes = walk ? LIST_LANES : L;
    const long long stride = (long long)gridDim.x * blockDim.x, total = (long long)d.nf * lanes;
    for (long long th = (long long)blockIdx.x * blockDim.x + threadIdx.x; (th & ~31LL) < total; th += stride) {
        const int i = (int)(th / lanes);
        if (walk) fluidWalk(d, i, i < d.nf);
        else fluidCandidates<L, P>(d, ring, i, i < d.nf);
    }
    if (walk || *d.status) return;
    const auto ref = [&](int a) {
        const int4 c = d.scell[a];
        const float4 h = d.sph[a];
        d.svref[a] = make_float4((float)c.x * d.grid.cs.x + h.x, (float)c.y * d.grid.cs.y + h.y,
                                 (float)c.z * d.grid.cs.z + h.z, 0.f);
    };
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < d.nrow; r += gridDim.x * blockDim.x) ref(solidOf(d, r));
    // dummy particles given a velocity move too
    if (d.ndummy > 0)
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.nmove; k += gridDim.x * blockDim.x) {
            const int a = d.moveFirst >= 0 ? d.moveFirst + k : d.moveList[k];
            if (rowOf(d, a) < 0) ref(a);
        }
}

// One lane per particle in the list kernels of large scenes: fewer instructions
// (no ballots), but eight times fewer threads.  Filter, eight lanes against
// one: 12k particles 15 / 37 us, 48k 29 / 41, 80k 39 / 45, 120k 56 / 50, 400k
// 166 / 140, 1.0M 397 / 316; the rebuild, averaged over the steps of a flowing
// 400k dam break, 107 / 60.
#ifndef DEMSPH_LANE_LISTS
#define DEMSPH_LANE_LISTS 100000
#endif
static bool laneLists(int nf) { return nf >= DEMSPH_LANE_LISTS; }

void launchFluidWalk(const DeviceState& d, bool walk, cudaStream_t s)
{
    if (d.nf <= 0) return;
    RunIf lists;  // the reference's walk every fluid step (a fluid or a solid left the domain)
    lists.always = walk ? 1 : 0;
    lists.a = d.fslowMode;
    lists.b = d.slowMode;
    RunIf cands;  // Verlet candidates, when stale
    cands.always = 0;
    cands.a = d.frebuild;
    cands.unless = d.fslowMode;
    cands.unless2 = d.slowMode;
    // the launch is idle on most steps: no more blocks than the GPU holds at
    // once (eight per SM by registers)
    const bool one = laneLists(d.nf);
    const unsigned blocks = (unsigned)std::min(152LL * 8, ((long long)d.nf * (one ? 1 : LIST_LANES) + T - 1) / T);
    if (one) launchStep(d.cellPack ? kFluidWalk<1, true> : kFluidWalk<1, false>, blocks, T, s, d, lists, cands);
    else launchStep(d.cellPack ? kFluidWalk<LIST_LANES, true> : kFluidWalk<LIST_LANES, false>, blocks, T, s, d, lists, cands);
}

void launchFluidFilter(const DeviceState& d, cudaStream_t s)
{
    if (d.nf <= 0) return;
    if (d.cellPack && laneLists(d.nf)) launchStep(kFluidFilterLane, blocksFor(d.nf, T), T, s, d);
    else launchStep(d.cellPack ? kFluidFilter<true> : kFluidFilter<false>, blocksFor((long long)d.nf * LIST_LANES, T), T, s, d);
}

void launchCouplingLists(const DeviceState& d, cudaStream_t s)
{
    if (d.nf <= 0 || d.ns <= 0) return;
    cudaMemsetAsync(d.coupCount, 0, sizeof(int) * d.ns, s);
    launchStep(kCoupCount, blocksFor(d.nf, 256), 256, s, d);
    scanExclusive(d.coupCount, d.coupStart, d.ns, d.scanWork, s);
    cudaMemsetAsync(d.coupCount, 0, sizeof(int) * d.ns, s);
    launchStep(kCoupFill, blocksFor(d.nf, 256), 256, s, d);
    launchStep(kCoupSort, blocksFor(d.ns, 256), 256, s, d);
}

void launchContactDetect(const DeviceState& d, int par, bool forceWalk, cudaStream_t s, bool fromPairs)
{
    if (d.nrow <= 0) return;
    // rows holding many contacts and bonds (the force kernel's rows per warp
    // adapted down to 16 or fewer) have many candidates: four lanes per row
    if (d.forceRows <= 16)
        launchStep(kContactDetect<4>, blocksFor((long long)d.nrow * 4, T), T, s, d, par, forceWalk ? 1 : 0, fromPairs ? 1 : 0);
    else
        launchStep(kContactDetect<1>, blocksFor(d.nrow, T), T, s, d, par, forceWalk ? 1 : 0, fromPairs ? 1 : 0);
}

void launchRowStats(const DeviceState& d, int par, cudaStream_t s)
{
    if (d.nrow <= 0) return;
    cudaMemsetAsync(d.rowStats, 0, 2 * sizeof(int), s);
    launchStep(kRowStats, ROW_SAMPLES / 256, 256, s, d, par);
}

// Bond creation from the contact list (addBondData at initialisation,
// core/dataBase.cpp:270-308), in two launches: flags + exclusive scan give each
// new bond its index in list order; returns the bond count (synchronises).
// flag and pos hold nrow * scap + 1 ints.
int launchBondFlags(const DeviceState& d, int par, int* flag, int* pos, int* work, cudaStream_t s)
{
    const long long n = (long long)d.nrow * d.scap;
    if (n <= 0) return 0;
    launchStep(kBondFlags, (unsigned)((n + 255) / 256), 256, s, d, par, flag);
    scanExclusive(flag, pos, (int)n, work, s);
    int nb = 0;
    cudaMemcpyAsync(&nb, pos + n, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    return nb;
}

void launchBondWrite(const DeviceState& d, int par, const int* flag, const int* pos, cudaStream_t s)
{
    const long long n = (long long)d.nrow * d.scap;
    if (n <= 0 || d.nb <= 0) return;
    launchStep(kBondWrite, (unsigned)((n + 255) / 256), 256, s, d, par, flag, pos);
}

void launchSolidNormals(const DeviceState& d, double h, cudaStream_t s)
{
    if (d.ns <= 0 || !(h > 0.0)) return;
    launchStep(kSolidNormals, blocksFor(d.ns, T), T, s, d, h);
}

}  // namespace demsph
