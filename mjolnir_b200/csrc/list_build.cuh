// The parts of a list rebuild that work on one participant or one slot, shared
// by the rebuild's launches (cells.cu) and the multi-step kernel of small arenas (run.cu).
#pragma once
#include "kernels.cuh"

namespace mjg {

constexpr int CELL_CHUNK = 1024;     // cells per scan item

// A system's chunk sums lie where its cells do, one word per chunk: chunk k's at
// cell cell_off + k.
__device__ __forceinline__ int chunk_sum_index(const GlobalParams& G, int k) {return G.cell_off + k;}

// Bins participant p of the system: its cell and its place in the cell; counts
// the cell and the cell's chunk (one atomic per chunk and warp; the only chunk of
// a small grid is never summed up).
__device__ __forceinline__ void bin_participant(const Arena& a, const TermArrays& t, const GlobalParams& G, int p)
{
    const double4 r = a.pos[t.part_particle[p]];
    const int c = cell_coord(r.x, G, 0) + G.dims[0] * (cell_coord(r.y, G, 1) + G.dims[1] * cell_coord(r.z, G, 2));
    t.part_cell[p] = G.cell_off + c;
    t.nnb[p] = atomicAdd(&t.cell_count[G.cell_off + c], 1);    // scratch until the build writes the lengths
    if(G.ncell > CELL_CHUNK)
    {
        const int chunk = chunk_sum_index(G, c / CELL_CHUNK);
        const unsigned same = __match_any_sync(__activemask(), chunk);
        if((threadIdx.x & 31) == __ffs(same) - 1) {atomicAdd(&t.cell_sum[chunk], __popc(same));}
    }
}

// participants in cell order, in any order within a cell
__device__ __forceinline__ void scatter_participant(const TermArrays& t, int p)
{
    t.slot_part[t.cell_start[t.part_cell[p]] + t.nnb[p]] = p;
}

// Participant p's slot, its rank by participant index within its cell (so that
// the slot order depends only on the cell assignment), and the slot's entries.
// A thread per participant ranks against the whole cell: a cell of m members
// costs each m loads in parallel, where sorting a cell by one lane or warp made
// one long chain of it (cells of 45 members: 187 us, now 6).
__device__ __forceinline__ void place_participant(const Arena& a, const TermArrays& t, int sys, int p)
{
    const int c = t.part_cell[p];
    const int i = t.part_particle[p];
    const int b = t.cell_start[c], m = t.cell_count[c];
    const double4 r = a.pos[i];
    int slot = b;
    for(int u = 0; u < m; ++u) {slot += t.slot_part[b + u] < p ? 1 : 0;}
    t.slot_particle[slot] = i;
    t.slot_of[i]          = slot;
    t.slot_sys[slot]      = sys;
    t.slot_pd[slot]       = make_double4(r.x, r.y, r.z, t.part_p0[p]);
    if(t.part_p1) {t.slot_p1[slot] = t.part_p1[p];}
}

// A slot's exclusion row staged in shared memory once per slot: the CSR row of
// particle i holds every particle excluded together with i (the relation is
// symmetric: topology distance and molecule rules; i itself included), so
// is_excluded(min(i, j), max(i, j)) is "j is in i's row" -- a comparison
// against the staged row instead of a chain of dependent loads per candidate.
// Rows longer than EXMAX are scanned in global memory as before.
constexpr int EXMAX = 16;
struct ExRow {
    int n;              // entries staged, or -1: the row is longer than EXMAX
    int mol;            // molecule of particle i
    int v[EXMAX];       // sorted excluded partners of i
};
// lanes [0, nl) of the slot's group stage particle i's row (every lane of the
// group must call it, then synchronise the group before reading the row)
__device__ __forceinline__ void stage_ex_row(const Arena& a, int g, int i, int gl, int nl, ExRow& r)
{
    const long long b = a.ex_start[g][i], e = a.ex_start[g][i + 1];
    const int n = (int)(e - b);
    if(gl == 0) {r.n = n <= EXMAX ? n : -1; r.mol = a.mol[i];}
    if(n <= EXMAX) {for(int k = gl; k < n; k += nl) {r.v[k] = a.ex_idx[g][b + k];}}
}
__device__ __forceinline__ bool is_excluded(const Arena& a, int g, int ignore_mol, int i, int j);
// is_excluded(min(i, j), max(i, j)) for the slot's particle i and candidate j
__device__ __forceinline__ bool excluded_staged(const Arena& a, int g, int ignore_mol, const ExRow& r, int i, int j)
{
    if(ignore_mol != IGN_NOTHING)
    {
        const int mj = a.mol[j];
        if(ignore_mol == IGN_SELF   && r.mol == mj) {return true;}
        if(ignore_mol == IGN_OTHERS && r.mol != mj) {return true;}
    }
    if(r.n < 0) {return is_excluded(a, g, IGN_NOTHING, i < j ? i : j, i < j ? j : i);}
    for(int k = 0; k < r.n; ++k)
    {
        const int x = r.v[k];
        if(x > j) {break;}
        if(x == j) {return true;}
    }
    return false;
}

__device__ __forceinline__ bool is_excluded(const Arena& a, int g, int ignore_mol, int i, int j)
{
    if(ignore_mol == IGN_SELF   && a.mol[i] == a.mol[j]) {return true;}
    if(ignore_mol == IGN_OTHERS && a.mol[i] != a.mol[j]) {return true;}
    const long long b = a.ex_start[g][i], e = a.ex_start[g][i + 1];
    for(long long q = b; q < e; ++q)
    {
        const int x = a.ex_idx[g][q];
        if(x > j) {break;}
        if(x == j) {return true;}
    }
    return false;
}

// Half lists keep a pair in the list of its lower slot only: a stencil cell's
// slot range [start, start + count) is cut to the slots above s (slots are in
// cell order, so a cell is one range), which leaves the full list's words
// above s in their order.  The full lists are symmetric (the distance test,
// the leading-participant rule and the exclusions do not depend on which
// partner asks), so every pair of them is in exactly one half list.
__device__ __forceinline__ void clip_half(int& start, int& count, int s)
{
    const int lo = max(start, s + 1);
    count = max(0, start + count - lo);
    start = lo;
}

// The list of slot s by LPS lanes (4, 8, 16 or 32; a warp builds 32 / LPS
// lists at once, so that short candidate sequences do not leave most of a warp
// idle while it waits on memory).  The 27 stencil cells, in the reference's
// order z, y, x from -1 to +1, are nine rows of three cells along x, and cells
// are in slot order along x: a row is one range of slots, or two where it
// wraps.  The at most 18 ranges, with their exclusive prefix, go through shared
// memory; candidate k of the flattened sequence belongs to the last range that
// starts at or before k, and as k only grows a lane walks forward from its
// previous range.  The next candidate's coordinates and particle are requested
// before the current one is tested.  The distance test reads the cell-ordered slot
// coordinates (consecutive candidates are consecutive in memory), the topology
// checks run only inside the list radius, and an ordered compaction within the
// group keeps the output order of a serial walk at every LPS.
constexpr int NRANGE = 18;
template<int LPS, int THREADS>
struct BuildShared {
    int start[THREADS / LPS][NRANGE];
    int excl[THREADS / LPS][NRANGE + 1];           // exclusive prefix; [NRANGE] = total
    ExRow ex_rows[THREADS / LPS];
};

// every lane of the warp must call it; valid: the group has a slot
template<int LPS, int THREADS>
__device__ __forceinline__ void build_list_group(const Arena& a, int g, const TermArrays& t, bool valid, int sys, int s,
                                                 BuildShared<LPS, THREADS>& sh)
{
    constexpr int CPL = (NRANGE + LPS - 1) / LPS;  // ranges per lane
    const int lane = threadIdx.x & 31;
    const int grp = threadIdx.x / LPS, gl = threadIdx.x % LPS;
    const unsigned full = 0xffffffffu;
    const unsigned gmask = ((LPS == 32) ? full : ((1u << LPS) - 1u)) << (lane - gl);
    int* const start = sh.start[grp];
    int* const excl = sh.excl[grp];
    ExRow& exr = sh.ex_rows[grp];
    const int cap = t.cap;
    const long long np = t.np;
    const int lt = __ffs(t.tpp) - 1;               // tpp is a power of two
    const SysDev& S = a.sys[sys];
    const GlobalParams& G = S.g[g];
    const bool periodic = S.boundary == B_PERIODIC;
    const double rl2 = G.rl2;
    const int halfw_hi = S.halfw_hi;
    const int last = G.last;                       // leads no list
    const int longest = *t.max_count;
    int i = 0;
    double4 ri = make_double4(0.0, 0.0, 0.0, 0.0);
    if(valid)
    {
        i = t.slot_particle[s];
        ri = t.slot_pd[s];
        stage_ex_row(a, g, i, gl, LPS, exr);
    }
    // the slot's cell, one axis per lane
    const int axis = gl < 3 ? gl : 0;
    const int cc = valid ? cell_coord(axis == 0 ? ri.x : (axis == 1 ? ri.y : ri.z), G, axis) : 0;
    const int cx = __shfl_sync(full, cc, 0, LPS), cy = __shfl_sync(full, cc, 1, LPS), cz = __shfl_sync(full, cc, 2, LPS);
    if(valid)
    {
        const int nx = G.dims[0], ny = G.dims[1], nz = G.dims[2];
        const bool wrap = periodic || G.hashed;
        for(int j = gl; j < 9; j += LPS)
        {
            int y = cy + j % 3 - 1, z = cz + j / 3 - 1;
            bool inside = true;
            if(wrap)
            {
                y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
                z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
            }
            else if(y < 0 || z < 0 || y >= ny || z >= nz) {inside = false;}
            int s0 = 0, c0 = 0, s1 = 0, c1 = 0;
            if(inside)
            {
                const int row = G.cell_off + nx * (y + ny * z);
                int lo = cx - 1, hi = cx + 1;                  // the first range; the wrapped rest is the second
                int lo1 = 0, hi1 = -1;
                if(wrap && lo < 0)        {lo = hi = nx - 1; hi1 = cx + 1;}
                else if(wrap && hi >= nx) {hi = nx - 1; hi1 = 0;}
                lo = max(lo, 0);
                hi = min(hi, nx - 1);
                s0 = t.cell_start[row + lo];
                c0 = t.cell_start[row + hi] + t.cell_count[row + hi] - s0;
                if(hi1 >= lo1)
                {
                    s1 = t.cell_start[row + lo1];
                    c1 = t.cell_start[row + hi1] + t.cell_count[row + hi1] - s1;
                }
                if(t.half) {clip_half(s0, c0, s); clip_half(s1, c1, s);}
            }
            start[2 * j] = s0;
            start[2 * j + 1] = s1;
            excl[2 * j] = c0;
            excl[2 * j + 1] = c1;
        }
    }
    __syncwarp();
    // exclusive prefix of the counts: within each lane's block, then across
    // the group's lanes with shuffles
    {
        int cnt[CPL];
        int sum = 0;
#pragma unroll
        for(int j = 0; j < CPL; ++j)
        {
            const int k = gl * CPL + j;
            cnt[j] = (valid && k < NRANGE) ? excl[k] : 0;
            sum += cnt[j];
        }
        int incl = sum;
#pragma unroll
        for(int o = 1; o < LPS; o <<= 1)
        {
            const int y = __shfl_up_sync(full, incl, o, LPS);
            if(gl >= o) {incl += y;}
        }
        int run = incl - sum;
#pragma unroll
        for(int j = 0; j < CPL; ++j)
        {
            const int k = gl * CPL + j;
            if(valid && k < NRANGE) {excl[k] = run;}
            run += cnt[j];
        }
        if(valid && gl == LPS - 1) {excl[NRANGE] = incl;}
    }
    __syncwarp();
    const int total = valid ? excl[NRANGE] : 0;
    int tmax = total;
#pragma unroll
    for(int o = LPS; o < 32; o <<= 1) {tmax = max(tmax, __shfl_xor_sync(full, tmax, o));}
    int count = 0;
    int at = 0;             // this lane's range
    auto candidate = [&](int k) {
        if(k >= total) {return s;}                 // none: the slot itself, which the test drops
        while(at < NRANGE - 1 && excl[at + 1] <= k) {++at;}
        return start[at] + (k - excl[at]);
    };
    int q = candidate(gl);
    double4 rj = t.slot_pd[q];
    int j = t.slot_particle[q];
    for(int b = 0; b < tmax; b += LPS)
    {
        const int qn = candidate(b + LPS + gl);
        const double4 rn = t.slot_pd[qn];
        const int jn = t.slot_particle[qn];
        bool keep = false;
        if(q != s)
        {
            double ddx = __dsub_rn(rj.x, ri.x);
            double ddy = __dsub_rn(rj.y, ri.y);
            double ddz = __dsub_rn(rj.z, ri.z);
            if(image_needed(ddx, ddy, ddz, halfw_hi))
            {
                ddx = min_image(ddx, S.halfw[0], S.width[0]);
                ddy = min_image(ddy, S.halfw[1], S.width[1]);
                ddz = min_image(ddz, S.halfw[2], S.width[2]);
            }
            const double l2 = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
            if(l2 < rl2)
            {
                keep = min(i, j) != last && !excluded_staged(a, g, G.ignore_mol, exr, i, j);
            }
        }
        const unsigned m = __ballot_sync(full, keep) & gmask;
        if(keep)
        {
            const int k = count + __popc(m & ((1u << lane) - 1u));
            // nbr_pos with the power of two as a shift
            if(k < cap) {t.nbr[t.slot_major ? (long long)s * t.words + k : ((((long long)(k >> lt) * np + s) << lt) + (k & (t.tpp - 1)))] = q;}
        }
        count += __popc(m);
        q = qn;
        rj = rn;
        j = jn;
    }
    if(valid && gl == 0)
    {
        t.nnb[s] = count < cap ? count : cap;
        t.slot_part[s] = count;                    // uncut, for the mean length (scratch until the next rebuild)
        // one word for the whole term: only a list longer than any before it
        // goes to the atomic (every slot there took turns at one address)
        if(count > longest) {atomicMax(t.max_count, count);}
        if(count > cap) {atomicOr(&a.sys[sys].status, ST_LIST_OVERFLOW);}
    }
    __syncwarp();
}

}  // namespace mjg
