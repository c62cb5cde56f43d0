// Cell-list rebuild of the Verlet lists by counting sort and prefix scan.
//
// Replaces PeriodicGridCellList::make / UnlimitedGridCellList::make
// (core/PeriodicGridCellList.hpp:198-351, core/UnlimitedGridCellList.hpp
// :152-255) for every system of the arena that reduce_margin flagged.  A
// planning kernel turns the flagged systems into a work list of 256-item
// chunks (participants and cells); every later kernel is a persistent grid
// that walks only those chunks, so a step in which 5 of 256 systems rebuild
// costs 5 systems' worth of work:
//   1. zero the flagged systems' cell counters,
//   2. bin their participants (one atomic increment per participant),
//   3. exclusive scan of each flagged system's cells (one block per system),
//   4. scatter participants into cell order, sort each cell by participant,
//   5. renumber: slot = position in cell order (spatially coherent slots),
//   6. build each slot's partner list from the 27 neighbouring cells (one
//      warp per slot) with the reference's membership test, evaluated in FP64
//      without contraction:
//      has_interaction (i < j of a leading participant, not excluded) and
//      |adjust_direction(r_i, r_j)|^2 < (cutoff (1 + margin))^2.
// The lists hold both directions of every pair (full lists); a pair (a, b) is
// present iff the reference's half list holds (min(a,b), max(a,b)).
#include "list_build.cuh"

namespace mjg {

namespace {

constexpr int TPB = 256;
constexpr int CHUNK = 256;          // items per work chunk
constexpr int GRID = 148 * 8;       // persistent grid: 8 blocks of 256 per SM
constexpr int SCAN_TPB = 1024;

// work counters in t.work: [0] participant chunks, [1] cell chunks, [2] flagged systems

__global__ void k_plan(Arena a, int g, TermArrays t, int force_all)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s >= a.nsys) {return;}
    GlobalParams& G = a.sys[s].g[g];
    if(!G.on) {return;}
    if(force_all) {G.rebuild = 1;}
    if(!G.rebuild) {return;}
    const int np = (G.nslot + CHUNK - 1) / CHUNK;
    const int nc = (G.ncell + CHUNK - 1) / CHUNK;
    const int bp = atomicAdd(&t.work[0], np);
    const int bc = atomicAdd(&t.work[1], nc);
    t.flagged[atomicAdd(&t.work[2], 1)] = s;
    for(int k = 0; k < np; ++k)
    {
        const int b = G.slot_off + k * CHUNK;
        t.part_chunks[bp + k] = make_int4(s, b, min(b + CHUNK, G.slot_off + G.nslot), 0);
    }
    for(int k = 0; k < nc; ++k)
    {
        const int b = G.cell_off + k * CHUNK;
        t.cell_chunks[bc + k] = make_int4(s, b, min(b + CHUNK, G.cell_off + G.ncell), 0);
    }
}

__global__ void __launch_bounds__(TPB) k_cells_zero(TermArrays t)
{
    const int n = t.work[1];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.cell_chunks[c];
        const int cell = w.y + threadIdx.x;
        if(cell < w.z) {t.cell_count[cell] = 0; t.cell_fill[cell] = 0;}
    }
}

__global__ void __launch_bounds__(TPB) k_cells_assign(Arena a, int g, TermArrays t)
{
    const int n = t.work[0];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.part_chunks[c];
        const int p = w.y + threadIdx.x;      // participant index (same range as slots)
        if(p >= w.z) {continue;}
        const GlobalParams& G = a.sys[w.x].g[g];
        const double4 r = a.pos[t.part_particle[p]];
        const int cx = cell_coord(r.x, G, 0);
        const int cy = cell_coord(r.y, G, 1);
        const int cz = cell_coord(r.z, G, 2);
        const int cell = G.cell_off + cx + G.dims[0] * (cy + G.dims[1] * cz);
        t.part_cell[p] = cell;
        atomicAdd(&t.cell_count[cell], 1);
    }
}

// exclusive scan of one flagged system's cells per block (SCAN_ITEMS cells
// per thread and pass); cell_start of the system's first cell is its first
// slot
constexpr int SCAN_ITEMS = 4;
__global__ void __launch_bounds__(SCAN_TPB) k_scan_sys(Arena a, int g, TermArrays t)
{
    const int nf = t.work[2];
    __shared__ int warp_tot[SCAN_TPB / 32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for(int f = blockIdx.x; f < nf; f += gridDim.x)
    {
        const GlobalParams& G = a.sys[t.flagged[f]].g[g];
        if(threadIdx.x == 0) {carry = G.slot_off;}
        __syncthreads();
        for(int base = 0; base < G.ncell; base += SCAN_TPB * SCAN_ITEMS)
        {
            const int first = base + threadIdx.x * SCAN_ITEMS;     // this thread's cells
            int v[SCAN_ITEMS];
            int sum = 0;
#pragma unroll
            for(int q = 0; q < SCAN_ITEMS; ++q)
            {
                v[q] = first + q < G.ncell ? t.cell_count[G.cell_off + first + q] : 0;
                sum += v[q];
            }
            int incl = sum;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if(lane >= o) {incl += y;}
            }
            if(lane == 31) {warp_tot[w] = incl;}
            __syncthreads();
            if(w == 0)
            {
                const int x = warp_tot[lane];
                int xi = x;
#pragma unroll
                for(int o = 1; o < 32; o <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, xi, o);
                    if(lane >= o) {xi += y;}
                }
                warp_tot[lane] = xi - x;
            }
            __syncthreads();
            int run = carry + warp_tot[w] + incl - sum;
#pragma unroll
            for(int q = 0; q < SCAN_ITEMS; ++q)
            {
                if(first + q < G.ncell) {t.cell_start[G.cell_off + first + q] = run;}
                run += v[q];
            }
            __syncthreads();
            if(threadIdx.x == SCAN_TPB - 1) {carry = run;}
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(TPB) k_cells_scatter(TermArrays t, int* slot_tmp)
{
    const int n = t.work[0];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.part_chunks[c];
        const int p = w.y + threadIdx.x;
        if(p >= w.z) {continue;}
        const int cell = t.part_cell[p];
        const int k = atomicAdd(&t.cell_fill[cell], 1);
        slot_tmp[t.cell_start[cell] + k] = p;
    }
}

// rank sort of each cell's members by participant index, so that the slot
// order depends only on the cell assignment.  A warp takes 32 cells: each
// lane sorts a small cell (up to SMALL members) by itself, then the warp sorts
// the larger ones together, one after the other.
constexpr int SMALL = 8;
__global__ void __launch_bounds__(TPB) k_cells_sort(TermArrays t, const int* slot_tmp)
{
    const int n = t.work[1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.cell_chunks[c];
        for(int cb = w.y + wid * 32; cb < w.z; cb += TPB)
        {
            const int cell = cb + lane;
            int b = 0, m = 0;
            if(cell < w.z) {b = t.cell_start[cell]; m = t.cell_count[cell];}
            if(m <= SMALL)
            {
                for(int e = 0; e < m; ++e)
                {
                    const int v = slot_tmp[b + e];
                    int rank = 0;
                    for(int u = 0; u < m; ++u) {rank += slot_tmp[b + u] < v ? 1 : 0;}
                    t.slot_part[b + rank] = v;
                }
            }
            unsigned big = __ballot_sync(full, m > SMALL);
            while(big)
            {
                const int src = __ffs(big) - 1;
                big &= big - 1;
                const int bb = __shfl_sync(full, b, src), mm = __shfl_sync(full, m, src);
                for(int e = lane; e < mm; e += 32)
                {
                    const int v = slot_tmp[bb + e];
                    int rank = 0;
                    for(int u = 0; u < mm; ++u) {rank += slot_tmp[bb + u] < v ? 1 : 0;}
                    t.slot_part[bb + rank] = v;
                }
            }
        }
    }
}

__global__ void __launch_bounds__(TPB) k_slots_setup(Arena a, TermArrays t)
{
    const int n = t.work[0];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.part_chunks[c];
        const int s = w.y + threadIdx.x;
        if(s >= w.z) {continue;}
        const int p = t.slot_part[s];
        const int i = t.part_particle[p];
        const double4 r = a.pos[i];
        t.slot_particle[s] = i;
        t.slot_of[i]       = s;
        t.slot_sys[s]      = w.x;
        t.slot_pd[s]       = make_double4(r.x, r.y, r.z, t.part_p0[p]);
        if(t.part_p1) {t.slot_p1[s] = t.part_p1[p];}
    }
}

// every group of LPS lanes of the grid takes the next (chunk, slot) pair, so
// that all of them have work even when only a few systems rebuild
template<int LPS>
__global__ void __launch_bounds__(TPB) k_build_list(Arena a, int g, TermArrays t)
{
    constexpr int GROUPS = TPB / LPS;              // slot groups per block
    constexpr int WG = 32 / LPS;                   // slot groups per warp
    __shared__ BuildShared<LPS, TPB> sh;
    const long long nwork = (long long)t.work[0] * CHUNK;
    const long long stride = (long long)gridDim.x * GROUPS;
    // warp-uniform loop over rounds; group (lane / LPS) of the warp takes item base + lane / LPS
    for(long long base = (long long)blockIdx.x * GROUPS + (threadIdx.x >> 5) * WG; base < nwork; base += stride)
    {
        const long long item = base + (threadIdx.x & 31) / LPS;
        bool valid = item < nwork;
        int s = 0, sys = 0;
        if(valid)
        {
            const int4 w = t.part_chunks[item / CHUNK];
            s = w.y + (int)(item % CHUNK);
            sys = w.x;
            valid = s < w.z;
        }
        build_list_group<LPS, TPB>(a, g, t, valid, sys, s, sh);
    }
}

__global__ void k_rebuild_done(Arena a, int g, TermArrays t, int forced)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s < a.nsys)
    {
        GlobalParams& G = a.sys[s].g[g];
        if(G.on && G.rebuild)
        {
            G.rebuild = 0;
            G.current_margin = __dmul_rn(G.cutoff, G.margin);   // ...GridCellList::make, last line
            if(!forced) {G.rebuilds += 1;}   // count only reduce_margin rebuilds
        }
    }
    if(s == 0) {t.work[0] = 0; t.work[1] = 0; t.work[2] = 0; *t.any_rebuild = 0;}
}

__global__ void k_scatter_param(TermArrays t, double* w)
{
    const long long p = (long long)blockIdx.x * TPB + threadIdx.x;
    if(p < t.np) {w[t.part_particle[p]] = t.part_p0[p];}
}

__global__ void __launch_bounds__(TPB) k_sum_counts(TermArrays t)
{
    unsigned long long v = 0;
    for(long long s = (long long)blockIdx.x * TPB + threadIdx.x; s < t.np; s += (long long)gridDim.x * TPB) {v += t.slot_part[s];}
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {v += __shfl_xor_sync(0xffffffffu, v, o);}
    if((threadIdx.x & 31) == 0) {atomicAdd(t.total_count, v);}
}

inline unsigned blocks(long long n, int tpb = TPB) {return (unsigned)((n + tpb - 1) / tpb);}

}  // namespace

void launch_scatter_param(const TermArrays& t, double* w, cudaStream_t s)
{
    if(!t.on || t.np == 0) {return;}
    k_scatter_param<<<blocks(t.np), TPB, 0, s>>>(t, w);
    note_launches(1);
}

void launch_sum_counts(const TermArrays& t, cudaStream_t s)
{
    k_sum_counts<<<min(blocks(t.np), (unsigned)GRID), TPB, 0, s>>>(t);
    note_launches(1);
}

void launch_rebuild(const Arena& a, int g, TermArrays& t, int force_all, cudaStream_t s)
{
    if(!t.on || t.np == 0) {return;}
    k_plan        <<<blocks(a.nsys, 128), 128, 0, s>>>(a, g, t, force_all);
    k_cells_zero  <<<GRID, TPB, 0, s>>>(t);
    k_cells_assign<<<GRID, TPB, 0, s>>>(a, g, t);
    k_scan_sys    <<<min(a.nsys, 1024), SCAN_TPB, 0, s>>>(a, g, t);
    k_cells_scatter<<<GRID, TPB, 0, s>>>(t, t.slot_particle);
    k_cells_sort  <<<GRID, TPB, 0, s>>>(t, t.slot_particle);
    k_slots_setup <<<GRID, TPB, 0, s>>>(a, t);
    if(t.build_lanes == 4)       {k_build_list<4> <<<GRID, TPB, 0, s>>>(a, g, t);}
    else if(t.build_lanes == 8)  {k_build_list<8> <<<GRID, TPB, 0, s>>>(a, g, t);}
    else if(t.build_lanes == 16) {k_build_list<16><<<GRID, TPB, 0, s>>>(a, g, t);}
    else                         {k_build_list<32><<<GRID, TPB, 0, s>>>(a, g, t);}
    k_rebuild_done<<<blocks(a.nsys, 128), 128, 0, s>>>(a, g, t, force_all);
    note_launches(9);
}

}  // namespace mjg
