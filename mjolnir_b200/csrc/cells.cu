// Cell-list rebuild of the Verlet lists by counting sort and prefix scan.
//
// Replaces PeriodicGridCellList::make / UnlimitedGridCellList::make
// (core/PeriodicGridCellList.hpp:198-351, core/UnlimitedGridCellList.hpp
// :152-255) for every system of the arena that reduce_margin flagged.  A
// planning kernel turns the flagged systems into a work list of chunks
// (participants and cells); every later kernel is a persistent grid that walks
// only those chunks, so a step in which 5 of 256 systems rebuild costs 5
// systems' worth of work:
//   1. bin the flagged systems' participants (one atomic increment per
//      participant, which gives its place within its cell),
//   2. exclusive scan of the cells, chunk by chunk (each chunk adds up the sums
//      of its system's earlier chunks, which the binning counted),
//   3. scatter participants into cell order,
//   4. renumber: slot = first slot of the cell + rank by participant index in
//      the cell (spatially coherent slots that depend on the cells alone),
//   5. build each slot's partner list from the 27 neighbouring cells with the
//      reference's membership test, evaluated in FP64 without contraction:
//      has_interaction (i < j of a leading participant, not excluded) and
//      |adjust_direction(r_i, r_j)|^2 < (cutoff (1 + margin))^2,
//   6. clear the counters for the next rebuild.
// The lists hold both directions of every pair (full lists); a pair (a, b) is
// present iff the reference's half list holds (min(a,b), max(a,b)).
// The cell counters and chunk sums are zero between rebuilds.
//
// The launches before the build are bounded by latency, a few microseconds
// each: what helps is fewer of them and no serial chain in any.
#include "list_build.cuh"

namespace mjg {

namespace {

constexpr int TPB = 256;
constexpr int CHUNK = 256;          // items per work chunk
constexpr int GRID = 148 * 8;       // persistent grid: 8 blocks of 256 per SM
constexpr int CLEAR_GRID = 148;     // the clearing launch: its last block finishes the rebuild

// work counters in t.work: [0] participant chunks, [1] cell chunks, [2] blocks of the last launch done

// one block per system
__global__ void __launch_bounds__(128) k_plan(Arena a, int g, TermArrays t, int force_all)
{
    const int s = blockIdx.x;
    GlobalParams& G = a.sys[s].g[g];
    if(!G.on || !(force_all || G.rebuild)) {return;}
    const int np = (G.nslot + CHUNK - 1) / CHUNK;
    const int nc = (G.ncell + CELL_CHUNK - 1) / CELL_CHUNK;
    __shared__ int base[2];
    if(threadIdx.x == 0)
    {
        G.rebuild = 1;
        base[0] = atomicAdd(&t.work[0], np);
        base[1] = atomicAdd(&t.work[1], nc);
    }
    __syncthreads();
    for(int k = threadIdx.x; k < np; k += 128)
    {
        const int b = G.slot_off + k * CHUNK;
        t.part_chunks[base[0] + k] = make_int4(s, b, min(b + CHUNK, G.slot_off + G.nslot), 0);
    }
    for(int k = threadIdx.x; k < nc; k += 128)
    {
        const int b = G.cell_off + k * CELL_CHUNK;
        t.cell_chunks[base[1] + k] = make_int4(s, b, min(b + CELL_CHUNK, G.cell_off + G.ncell), k);
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
        bin_participant(a, t, a.sys[w.x].g[g], p);
    }
}

// cell_start of one chunk of cells per block and pass, SCAN_ITEMS cells per thread
constexpr int SCAN_ITEMS = CELL_CHUNK / TPB;
__global__ void __launch_bounds__(TPB) k_scan_cells(Arena a, int g, TermArrays t)
{
    const int n = t.work[1];
    __shared__ int warp_tot[TPB / 32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 ch = t.cell_chunks[c];
        const GlobalParams& G = a.sys[ch.x].g[g];
        int before = 0;
        for(int k = threadIdx.x; k < ch.w; k += TPB) {before += t.cell_sum[chunk_sum_index(G, k)];}
        before = __reduce_add_sync(0xffffffffu, before);
        const int first = ch.y + threadIdx.x * SCAN_ITEMS;     // this thread's cells
        int v[SCAN_ITEMS];
        int sum = 0;
#pragma unroll
        for(int q = 0; q < SCAN_ITEMS; ++q)
        {
            v[q] = first + q < ch.z ? t.cell_count[first + q] : 0;
            sum += v[q];
        }
        int incl = sum;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if(lane >= o) {incl += y;}
        }
        if(threadIdx.x == 0) {carry = G.slot_off;}
        if(lane == 31) {warp_tot[w] = incl;}
        __syncthreads();
        if(lane == 0 && before) {atomicAdd(&carry, before);}
        __syncthreads();
        int run = carry + incl - sum;
        for(int k = 0; k < w; ++k) {run += warp_tot[k];}
#pragma unroll
        for(int q = 0; q < SCAN_ITEMS; ++q)
        {
            if(first + q < ch.z) {t.cell_start[first + q] = run;}
            run += v[q];
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(TPB) k_cells_scatter(TermArrays t)
{
    const int n = t.work[0];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.part_chunks[c];
        const int p = w.y + threadIdx.x;
        if(p < w.z) {scatter_participant(t, p);}
    }
}

__global__ void __launch_bounds__(TPB) k_slots_place(Arena a, TermArrays t)
{
    const int n = t.work[0];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 w = t.part_chunks[c];
        const int p = w.y + threadIdx.x;
        if(p < w.z) {place_participant(a, t, w.x, p);}
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

// clears the rebuilt systems' cell counters and chunk sums, then (the last
// block to finish) their flags and the work lists
__global__ void __launch_bounds__(TPB) k_rebuild_done(Arena a, int g, TermArrays t, int forced)
{
    const int n = t.work[1];
    for(int c = blockIdx.x; c < n; c += gridDim.x)
    {
        const int4 ch = t.cell_chunks[c];
        for(int cell = ch.y + threadIdx.x; cell < ch.z; cell += TPB) {t.cell_count[cell] = 0;}
        if(threadIdx.x == 0) {t.cell_sum[chunk_sum_index(a.sys[ch.x].g[g], ch.w)] = 0;}
    }
    __shared__ bool last;
    __syncthreads();
    if(threadIdx.x == 0) {last = atomicAdd(&t.work[2], 1) == (int)gridDim.x - 1;}
    __syncthreads();
    if(!last) {return;}
    for(int s = threadIdx.x; s < a.nsys; s += TPB)
    {
        GlobalParams& G = a.sys[s].g[g];
        if(G.on && G.rebuild)
        {
            G.rebuild = 0;
            G.current_margin = __dmul_rn(G.cutoff, G.margin);   // ...GridCellList::make, last line
            if(!forced) {G.rebuilds += 1;}   // count only reduce_margin rebuilds
        }
    }
    if(threadIdx.x < 3) {t.work[threadIdx.x] = 0;}
    if(threadIdx.x == 0) {*t.any_rebuild = 0;}
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
    k_plan         <<<a.nsys, 128, 0, s>>>(a, g, t, force_all);
    k_cells_assign <<<GRID, TPB, 0, s>>>(a, g, t);
    k_scan_cells   <<<GRID, TPB, 0, s>>>(a, g, t);
    k_cells_scatter<<<GRID, TPB, 0, s>>>(t);
    k_slots_place  <<<GRID, TPB, 0, s>>>(a, t);
    if(t.build_lanes == 4)       {k_build_list<4> <<<GRID, TPB, 0, s>>>(a, g, t);}
    else if(t.build_lanes == 8)  {k_build_list<8> <<<GRID, TPB, 0, s>>>(a, g, t);}
    else if(t.build_lanes == 16) {k_build_list<16><<<GRID, TPB, 0, s>>>(a, g, t);}
    else                         {k_build_list<32><<<GRID, TPB, 0, s>>>(a, g, t);}
    k_rebuild_done <<<CLEAR_GRID, TPB, 0, s>>>(a, g, t, force_all);
    note_launches(7);
}

}  // namespace mjg
