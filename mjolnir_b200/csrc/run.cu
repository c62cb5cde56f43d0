// Many MD steps in one launch, for arenas small enough that a step's launches
// and the gaps between them, not its work, set its time.
//
// One resident grid (one block of 1,024 threads per SM at most, launched
// cooperatively) walks the step's phases itself -- integrator pass, margin
// bookkeeping, list rebuilds of the systems that need them, forces -- with a
// barrier between phases, so a step without a rebuild costs two barriers
// instead of a chain of dependent graph nodes.  (The arenas it takes: run_fits in
// context.cu.)  What bounds it is the latency
// of each phase's chain of dependent loads plus the barriers (about a
// microsecond each over the whole GPU, less within one cluster), so the work
// of a phase is spread warp by warp over every SM: consecutive warp items go
// to different blocks.  The arithmetic is that of the step's launches
// (advance_particle, PairEval, the bonded formulas, the list builds), so in
// the mixed form, whose force sums are exact, a chunk gives the same bits
// either way.  The FP64 form adds a particle's terms in the launches' order
// (run_force).
//
// Measured (graph of launches / this kernel, us per step, calls of 50 to 100
// steps): 200-bead chain 23 / 8.6, 4,096-particle Lennard-Jones fluid 33 / 16.7
// mixed and 32 / 16.0 FP64, 2,997-bead G-JF melt 26 / 10.9, 10,000-bead melt FP64
// 30 / 14.6.  Of the Lennard-Jones fluid's 16.7 the integrator pass takes 1.8, its
// barrier 1.6, the margins 0.7, the forces 5.4, the second barrier with the noise
// drawn meanwhile 2.3, and a twelfth of a rebuild 3.5.
//
// Every load here is a plain one: lists, slot coordinates and cells are
// rewritten during the launch, which the read-only path must not see.
#include "integrate.cuh"
#include "list_build.cuh"
#include "local_terms.cuh"
#include "pair_eval.cuh"

#include <algorithm>

namespace mjg {

namespace {

constexpr int RT = 1024;                 // threads per block
constexpr int RUN_BATCH = 2;             // partners a thread requests together
static_assert(CELL_CHUNK == RT, "one cell per thread of a scan item");

using ull = unsigned long long;

// ------------------------------------------------------------------ barrier
// All blocks of the grid.  A launch that fits one cluster uses the cluster's
// hardware barrier.  Otherwise a word counts the launch's arrivals: barrier e (from
// 1) is complete when it has reached e times the number of blocks.  A second word
// counts the blocks that have left the last barrier, and the last of them sets
// both back to zero for the next launch.  The wait is bounded in time
// (RunArgs::wait_cycles): a block that gives up raises ST_BARRIER, every block
// returns at its next barrier, and the chunk's later launches return at once, since
// the words have stopped half-way.  The host then clears what the steps left
// behind (run_steps, context.cu).

// The last warp's first lane arrives and polls: the first warps hold the
// particles (Grid::warp), whose noise is drawn meanwhile.
constexpr int POLLER = RT - 32;
struct Barrier {
    const RunArgs& r;
    unsigned due;                            // arrivals that complete the current barrier
    __device__ __forceinline__ void arrive()
    {
        if(r.cluster)
        {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            return;
        }
        __syncthreads();
        if(threadIdx.x == POLLER)
        {
            due += gridDim.x;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(r.barrier) : "memory");
        }
    }
    __device__ __forceinline__ bool wait()
    {
        if(r.cluster)
        {
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            return true;
        }
        int ok = 1;
        if(threadIdx.x == POLLER)
        {
            const long long t0 = clock64();
            for(;;)
            {
                unsigned arrived;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(arrived) : "l"(r.barrier) : "memory");
                if(arrived >= due) {break;}
                if(clock64() - t0 > r.wait_cycles) {atomicOr(&r.a.sys[0].status, ST_BARRIER); ok = 0; break;}
            }
        }
        return __syncthreads_and(ok) != 0;
    }
    __device__ __forceinline__ bool sync() {arrive(); return wait();}
    // after the launch's last barrier
    __device__ __forceinline__ void leave()
    {
        if(r.cluster || threadIdx.x != POLLER) {return;}
        if(atomicAdd(r.barrier + RUN_LEFT, 1u) == gridDim.x - 1)
        {
            r.barrier[0] = 0;
            r.barrier[RUN_LEFT] = 0;
        }
    }
};

// ------------------------------------------------- bonded forces, one by one
// Each term adds its forces to the particles directly: in a small arena the
// block-wide window of the bonded launch would only lengthen the chain.
struct InLine {static constexpr bool DEFER = false;};
template<int PREC>
struct DirectAdd : InLine {
    __device__ __forceinline__ void add(void* force, int i, double fx, double fy, double fz)
    {
        Window<PREC>::global_add(force, i, fx, fy, fz);
    }
    __device__ __forceinline__ void add_fx(void* force, int i, long long x, long long y, long long z)
    {
        Window<PREC>::global_add_fx(force, i, x, y, z);
    }
};

// A pair term's force on particle i.  The mixed form adds integers, exact in any
// order.  The plain form keeps each global term's forces apart and whoever reads
// the particle's force adds them in the order of a step's launches (run_force):
// FP64 sums by atomics would land in any order, and a run would not repeat.
__device__ __forceinline__ void put_force(const Arena& a, double4*, long long i, const Acc<P_MIXED>& acc) {acc.store(a.force, i);}
__device__ __forceinline__ void put_force(const Arena&, double4* pair_force, long long i, const Acc<P_FP64>& acc)
{
    pair_force[i] = make_double4(acc.x, acc.y, acc.z, 0.0);
}

// Particle i's force after a step of this launch: in the plain form the bonded
// terms' sum, then ExcludedVolume, DebyeHuckel and Lennard-Jones (zero where the
// particle has no slot), all requested together.  whole: the force array holds
// the whole force, as between launches.
template<int PREC>
__device__ __forceinline__ void run_force(const RunArgs& r, bool whole, long long i, double& fx, double& fy, double& fz)
{
    load_force<PREC>(r.a.force, i, fx, fy, fz);
    if constexpr(PREC == P_FP64)
    {
        double4 t[NGLOBAL];
#pragma unroll
        for(int g = 0; g < NGLOBAL; ++g) {t[g] = load_pd(r.pair_force + g * r.a.n + i);}
#pragma unroll
        for(int g = 0; g < NGLOBAL; ++g)
        {
            fx += whole ? 0.0 : t[g].x; fy += whole ? 0.0 : t[g].y; fz += whole ? 0.0 : t[g].z;
        }
    }
}

// ------------------------------------------------------------------ rebuild

// The launch works on its own copy of the system records in shared memory
// (dynamic; the arena's pointer is replaced by it), read by every phase without
// a trip to L2; the remaining skins are kept there by every block for itself.
struct Shared {
    int rebuilds[RUN_MAX_SYSTEMS][NGLOBAL];
    ull flag[NGLOBAL];                           // systems to rebuild, a bit each
    int scan[32];
    int carry;
    union {
        BuildShared<8, RT> narrow;
        BuildShared<32, RT> wide;
    };
};

// element k of the concatenation of the flagged systems' ranges (n(s)
// elements each): the system and the index in its range
template<class N>
__device__ __forceinline__ bool locate(ull mask, int& k, int& s, N&& n)
{
    for(; mask; mask &= mask - 1)
    {
        s = __ffsll((long long)mask) - 1;
        const int c = n(s);
        if(k < c) {return true;}
        k -= c;
    }
    return false;
}

struct Grid {
    int nwarp, warp;             // warps of the grid; this warp, consecutive warps on different SMs
    int nthread, thread;
    __device__ Grid()
    {
        nwarp = gridDim.x * (RT / 32);
        warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
        nthread = nwarp * 32;
        thread = warp * 32 + (threadIdx.x & 31);
    }
};

template<int LPS>
__device__ __forceinline__ void build(const Arena& a, int g, const TermArrays& t, ull mask, const Grid& G,
                                      BuildShared<LPS, RT>& sh)
{
    constexpr int WG = 32 / LPS;             // slots per warp
    auto nslot = [&](int s) {return a.sys[s].g[g].nslot;};
    int s = 0;
    for(int base = G.warp * WG;; base += G.nwarp * WG)
    {
        int k = base;
        if(!locate(mask, k, s, nslot)) {break;}
        k = base + (threadIdx.x & 31) / LPS;
        const bool valid = locate(mask, k, s, nslot);
        build_list_group<LPS, RT>(a, g, t, valid, s, valid ? a.sys[s].g[g].slot_off + k : 0, sh);
    }
}

// The lists of the flagged systems of term g at the current positions.  The
// cell counters and chunk sums are zero on entry (cells.cu); the force phase that
// follows each rebuild clears them.
template<int g>
__device__ __forceinline__ bool rebuild(const Arena& a, const TermArrays& t, ull mask, const Grid& G, Shared& sh,
                                        Barrier& bar)
{
    auto nslot = [&](int s) {return a.sys[s].g[g].nslot;};
    int k, s = 0;
    // bin the participants; each takes its place within its cell
    for(int e = G.thread;; e += G.nthread)
    {
        k = e;
        if(!locate(mask, k, s, nslot)) {break;}
        const GlobalParams& P = a.sys[s].g[g];
        bin_participant(a, t, P, P.slot_off + k);
    }
    if(!bar.sync()) {return false;}
    // first slot of each cell: one block per chunk of cells; the sums of the
    // system's earlier chunks are added up by the block that needs them
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for(int e = blockIdx.x;; e += gridDim.x)
    {
        k = e;
        if(!locate(mask, k, s, [&](int x) {return (a.sys[x].g[g].ncell + CELL_CHUNK - 1) / CELL_CHUNK;})) {break;}
        const GlobalParams& q = a.sys[s].g[g];
        int before = 0;
        for(int c = threadIdx.x; c < k; c += RT) {before += t.cell_sum[chunk_sum_index(q, c)];}
        before = __reduce_add_sync(0xffffffffu, before);
        const int cell = k * CELL_CHUNK + threadIdx.x;
        const int v = cell < q.ncell ? t.cell_count[q.cell_off + cell] : 0;
        int incl = v;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if(lane >= o) {incl += y;}
        }
        if(threadIdx.x == 0) {sh.carry = q.slot_off;}
        __syncthreads();
        if(lane == 31) {sh.scan[w] = incl;}
        if(lane == 0 && before) {atomicAdd(&sh.carry, before);}
        __syncthreads();
        if(w == 0)
        {
            const int x = sh.scan[lane];
            int xi = x;
#pragma unroll
            for(int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, xi, o);
                if(lane >= o) {xi += y;}
            }
            sh.scan[lane] = xi - x;
        }
        __syncthreads();
        if(cell < q.ncell) {t.cell_start[q.cell_off + cell] = sh.carry + sh.scan[w] + incl - v;}
        __syncthreads();
    }
    if(!bar.sync()) {return false;}
    // participants in cell order (any order within a cell)
    for(int e = G.thread;; e += G.nthread)
    {
        k = e;
        if(!locate(mask, k, s, nslot)) {break;}
        scatter_participant(t, a.sys[s].g[g].slot_off + k);
    }
    if(!bar.sync()) {return false;}
    for(int e = G.thread;; e += G.nthread)
    {
        k = e;
        if(!locate(mask, k, s, nslot)) {break;}
        place_participant(a, t, s, a.sys[s].g[g].slot_off + k);
    }
    if(!bar.sync()) {return false;}
    // narrow groups for short candidate sequences, as the launched build
    if(t.build_lanes <= 8) {build<8>(a, g, t, mask, G, sh.narrow);}
    else                   {build<32>(a, g, t, mask, G, sh.wide);}
    return bar.sync();
}

// clears the flagged systems' cell counters and chunk sums for the next rebuild
__device__ __forceinline__ void clear_cells(const Arena& a, const TermArrays& t, int g, ull mask, const Grid& G)
{
    for(ull m = mask; m; m &= m - 1)
    {
        const int s = __ffsll((long long)m) - 1;
        const GlobalParams& q = a.sys[s].g[g];
        for(int c = G.thread; c < q.ncell; c += G.nthread) {t.cell_count[q.cell_off + c] = 0;}
        const int nc = (q.ncell + CELL_CHUNK - 1) / CELL_CHUNK;
        for(int c = G.thread; c < nc; c += G.nthread) {t.cell_sum[chunk_sum_index(q, c)] = 0;}
    }
}

// ------------------------------------------------------------------- forces

// warp item e of term g: 32 / tpp slots, tpp lanes each (as k_pair).  The
// slot's head, coordinates, particle and first list word are requested
// together (every slot owns at least 32 words; those past the length are never
// used as indices), so the chain is two loads deep: these, then the partners.
template<int PREC, int G>
__device__ __forceinline__ void pair_item(const Arena& a, const TermArrays& t, double4* pair_force, int e)
{
    const int lane = threadIdx.x & 31;
    const int tpp = t.tpp, lt = __ffs(tpp) - 1;
    const long long s = ((long long)e * 32 + lane) >> lt;
    const int lg = lane & (tpp - 1);
    const bool active = s < t.np;
    SlotHead head{0, 0};
    int particle = 0;
    bool ovf = false;
    Acc<PREC> acc;
    if(active)
    {
        const long long np = t.np;
        const bool sm = t.slot_major != 0;
        const long long rs = sm ? tpp : np * tpp;
        const int* nbr = t.nbr + (sm ? s * t.words : s * tpp) + lg;
        const double4* pd = t.slot_pd;
        const double4 self = load_pd(pd + s);
        const int first = nbr[0];
        particle = t.slot_particle[s];
        head = slot_head(a, t, s);
        const int n = head.n;
        const PairEval<PREC, G, true, false, true, PREC == P_MIXED, true> eval(a, t, s, head.sys, self);
        double energy = 0.0;
        // RUN_BATCH partners requested together: words, then coordinates
        for(int k = lg; k < n; k += RUN_BATCH * tpp)
        {
            int q[RUN_BATCH];
            double4 pj[RUN_BATCH];
            double p1[RUN_BATCH];
#pragma unroll
            for(int u = 0; u < RUN_BATCH; ++u)
            {
                q[u] = u == 0 && k == lg ? first : (k + u * tpp < n ? nbr[u * rs] : -1);
            }
#pragma unroll
            for(int u = 0; u < RUN_BATCH; ++u)
            {
                pj[u] = q[u] >= 0 ? load_pd(pd + q[u]) : self;
                p1[u] = q[u] >= 0 ? eval.partner_p1(q[u]) : 0.0;
            }
            nbr += RUN_BATCH * rs;
#pragma unroll
            for(int u = 0; u < RUN_BATCH; ++u) {if(q[u] >= 0) {eval(pj[u], p1[u], q[u], acc, energy, ovf);}}
        }
    }
    for(int o = tpp / 2; o > 0; o >>= 1) {acc.shfl_add(o);}
    if(active && lg == 0 && (PREC == P_FP64 || head.n > 0)) {put_force(a, pair_force, particle, acc);}
    if(ovf) {atomicOr(&a.sys[head.sys].status, ST_FIXED_OVERFLOW);}
}

__host__ __device__ inline int warps_of(long long n) {return (int)((n + 31) / 32);}

// Warp item e of the bonded terms: records in the mixed form; in the plain form,
// whose formulas are long enough that one thread's three terms in a row would
// set the phase's time, dihedrals, angles and bonds by themselves.
template<int PREC>
__device__ __forceinline__ void local_item(const Arena& a, const LocalArrays& l, int e)
{
    const int lane = threadIdx.x & 31;
    DirectAdd<PREC> W;
    if constexpr(PREC == P_MIXED)
    {
        const long long b = (long long)e * 32 + lane;
        if(b < l.nrec) {do_record(a, l, b, W);}
    }
    else
    {
        const int n_di = warps_of(l.ndihd), n_an = warps_of(l.nangle);
        const int kind = e < n_di ? 2 : (e < n_di + n_an ? 1 : 0);
        const long long b = (long long)(e - (kind == 2 ? 0 : (kind == 1 ? n_di : n_di + n_an))) * 32 + lane;
        if(b >= (kind == 2 ? l.ndihd : (kind == 1 ? l.nangle : l.nbond))) {return;}
        if(a.any_frozen && a.sys[kind == 2 ? l.dihd_sys[b] : (kind == 1 ? l.angle_sys[b] : l.bond_sys[b])].frozen) {return;}
        if(kind == 2)      {dihedral_fp64<PREC, true, false>(a, l, b, W);}
        else if(kind == 1) {angle_fp64<PREC, true, false>(a, l, b, W);}
        else               {do_bond<PREC, true, false>(a, l, b, true, W);}
    }
}
__host__ __device__ inline int local_items(int precision, const LocalArrays& l)
{
    return precision == P_MIXED ? warps_of(l.nrec) : warps_of(l.ndihd) + warps_of(l.nangle) + warps_of(l.nbond);
}

__host__ __device__ inline int pair_items(const TermArrays& t) {return t.on ? (int)((t.np * t.tpp + 31) / 32) : 0;}

// The step's forces, longest items first: the dense DebyeHuckel lists, the
// other pair terms, then the bonded terms.
template<int PREC>
__device__ __forceinline__ void forces(const Arena& a, const RunArgs& r, const Grid& G)
{
    const int n_dh = pair_items(r.t[G_DH]), n_lj = pair_items(r.t[G_LJ]), n_ex = pair_items(r.t[G_EXV]);
    const int total = n_dh + n_lj + n_ex + local_items(PREC, r.l);
    for(int e = G.warp; e < total; e += G.nwarp)
    {
        int k = e;
        if(k < n_dh) {pair_item<PREC, G_DH>(a, r.t[G_DH], r.pair_force + G_DH * a.n, k); continue;}
        k -= n_dh;
        if(k < n_lj) {pair_item<PREC, G_LJ>(a, r.t[G_LJ], r.pair_force + G_LJ * a.n, k); continue;}
        k -= n_lj;
        if(k < n_ex) {pair_item<PREC, G_EXV>(a, r.t[G_EXV], r.pair_force + G_EXV * a.n, k); continue;}
        local_item<PREC>(a, r.l, k - n_ex);
    }
}

// --------------------------------------------------------------------- steps

template<int PREC, bool AUX>
__global__ void __launch_bounds__(RT, 1) k_run(const __grid_constant__ RunArgs r)
{
    __shared__ Shared sh;
    extern __shared__ __align__(16) unsigned char dyn[];
    SysDev* const sys = reinterpret_cast<SysDev*>(dyn);
    Arena a = r.a;
    a.sys = sys;
    const int nsys = a.nsys;
    const Grid G;
    Barrier bar{r, 0u};
    const unsigned full = 0xffffffffu;
    {
        static_assert(sizeof(SysDev) % sizeof(int4) == 0, "copied in 16-byte words");
        const int4* src = reinterpret_cast<const int4*>(r.a.sys);
        for(int w = threadIdx.x; w < nsys * (int)(sizeof(SysDev) / sizeof(int4)); w += RT)
        {
            const int4 v = src[w];
            reinterpret_cast<int4*>(dyn)[w] = v;
            if(blockIdx.x == 0 && r.b_pos) {reinterpret_cast<int4*>(r.b_sys)[w] = v;}
        }
        for(int w = threadIdx.x; w < nsys * NGLOBAL; w += RT) {(&sh.rebuilds[0][0])[w] = 0;}
    }
    __syncthreads();
    // a wait of an earlier launch of the chunk ran out (the first launch, which
    // alone writes the rollback copies, never starts with the bit set)
    if(r.kick && (sys[0].status & ST_BARRIER)) {return;}
    ull* const disp = r.disp2;                    // [2][nsys], zero between launches

    // this thread's first particle and its noise, drawn while the grid waits
    const long long i0 = G.thread;
    const int sys0 = i0 < a.n ? a.psys[i0] : -1;
    const int kind0 = sys0 >= 0 ? sys[sys0].integrator : I_VV;
    const bool noisy0 = sys0 >= 0 && !sys[sys0].frozen && (kind0 == I_BAOAB || kind0 == I_GBAOAB || (AUX && kind0 == I_GJF));
    double n0 = 0.0, n1 = 0.0, n2 = 0.0;
    auto draw = [&](int k) {
        if(noisy0) {const SysDev& S = sys[sys0]; gaussian3(S.seed, (ull)(i0 - S.off), S.step + k, n0, n1, n2);}
    };
    draw(0);

    for(int k = 0; k < r.nsteps; ++k)
    {
        ull* const d = disp + (k & 1) * nsys;
        // ---- integrator pass
        for(long long i = i0; i - (threadIdx.x & 31) < a.n; i += G.nthread)
        {
            const int s = i == i0 ? sys0 : (i < a.n ? a.psys[i] : -1);
            double d2 = 0.0;
            if(k == 0 && r.b_pos && s >= 0)       // the state before the chunk
            {
                r.b_pos[i] = a.pos[i];
                r.b_vel[i] = a.vel[i];
                r.b_force[i] = static_cast<const longlong4*>(a.force)[i];
                if(AUX) {r.b_accel[i] = a.accel[i];}
            }
            if(s >= 0 && !sys[s].frozen)
            {
                SysDev& S = sys[s];
                const ull step = S.step + k;
                d2 = advance_particle<PREC, AUX>(a, S, i, k > 0 || r.kick, step, [&](double& x, double& y, double& z) {
                    if(i == i0) {x = n0; y = n1; z = n2;}
                    else        {gaussian3(S.seed, (ull)(i - S.off), step, x, y, z);}
                }, [&](double& fx, double& fy, double& fz) {run_force<PREC>(r, k == 0, i, fx, fy, fz);});
            }
            const int s0 = __shfl_sync(full, s, 0);
            if(__all_sync(full, s == s0 || s < 0))
            {
                double m = d2;
#pragma unroll
                for(int o = 16; o > 0; o >>= 1) {m = fmax(m, __shfl_xor_sync(full, m, o));}
                if((threadIdx.x & 31) == 0) {atomicMax(&d[s0], (ull)__double_as_longlong(m));}
            }
            else if(s >= 0) {atomicMax(&d[s], (ull)__double_as_longlong(d2));}
        }
        if(threadIdx.x < NGLOBAL) {sh.flag[threadIdx.x] = 0;}
        if(!bar.sync()) {return;}
        // ---- reduce_margin of every system (core/PeriodicGridCellList.hpp:100-110),
        // by every block for itself
        for(int s = threadIdx.x; s < nsys; s += RT)
        {
            SysDev& S = sys[s];
            if(S.frozen) {continue;}
            const double dd = 2 * sqrt(__longlong_as_double((long long)d[s]));
            for(int g = 0; g < NGLOBAL; ++g)
            {
                GlobalParams& P = S.g[g];
                if(!r.t[g].on || !P.on) {continue;}
                P.current_margin = __dsub_rn(P.current_margin, dd);
                if(P.current_margin < 0)
                {
                    atomicOr(&sh.flag[g], 1ull << s);
                    P.current_margin = __dmul_rn(P.cutoff, P.margin);
                    sh.rebuilds[s][g] += 1;
                }
            }
        }
        // the other displacement buffer, read by every block before the last barrier
        if(blockIdx.x == 0) {for(int s = threadIdx.x; s < nsys; s += RT) {disp[((k & 1) ^ 1) * nsys + s] = 0;}}
        __syncthreads();
        if(sh.flag[G_EXV] && !rebuild<G_EXV>(a, r.t[G_EXV], sh.flag[G_EXV], G, sh, bar)) {return;}
        if(sh.flag[G_DH] && !rebuild<G_DH>(a, r.t[G_DH], sh.flag[G_DH], G, sh, bar)) {return;}
        if(sh.flag[G_LJ] && !rebuild<G_LJ>(a, r.t[G_LJ], sh.flag[G_LJ], G, sh, bar)) {return;}
        // ---- forces
        forces<PREC>(a, r, G);
        for(int g = 0; g < NGLOBAL; ++g) {if(sh.flag[g]) {clear_cells(a, r.t[g], g, sh.flag[g], G);}}
        bar.arrive();
        draw(k + 1);                              // while the others finish
        if(!bar.wait()) {return;}
    }
    bar.leave();
    // ---- the whole force, closing half of the last step, counters
    if(r.close || PREC == P_FP64)
    {
        for(long long i = i0; i < a.n; i += G.nthread)
        {
            const int s = a.psys[i];
            if(sys[s].frozen) {continue;}
            double fx, fy, fz;
            run_force<PREC>(r, false, i, fx, fy, fz);
            if constexpr(PREC == P_FP64) {static_cast<double4*>(a.force)[i] = make_double4(fx, fy, fz, 0.0);}
            if(r.close) {close_particle(a, sys[s], i, sys[s].step + r.nsteps, fx, fy, fz);}
        }
    }
    __syncthreads();
    for(int s = threadIdx.x; s < nsys; s += RT)
    {
        SysDev& S = r.a.sys[s];
        if(sys[s].status) {atomicOr(&S.status, sys[s].status);}
        if(blockIdx.x != 0) {continue;}
        disp[s] = 0;
        disp[nsys + s] = 0;
        if(sys[s].frozen) {continue;}
        S.step = sys[s].step + r.nsteps;
        for(int g = 0; g < NGLOBAL; ++g)
        {
            S.g[g].current_margin = sys[s].g[g].current_margin;
            S.g[g].rebuilds += sh.rebuilds[s][g];
        }
    }
}

}  // namespace

cudaError_t launch_run(RunArgs r, int sms, cudaStream_t s)
{
    // blocks: a warp per item of the force phase, at most one block per SM
    int items = 0;
    for(int g = 0; g < NGLOBAL; ++g) {items += pair_items(r.t[g]);}
    items += local_items(r.a.precision, r.l);
    items = std::max(items, warps_of(r.a.n));
    const int blocks = r.blocks > 0 ? r.blocks : std::max(1, std::min(sms, (items + RT / 32 - 1) / (RT / 32)));
    r.cluster = blocks <= RUN_CLUSTER_MAX ? 1 : 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(RT);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    if(r.cluster)
    {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = blocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    }
    else
    {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cfg.dynamicSmemBytes = sizeof(SysDev) * r.a.nsys;
    const bool aux = r.a.accel != nullptr;
    auto* kernel = r.a.precision == P_FP64 ? (aux ? k_run<P_FP64, true> : k_run<P_FP64, false>)
                                           : (aux ? k_run<P_MIXED, true> : k_run<P_MIXED, false>);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(sizeof(SysDev) * RUN_MAX_SYSTEMS));
    if(e != cudaSuccess) {return e;}
    const cudaError_t launched = cudaLaunchKernelEx(&cfg, kernel, r);
    if(launched == cudaSuccess) {note_launches(1);}
    return launched;
}

}  // namespace mjg
