// The pair kernels and their dispatch, instantiated term by term (pair_exv.cu,
// pair_dh.cu, pair_lj.cu), so that the units compile side by side.
//
// One thread owns one slot (particle) and walks its column-major list, so a
// warp of 32 consecutive slots -- 32 spatial neighbours after the cell-order
// renumbering -- loads 32 consecutive list words per step and mostly the same
// partner coordinates.  The owner accumulates and writes its particle's force
// once: no scattered atomics.  Each pair is evaluated from both sides (the
// reference evaluates it once and applies Newton's third law).
//
// P_FP64  : the reference's arithmetic in FP64 (the plain form).
// P_MIXED : the displacement and the cutoff test in FP64, the potential in FP32,
//           every pair force rounded to 2^-28 fixed point and summed as int64,
//           so the sum does not depend on list order or launch shape.
#pragma once
#include "pair_eval.cuh"

namespace mjg {

namespace {

constexpr int TPB = 256;

// List words PF_ROWS block rows ahead of the walk are requested into L2
// (prefetch.global.L2: no register, no wait), so that the walk's own loads of
// those words hit L2 instead of waiting on DRAM: a long list is a chain of
// dependent loads, and the rows a warp reads are np * TPP words apart.
constexpr int PF_ROWS = 8;
__device__ __forceinline__ void prefetch_l2(const void* p)
{
    asm volatile("prefetch.global.L2 [%0];" :: "l"(p));
}
// One request to the bulk copy engine for `bytes` (a multiple of 16) from p
// (16-byte aligned) into L2; nothing waits on it.
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(p), "r"(bytes) : "memory");
}

// One slot per TPP consecutive threads.  UNR: partners requested per batch.
// 1 keeps one partner in flight ahead of the pair being evaluated; 2 and 4
// issue the batch's list words, then its coordinates, before evaluating any
// of them (more loads in flight per thread, more registers).

// Counting sort of a block's slots by their list length (in units of `per`
// partners, 32 bins): returns the block-local index of the slot this group of
// threads takes, with that slot's head (read once by the group that loaded
// it, handed over in shared memory).  Slot numbering is unchanged; only
// which threads walk which list.  Every thread of the block must call it.
template<int GROUPS>
__device__ __forceinline__ int sorted_group(const Arena& a, const TermArrays& t, long long first_slot,
                                            int group, bool leader, int per, SlotHead& head)
{
    constexpr int NB = 32;
    __shared__ int bin_count[NB];
    __shared__ int perm[GROUPS];
    __shared__ SlotHead heads[GROUPS];
    if(threadIdx.x < NB) {bin_count[threadIdx.x] = 0;}
    const long long s = first_slot + group;
    SlotHead h{0, 0};
    if(leader && s < t.np) {h = slot_head(a, t, s);}
    __syncthreads();
    const int nb = (h.n + per - 1) / per;
    const int bin = nb < NB - 1 ? nb : NB - 1;
    const int rank = leader ? atomicAdd(&bin_count[bin], 1) : 0;
    if(leader) {heads[group] = h;}
    __syncthreads();
    if(threadIdx.x < 32)
    {
        const int v = bin_count[threadIdx.x];
        int incl = v;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if((int)threadIdx.x >= o) {incl += y;}
        }
        bin_count[threadIdx.x] = incl - v;
    }
    __syncthreads();
    if(leader) {perm[bin_count[bin] + rank] = group;}
    __syncthreads();
    const int g = perm[group];
    head = heads[g];
    return g;
}

// Both pair kernels are held to 64 registers (four 256-thread blocks per SM):
// they wait on memory, and the occupancy is worth more than the few words
// spilled in the widest variants.
template<int PREC, int G, bool NF, bool NE, int TPP, bool PER, int UNR, bool SORT = false, bool HALF = false>
__global__ void __launch_bounds__(TPB, 4) k_pair(Arena a, TermArrays t)
{
    // TPP consecutive threads share one slot; lane lg walks partners lg,
    // lg + TPP, ... which the blocked list layout stores next to each other.
    // SORT: the block's groups take its slots in order of list length.
    const long long gt = (long long)blockIdx.x * TPB + threadIdx.x;
    long long s = gt / TPP;
    const int lg = (int)(threadIdx.x % TPP);
    SlotHead head{0, 0};
    if(SORT)
    {
        const long long first = (long long)blockIdx.x * (TPB / TPP);
        s = first + sorted_group<TPB / TPP>(a, t, first, (int)(threadIdx.x / TPP), lg == 0, TPP * UNR, head);
    }
    const bool active = s < t.np;
    double energy = 0.0;
    bool ovf = false;
    Acc<PREC> acc;
    int particle = 0;
    if(active && (!SORT || head.n > 0))    // a sorted group knows that its list is empty
    {
        // word k = lg + r TPP of the slot's list: blocked layout, rows np TPP
        // words apart; slot-major layout, the slot's words in a row, the
        // whole list requested into L2 (16-byte aligned: a multiple of 32
        // words per slot) before the walk starts
        const bool sm = t.slot_major != 0;
        const long long rs = sm ? TPP : t.np * TPP;
        const int* __restrict__ nbr = t.nbr + (sm ? s * t.words : s * TPP) + lg;
        const double4* __restrict__ pd = t.slot_pd;
        // the slot's coordinates, particle and first list word are requested
        // with its head (every slot owns at least TPP words; a word past the
        // length is never used as an index), so the walk starts one load
        // latency after the launch
        const double4 self = load_pd(pd + s);
        int q = __ldg(nbr);
        particle = t.slot_particle[s];
        if(!SORT) {head = slot_head(a, t, s);}
        const int n = head.n;
        if(sm && lg == 0 && n > 0) {bulk_prefetch_l2(t.nbr + s * t.words, (unsigned)((n + 3) / 4) * 16u);}
        if(n > 0)
        {
        const PairEval<PREC, G, NF, NE, PER, HALF> eval(a, t, s, head.sys, self);
        if(UNR == 1)
        {
            // software pipeline: the next partner's index and coordinates are
            // requested before the current pair is evaluated
            int k = lg;
            double4 pj = self;
            double p1 = 0.0;
            if(k < n) {pj = load_pd(pd + q); p1 = eval.partner_p1(q);}
            for(; k < n; k += TPP)
            {
                const int kn = k + TPP;
                nbr += rs;
                if(!sm && k + PF_ROWS * TPP < n) {prefetch_l2(nbr + (PF_ROWS - 1) * rs);}
                int qn = q;
                double4 pn = pj;
                double p1n = p1;
                if(kn < n) {qn = __ldg(nbr); pn = load_pd(pd + qn); p1n = eval.partner_p1(qn);}
                eval(pj, p1, q, acc, energy, ovf);
                q = qn;
                pj = pn;
                p1 = p1n;
            }
        }
        else
        {
            for(int k = lg; k < n; k += UNR * TPP)
            {
                int qv[UNR];
                double4 pv[UNR];
                double p1v[UNR];
#pragma unroll
                for(int u = 0; u < UNR; ++u)
                {
                    const int kp = k + (PF_ROWS + u) * TPP;
                    if(!sm && kp < n) {prefetch_l2(nbr + (PF_ROWS + u) * rs);}
                }
#pragma unroll
                for(int u = 0; u < UNR; ++u)
                {
                    const int kk = k + u * TPP;
                    qv[u] = kk < n ? (u == 0 && k == lg ? q : __ldg(nbr + u * rs)) : -1;
                }
#pragma unroll
                for(int u = 0; u < UNR; ++u)
                {
                    pv[u] = qv[u] >= 0 ? load_pd(pd + qv[u]) : self;
                    p1v[u] = qv[u] >= 0 ? eval.partner_p1(qv[u]) : 0.0;
                }
#pragma unroll
                for(int u = 0; u < UNR; ++u) {if(qv[u] >= 0) {eval(pv[u], p1v[u], qv[u], acc, energy, ovf);}}
                nbr += UNR * rs;
            }
        }
        }
    }
    const int sys = head.sys;
    // group reduction: exact in fixed point, fixed order in FP64
#pragma unroll
    for(int o = TPP / 2; o > 0; o >>= 1) {acc.shfl_add(o);}
    if(NF && lg == 0 && head.n > 0) {acc.store(a.force, particle);}
    if(ovf) {atomicOr(&a.sys[sys].status, ST_FIXED_OVERFLOW);}
    if(NE)
    {
        const unsigned full = 0xffffffffu;
        const int s0 = __shfl_sync(full, sys, 0);
        const bool uniform = __all_sync(full, !active || sys == s0);
        if(uniform)
        {
            double e = energy;
#pragma unroll
            for(int o = 16; o > 0; o >>= 1) {e += __shfl_xor_sync(full, e, o);}
            if(__any_sync(full, active) && (threadIdx.x & 31) == 0) {atomicAdd(&a.sys[s0].energy[T_EXV + G], e);}
        }
        else if(active)
        {
            atomicAdd(&a.sys[sys].energy[T_EXV + G], energy);
        }
    }
}

// Block-vector schedule: one thread per slot reads its list L words at a
// time with one vector load (the blocked layout with L = tpp stores a slot's
// words k .. k + L - 1 next to each other, 4 L bytes aligned), the next block
// of words is requested before the current one is evaluated, and up to four
// partner coordinates are requested together.  A slot's list then costs one
// list latency per L partners instead of one per partner.
template<int L>
__device__ __forceinline__ void load_block(const int* __restrict__ p, int (&q)[L])
{
    if(L == 2)
    {
        const int2 v = __ldg(reinterpret_cast<const int2*>(p));
        q[0] = v.x; q[1] = v.y;
    }
    else
    {
#pragma unroll
        for(int c = 0; c < L / 4; ++c)
        {
            const int4 v = __ldg(reinterpret_cast<const int4*>(p) + c);
            q[4 * c] = v.x; q[4 * c + 1] = v.y; q[4 * c + 2] = v.z; q[4 * c + 3] = v.w;
        }
    }
}

// Schedules 2 and 3 (blocked list layout only).
// SORT: the block's threads take its 256 slots in order of their number of
// list blocks (a counting sort in shared memory), so that the lanes of a warp
// walk lists of about the same length; the slots themselves, and with them
// the spatial order of the partners, stay where they are.
template<int PREC, int G, bool PER, int L, bool SORT, bool HALF>
__global__ void __launch_bounds__(TPB, 4) k_pair_vec(Arena a, TermArrays t)
{
    long long s = (long long)blockIdx.x * TPB + threadIdx.x;
    SlotHead head{0, 0};
    if(SORT)
    {
        const long long first = (long long)blockIdx.x * TPB;
        s = first + sorted_group<TPB>(a, t, first, (int)threadIdx.x, true, L, head);
    }
    if(s >= t.np || (SORT && head.n == 0)) {return;}   // an empty list (frequent in half lists): nothing to add
    // the slot's coordinates, particle and first block of words are requested
    // with its head (every slot owns at least L words; words past the length are
    // never used as indices)
    const double4 self = load_pd(t.slot_pd + s);
    int q[L];
    load_block<L>(t.nbr + s * L, q);
    const int particle = t.slot_particle[s];
    if(!SORT)
    {
        head = slot_head(a, t, s);
        if(head.n == 0) {return;}
    }
    const int sys = head.sys;
    double energy = 0.0;
    bool ovf = false;
    Acc<PREC> acc;
    const PairEval<PREC, G, true, false, PER, HALF> eval(a, t, s, sys, self);
    const long long np = t.np;
    const int n = head.n;
    const double4* __restrict__ pd = t.slot_pd;
    constexpr int W = L < 4 ? L : 4;                 // partners requested together
    for(int k = 0; k < n; k += L)
    {
        int qn[L];
        if(k + L < n) {load_block<L>(t.nbr + ((long long)(k / L + 1) * np + s) * L, qn);}
        if(k + PF_ROWS * L < n) {prefetch_l2(t.nbr + ((long long)(k / L + PF_ROWS) * np + s) * L);}
        const int m = min(L, n - k);
#pragma unroll
        for(int u0 = 0; u0 < L; u0 += W)
        {
            double4 pv[W];
            int jv[W];                               // half lists: the partners' particles, read beside
#pragma unroll                                       // their coordinates, so the atomics wait on nothing
            for(int u = 0; u < W; ++u)
            {
                pv[u] = u0 + u < m ? load_pd(pd + q[u0 + u]) : self;
                jv[u] = HALF && u0 + u < m ? t.slot_particle[q[u0 + u]] : -1;
            }
#pragma unroll
            for(int u = 0; u < W; ++u) {if(u0 + u < m) {eval(pv[u], eval.partner_p1(q[u0 + u]), q[u0 + u], acc, energy, ovf, jv[u]);}}
        }
#pragma unroll
        for(int u = 0; u < L; ++u) {q[u] = qn[u];}
    }
    acc.store(a.force, particle);
    if(ovf) {atomicOr(&a.sys[sys].status, ST_FIXED_OVERFLOW);}
}

// Warp-balanced schedule of the mixed form's force launch (schedule 1,
// blocked list layout only): a warp owns 32
// consecutive slots and splits the concatenation of their lists into 32 equal
// contiguous chunks, one per lane, so every lane evaluates the same number of
// pairs whatever the list lengths (one slot per thread leaves the lanes of
// short lists idle).  A lane sums the pairs of one slot in registers and adds
// the sum to the particle's fixed-point force with integer atomics when its
// chunk leaves that slot; integer sums are exact, so the result does not
// depend on where the chunks start.
template<int G, bool PER, int UNR, bool HALF>
__global__ void __launch_bounds__(TPB) k_pair_warp(Arena a, TermArrays t)
{
    __shared__ int seg[TPB / 32][33];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const long long gt = (long long)blockIdx.x * TPB + threadIdx.x;
    const long long s0 = gt - lane;                  // first slot of this warp
    int n_my = 0;
    if(gt < t.np)
    {
        n_my = slot_head(a, t, gt).n;                // 0 in a frozen system
    }
    int incl = n_my;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(full, incl, o);
        if(lane >= o) {incl += y;}
    }
    seg[wl][lane] = incl - n_my;                     // first entry of slot s0 + lane
    if(lane == 31) {seg[wl][32] = incl;}
    __syncwarp();
    const int total = seg[wl][32];
    const int per = (total + 31) >> 5;
    int e = min(lane * per, total);
    const int e_end = min(e + per, total);
    if(e >= e_end) {return;}
    // slot of entry e: the last j with seg[j] <= e (seg is non-decreasing)
    int j = 0;
#pragma unroll
    for(int b = 16; b > 0; b >>= 1) {if(j + b < 32 && seg[wl][j + b] <= e) {j += b;}}

    const long long np = t.np;
    const int tpp = t.tpp;
    const int lt = __ffs(tpp) - 1;                   // tpp is a power of two
    const int* __restrict__ nbr = t.nbr;
    const double4* __restrict__ pd = t.slot_pd;
    while(e < e_end)
    {
        const long long s = s0 + j;
        const int b = seg[wl][j];
        const int kend = min(seg[wl][j + 1], e_end) - b;
        const int sys = t.slot_sys[s];
        const PairEval<P_MIXED, G, true, false, PER, HALF> eval(a, t, s, sys);
        Acc<P_MIXED> acc;
        double energy = 0.0;
        bool ovf = false;
        for(int k = e - b; k < kend; k += UNR)
        {
            int qv[UNR];
            double4 pv[UNR];
#pragma unroll
            for(int u = 0; u < UNR; ++u)
            {
                const int kk = k + u;
                qv[u] = kk < kend ? __ldg(nbr + (((long long)(kk >> lt) * np + s) << lt) + (kk & (tpp - 1))) : -1;
            }
#pragma unroll
            for(int u = 0; u < UNR; ++u) {pv[u] = qv[u] >= 0 ? load_pd(pd + qv[u]) : eval.pi;}
#pragma unroll
            for(int u = 0; u < UNR; ++u)
            {
                if(qv[u] >= 0) {eval(pv[u], eval.partner_p1(qv[u]), qv[u], acc, energy, ovf);}
            }
        }
        if(acc.x | acc.y | acc.z)
        {
            unsigned long long* f =
                reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(a.force) + t.slot_particle[s]);
            atomicAdd(f + 0, (unsigned long long)acc.x);
            atomicAdd(f + 1, (unsigned long long)acc.y);
            atomicAdd(f + 2, (unsigned long long)acc.z);
        }
        if(ovf) {atomicOr(&a.sys[sys].status, ST_FIXED_OVERFLOW);}
        e = b + kend;
        ++j;
        while(j < 32 && seg[wl][j + 1] == seg[wl][j]) {++j;}     // skip empty lists
    }
}

template<int PREC, int G, int TPP, bool PER, bool HALF>
void dispatch_per(const Arena& a, TermArrays& t, bool nf, bool ne, cudaStream_t s)
{
    const unsigned nb = (unsigned)((t.np * TPP + TPB - 1) / TPB);
    if(nf && ne)  {k_pair<PREC, G, true,  true,  TPP, PER, 1><<<nb, TPB, 0, s>>>(a, t);}
    else if(nf)
    {
        // the per-step force launch: schedule and partner batch depth are tunable
        if constexpr(TPP > 1 && TPP <= 16)   // 32-word blocks: the slot-per-group kernel instead
        {
            if(t.schedule == 2 || t.schedule == 3)
            {
                const unsigned nv = (unsigned)((t.np + TPB - 1) / TPB);
                if(t.schedule == 3) {k_pair_vec<PREC, G, PER, TPP, true,  HALF><<<nv, TPB, 0, s>>>(a, t);}
                else                {k_pair_vec<PREC, G, PER, TPP, false, HALF><<<nv, TPB, 0, s>>>(a, t);}
                return;
            }
        }
        if(PREC == P_MIXED && t.schedule == 1)
        {
            const unsigned nw = (unsigned)((t.np + TPB - 1) / TPB);
            if(t.unroll == 4)      {k_pair_warp<G, PER, 4, HALF><<<nw, TPB, 0, s>>>(a, t);}
            else if(t.unroll == 2) {k_pair_warp<G, PER, 2, HALF><<<nw, TPB, 0, s>>>(a, t);}
            else                   {k_pair_warp<G, PER, 1, HALF><<<nw, TPB, 0, s>>>(a, t);}
        }
        else if(t.schedule == 4)
        {
            if(t.unroll == 4)      {k_pair<PREC, G, true, false, TPP, PER, 4, true, HALF><<<nb, TPB, 0, s>>>(a, t);}
            else if(t.unroll == 2) {k_pair<PREC, G, true, false, TPP, PER, 2, true, HALF><<<nb, TPB, 0, s>>>(a, t);}
            else                   {k_pair<PREC, G, true, false, TPP, PER, 1, true, HALF><<<nb, TPB, 0, s>>>(a, t);}
        }
        else if(t.unroll == 4) {k_pair<PREC, G, true, false, TPP, PER, 4, false, HALF><<<nb, TPB, 0, s>>>(a, t);}
        else if(t.unroll == 2) {k_pair<PREC, G, true, false, TPP, PER, 2, false, HALF><<<nb, TPB, 0, s>>>(a, t);}
        else                   {k_pair<PREC, G, true, false, TPP, PER, 1, false, HALF><<<nb, TPB, 0, s>>>(a, t);}
    }
    else if(ne)   {k_pair<PREC, G, false, true,  TPP, PER, 1><<<nb, TPB, 0, s>>>(a, t);}
}

template<int PREC, int G, int TPP, bool HALF>
void dispatch_tpp(const Arena& a, TermArrays& t, bool nf, bool ne, cudaStream_t s)
{
    if(t.any_periodic) {dispatch_per<PREC, G, TPP, true,  HALF>(a, t, nf, ne, s);}
    else               {dispatch_per<PREC, G, TPP, false, HALF>(a, t, nf, ne, s);}
}

// HALF: the mixed form's force launch on half lists (the partner's share
// added by the same evaluation); a template argument, so that the full-list
// kernels carry none of its code
template<int PREC, int G, bool HALF = false>
void dispatch(const Arena& a, TermArrays& t, bool nf, bool ne, cudaStream_t s)
{
    switch(t.tpp)
    {
        case 1:  dispatch_tpp<PREC, G, 1 , HALF>(a, t, nf, ne, s); break;
        case 2:  dispatch_tpp<PREC, G, 2 , HALF>(a, t, nf, ne, s); break;
        case 4:  dispatch_tpp<PREC, G, 4 , HALF>(a, t, nf, ne, s); break;
        case 8:  dispatch_tpp<PREC, G, 8 , HALF>(a, t, nf, ne, s); break;
        case 16: dispatch_tpp<PREC, G, 16, HALF>(a, t, nf, ne, s); break;
        default: dispatch_tpp<PREC, G, 32, HALF>(a, t, nf, ne, s); break;
    }
}

}  // namespace

template<int G>
void pair_term(const Arena& a, TermArrays& t, bool need_force, bool need_energy, cudaStream_t s)
{
    note_launches(1);
    if(a.precision == P_FP64) {dispatch<P_FP64, G>(a, t, need_force, need_energy, s); return;}
    // mixed form: forces in FP32 with fixed-point sums (the per-step
    // path); energies, an observable read between steps, in the
    // reference's FP64 arithmetic
    if(need_force)
    {
        if(t.half) {dispatch<P_MIXED, G, true>(a, t, true, false, s);}
        else       {dispatch<P_MIXED, G>(a, t, true, false, s);}
    }
    if(need_energy)
    {
        // with the forces: the energy of calc_force_and_energy
        TermArrays te = t;
        te.fe_energy = need_force ? 1 : 0;
        if(need_force) {note_launches(1);}
        dispatch<P_FP64, G>(a, te, false, true, s);
    }
}

}  // namespace mjg
