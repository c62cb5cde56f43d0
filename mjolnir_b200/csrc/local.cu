// Local (bonded) terms; the FP64 form keeps the reference's formulas, the
// mixed form evaluates them in FP32 from FP64 displacements, and with the
// FP64 formulas where a bond angle is within 11.5 degrees of collinear (see
// below):
//   BondLength + Harmonic   forcefield/local/BondLengthInteraction.hpp:126-199,
//                           forcefield/local/HarmonicPotential.hpp:25-35 (V = k (v - v0)^2)
//   BondAngle  + Harmonic   forcefield/local/BondAngleInteraction.hpp:129-188
//   Dihedral   + Cosine     forcefield/local/DihedralAngleInteraction.hpp:157-227,
//                           forcefield/local/CosinePotential.hpp:29-39
// One fused launch: one thread per bond / angle / dihedral of every system;
// the forces are summed per block in shared memory and land in the particles
// by atomics (FP64 atomics in the plain form, int64 fixed point in the mixed
// form, where the sum is exact and order independent).
#include "local_terms.cuh"

namespace mjg {

namespace {

constexpr int TPB = 256;
// blocks per SM of the record kernel: 64 registers each; 3 (80 registers) and 5
// (48, spilling) were slower (100 steps of 256 melts 38.3 ms; 39.4 and 38.8)
constexpr int LOCAL_BLOCKS = 4;

// One block per window of SEG particles: every bond, angle and dihedral whose
// smallest particle index falls in the window (terms are sorted by it at
// commit; win_* hold the per-window term ranges) adds its forces to the
// block's shared accumulator of SEG + HALO particles, which is flushed once
// per particle.  The trip counts are uniform over the block, so the warp
// energy reductions see whole warps.
// The mixed form is held to 48 registers (five blocks per SM): its FP64
// fallback for near-collinear geometry would otherwise set the register count
// (and the occupancy) of every thread; the rare fallback spills instead.
template<int PREC, bool NF, bool NE>
__global__ void __launch_bounds__(TPB, PREC == P_MIXED ? 5 : 3) k_local(Arena a, LocalArrays l, int mask)
{
    __shared__ typename WinT<PREC>::type win[Window<PREC>::SIZE];
    const int w = blockIdx.x;
    Window<PREC> W{win, w * SEG};
    if(NF)
    {
        for(int k = threadIdx.x; k < Window<PREC>::SIZE; k += TPB) {win[k] = 0;}
        __syncthreads();
    }
    if(mask & 1)
    {
        const long long b0 = l.win_bond[w], b1 = l.win_bond[w + 1];
        for(long long base = b0; base < b1; base += TPB)
        {
            const long long b = base + threadIdx.x;
            if(PREC == P_FP64) {do_bond<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.bond_sys[b]].frozen), W);}
            else               {if(b < b1 && !(a.any_frozen && a.sys[l.bond_sys[b]].frozen)) {do_bond_f32(a, l, b, W);}}
        }
    }
    if(mask & 2)
    {
        const long long b0 = l.win_angle[w], b1 = l.win_angle[w + 1];
        for(long long base = b0; base < b1; base += TPB)
        {
            const long long b = base + threadIdx.x;
            if(PREC == P_FP64) {do_angle<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.angle_sys[b]].frozen), W);}
            else               {if(b < b1 && !(a.any_frozen && a.sys[l.angle_sys[b]].frozen)) {do_angle_f32(a, l, b, W);}}
        }
    }
    if(mask & 4)
    {
        const long long b0 = l.win_dihd[w], b1 = l.win_dihd[w + 1];
        for(long long base = b0; base < b1; base += TPB)
        {
            const long long b = base + threadIdx.x;
            if(PREC == P_FP64) {do_dihedral<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.dihd_sys[b]].frozen), W);}
            else               {if(b < b1 && !(a.any_frozen && a.sys[l.dihd_sys[b]].frozen)) {do_dihedral_f32(a, l, b, W);}}
        }
    }
    if(NF)
    {
        __syncthreads();
        W.flush(a.force, a.n);
    }
}

// The mixed form's bonded forces of a step: one block per window of SEG
// particles, a thread per record (local_terms.cuh), summed in the window as
// above.  The terms that need the FP64 formulas are put aside in shared memory and
// done by the block's threads side by side: a few in a hundred of them (a chain
// whose angles relax from a random walk) are enough to reach every warp, and each
// warp would then wait for the long FP64 evaluation of one or two lanes (256 melts
// from their first frame: 127 us with the FP64 formulas in line, 89 put aside; 114
// for the separate terms).
struct DeferringWindow : Window<P_MIXED> {
    static constexpr bool DEFER = true;
    int* count;          // [2] angles, dihedrals put aside
    int* queue;          // [2][TPB]
    __device__ __forceinline__ void defer_angle(int t)    {queue[atomicAdd(&count[0], 1)] = t;}
    __device__ __forceinline__ void defer_dihedral(int t) {queue[TPB + atomicAdd(&count[1], 1)] = t;}
};

__global__ void __launch_bounds__(TPB, LOCAL_BLOCKS) k_local_records(Arena a, LocalArrays l)
{
    __shared__ unsigned win[Window<P_MIXED>::SIZE];
    __shared__ int queue[2 * TPB];
    __shared__ int count[2];
    const int w = blockIdx.x;
    DeferringWindow W;
    W.w = win; W.base = w * SEG; W.count = count; W.queue = queue;
    for(int k = threadIdx.x; k < Window<P_MIXED>::SIZE; k += TPB) {win[k] = 0;}
    if(threadIdx.x < 2) {count[threadIdx.x] = 0;}
    __syncthreads();
    const long long end = l.win_rec[w + 1];
    for(long long first = l.win_rec[w]; first < end; first += TPB)
    {
        const long long r = first + threadIdx.x;
        if(r < end) {do_record(a, l, r, W);}
        __syncthreads();
        // angles by the first half of the block, dihedrals by the second
        const int half = threadIdx.x / (TPB / 2);
        const int n = count[half];
        Window<P_MIXED>& V = W;
        for(int k = threadIdx.x % (TPB / 2); k < n; k += TPB / 2)
        {
            if(half == 0) {angle_fp64<P_MIXED, true, false>(a, l, queue[k], V);}
            else          {dihedral_fp64<P_MIXED, true, false>(a, l, queue[TPB + k], V);}
        }
        __syncthreads();
        if(threadIdx.x < 2) {count[threadIdx.x] = 0;}
        __syncthreads();
    }
    W.flush(a.force, a.n);
}

template<int PREC, bool NF, bool NE>
void run_all(const Arena& a, const LocalArrays& l, int mask, cudaStream_t s)
{
    if(l.nwin == 0 || (l.nbond + l.nangle + l.ndihd) == 0) {return;}
    k_local<PREC, NF, NE><<<l.nwin, TPB, 0, s>>>(a, l, mask);
    note_launches(1);
}

}  // namespace

void launch_local(const Arena& a, const LocalArrays& l, int mask, bool nf, bool ne,
                  int /*calc_energy_form*/, cudaStream_t s)
{
    if(a.precision == P_MIXED && mask == 7 && nf && !ne)
    {
        if(l.nwin == 0 || l.nrec == 0) {return;}
        k_local_records<<<l.nwin, TPB, 0, s>>>(a, l);
        note_launches(1);
        return;
    }
    if(a.precision == P_FP64)
    {
        if(nf && ne) {run_all<P_FP64, true, true>(a, l, mask, s);}
        else if(nf)  {run_all<P_FP64, true, false>(a, l, mask, s);}
        else if(ne)  {run_all<P_FP64, false, true>(a, l, mask, s);}
    }
    else
    {
        // mixed form: forces in FP32 (the per-step path); energies, an
        // observable read between steps, in the reference's FP64 arithmetic
        if(nf)       {run_all<P_MIXED, true, false>(a, l, mask, s);}
        if(ne)       {run_all<P_FP64, false, true>(a, l, mask, s);}
    }
}

}  // namespace mjg
