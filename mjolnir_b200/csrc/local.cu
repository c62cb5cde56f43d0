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
            else               {do_bond_f32<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.bond_sys[b]].frozen), W);}
        }
    }
    if(mask & 2)
    {
        const long long b0 = l.win_angle[w], b1 = l.win_angle[w + 1];
        for(long long base = b0; base < b1; base += TPB)
        {
            const long long b = base + threadIdx.x;
            if(PREC == P_FP64) {do_angle<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.angle_sys[b]].frozen), W);}
            else               {do_angle_f32<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.angle_sys[b]].frozen), W);}
        }
    }
    if(mask & 4)
    {
        const long long b0 = l.win_dihd[w], b1 = l.win_dihd[w + 1];
        for(long long base = b0; base < b1; base += TPB)
        {
            const long long b = base + threadIdx.x;
            if(PREC == P_FP64) {do_dihedral<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.dihd_sys[b]].frozen), W);}
            else               {do_dihedral_f32<PREC, NF, NE>(a, l, b, b < b1 && !(a.any_frozen && a.sys[l.dihd_sys[b]].frozen), W);}
        }
    }
    if(NF)
    {
        __syncthreads();
        W.flush(a.force, a.n);
    }
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
