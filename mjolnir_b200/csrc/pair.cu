// Global pair forces and energies over the full Verlet lists.
//
//   ExcludedVolume  forcefield/global/GlobalPairExcludedVolumeInteraction.hpp:148-195
//   DebyeHuckel     forcefield/global/GlobalPairInteraction.hpp:148-213 with
//                   forcefield/global/DebyeHuckelPotential.hpp:44-61
//   LennardJones    forcefield/global/GlobalPairLennardJonesInteraction.hpp:148-198
//                   with the Lorentz-Berthelot rule (ParameterList.hpp:240-251)
//
// The kernels are in pair_kernels.cuh; this unit holds the launch wrappers, the
// coordinate gather and the cutoff pair count.
#include "kernels.cuh"

namespace mjg {

// one instantiation per unit: pair_exv.cu, pair_dh.cu, pair_lj.cu
template<int G>
void pair_term(const Arena& a, TermArrays& t, bool need_force, bool need_energy, cudaStream_t s);
extern template void pair_term<G_EXV>(const Arena&, TermArrays&, bool, bool, cudaStream_t);
extern template void pair_term<G_DH>(const Arena&, TermArrays&, bool, bool, cudaStream_t);
extern template void pair_term<G_LJ>(const Arena&, TermArrays&, bool, bool, cudaStream_t);

namespace {

__global__ void k_gather(Arena a, TermArrays t)
{
    const long long s = (long long)blockIdx.x * 256 + threadIdx.x;
    if(s >= t.np) {return;}
    const double4 r = a.pos[t.slot_particle[s]];
    double4& d = t.slot_pd[s];
    d.x = r.x; d.y = r.y; d.z = r.z;
}

// pairs (s < q) inside the potential's cutoff: the margin-free pair count
template<int G>
__global__ void k_count_cut(Arena a, TermArrays t, int sys_filter, unsigned long long* out)
{
    const long long s = (long long)blockIdx.x * 256 + threadIdx.x;
    unsigned long long cnt = 0;
    if(s < t.np && (sys_filter < 0 || t.slot_sys[s] == sys_filter))
    {
        const SysDev& S = a.sys[t.slot_sys[s]];
        const GlobalParams& P = S.g[G];
        const double4 pi = t.slot_pd[s];
        const int n = t.nnb[s];
        for(int k = 0; k < n; ++k)
        {
            const int q = t.nbr[nbr_pos(k, s, t.np, t.tpp, t.words, t.slot_major)];
            if(q <= s) {continue;}
            const double4 pj = t.slot_pd[q];
            double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
            if(S.boundary == B_PERIODIC)
            {
                dx = min_image(dx, S.halfw[0], S.width[0]);
                dy = min_image(dy, S.halfw[1], S.width[1]);
                dz = min_image(dz, S.halfw[2], S.width[2]);
            }
            const double l2 = fma(dz, dz, fma(dy, dy, dx * dx));
            bool in = false;
            if(G == G_EXV && P.kind == EXV_HARD_CORE)
            {
                const double sg = pi.w + pj.w, core = t.slot_p1[s] + t.slot_p1[q];
                in = !(sg * P.cutoff_ratio + core < sqrt(l2));
            }
            else if(G == G_EXV) {const double sg = pi.w + pj.w; in = !(sg * sg * P.cutoff_ratio_sq < l2);}
            else if(G == G_DH) {in = l2 < P.abs_cutoff * P.abs_cutoff;}
            else               {const double sg = (pi.w + pj.w) / 2; in = !(sg * sg * P.cutoff_ratio_sq < l2);}
            cnt += in ? 1 : 0;
        }
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {cnt += __shfl_xor_sync(0xffffffffu, cnt, o);}
    if((threadIdx.x & 31) == 0 && cnt) {atomicAdd(out, cnt);}
}

}  // namespace

void launch_gather(const Arena& a, TermArrays& t, cudaStream_t s)
{
    if(!t.on || t.np == 0) {return;}
    k_gather<<<(unsigned)((t.np + 255) / 256), 256, 0, s>>>(a, t);
    note_launches(1);
}

void launch_pair(const Arena& a, int g, TermArrays& t, bool need_force, bool need_energy,
                 int /*calc_energy_form*/, cudaStream_t s, bool gather)
{
    if(!t.on || t.np == 0) {return;}
    if(gather) {launch_gather(a, t, s);}
    if(g == G_EXV)     {pair_term<G_EXV>(a, t, need_force, need_energy, s);}
    else if(g == G_DH) {pair_term<G_DH>(a, t, need_force, need_energy, s);}
    else               {pair_term<G_LJ>(a, t, need_force, need_energy, s);}
}

void launch_count_cut(const Arena& a, int g, TermArrays& t, int sys, unsigned long long* out,
                      cudaStream_t s)
{
    if(!t.on || t.np == 0) {return;}
    k_gather<<<(unsigned)((t.np + 255) / 256), 256, 0, s>>>(a, t);
    const unsigned nb = (unsigned)((t.np + 255) / 256);
    if(g == G_EXV)     {k_count_cut<G_EXV><<<nb, 256, 0, s>>>(a, t, sys, out);}
    else if(g == G_DH) {k_count_cut<G_DH ><<<nb, 256, 0, s>>>(a, t, sys, out);}
    else               {k_count_cut<G_LJ ><<<nb, 256, 0, s>>>(a, t, sys, out);}
    note_launches(2);
}

}  // namespace mjg
