// Evaluation of one pair and its force accumulator, shared by the pair
// launches (pair.cu) and the multi-step kernel of small arenas (run.cu).
#pragma once
#include "kernels.cuh"

#include <type_traits>

namespace mjg {

// Single-instruction forms of the mixed form's reciprocal root and power of
// two.  Squared distances and exponents of listed pairs are normal numbers, for
// which these give the floats of the general forms (rsqrtf, __expf, __frcp_rn: every
// mantissa from 2^-60 to 2^60, tests/test_gpu_fast_math.py), which spend as many
// instructions again on subnormal ones.  A subnormal or zero squared distance ends
// in an infinite or NaN force, which the fixed-point range check reports.
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float exp2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 1 / x: the hardware's approximation and one Newton step, r + r (1 - x r), whose
// residual is exact in the fused product-sum: the nearest float.
__device__ __forceinline__ float reciprocal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}

// slot coordinates and parameter in one 32-byte load (32-byte aligned)
__device__ __forceinline__ double4 load_pd(const double4* p)
{
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

template<int PREC>
struct Acc;

template<> struct Acc<P_FP64>
{
    double x = 0, y = 0, z = 0;
    __device__ __forceinline__ void add(double c, double dx, double dy, double dz, bool&)
    {
        x = fma(dx, c, x); y = fma(dy, c, y); z = fma(dz, c, z);
    }
    __device__ __forceinline__ void shfl_add(int o)
    {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    __device__ __forceinline__ void store(void* force, long long i) const
    {
        double4* f = static_cast<double4*>(force) + i;
        double4 v = *f;
        v.x += x; v.y += y; v.z += z;
        *f = v;
    }
};

template<> struct Acc<P_MIXED>
{
    long long x = 0, y = 0, z = 0;
    __device__ __forceinline__ void add(double c, double dx, double dy, double dz, bool& ovf)
    {
        const double fx = c * dx, fy = c * dy, fz = c * dz;
        const double m = fmax(fabs(fx), fmax(fabs(fy), fabs(fz)));
        ovf |= !(m < FX_LIMIT * FX_INV_SCALE);
        x += fx_from_double(fx); y += fx_from_double(fy); z += fx_from_double(fz);
    }
    // the mixed form's plain potentials: the FP32 pair coefficient c times
    // the FP64 displacement, each component rounded once to the fixed-point
    // grid (fx_product); `bound` >= |c| |r| (|c| max(|r|^2, 1) or |c| |r|, in
    // FP32) flags a force outside the fixed-point range
    __device__ __forceinline__ void add_c(float c, float bound, double dx, double dy, double dz, bool& ovf)
    {
        const double cs = fx_coefficient(c);
        ovf |= !(bound < (float)(FX_LIMIT * FX_INV_SCALE));
        x += fx_product(cs, dx);
        y += fx_product(cs, dy);
        z += fx_product(cs, dz);
    }
    __device__ __forceinline__ void shfl_add(int o)
    {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    // integer atomics: exact and order independent, so the force launches of
    // different terms and the bonded launch may run concurrently
    __device__ __forceinline__ void store(void* force, long long i) const
    {
        unsigned long long* f = reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + i);
        if(x) {atomicAdd(f + 0, (unsigned long long)x);}
        if(y) {atomicAdd(f + 1, (unsigned long long)y);}
        if(z) {atomicAdd(f + 2, (unsigned long long)z);}
    }
};

// Constants of one slot's pair evaluations and the evaluation of one pair
// (slot s, partner q).  PER: some system of the arena is periodic (the
// minimum image is applied where the system asks for it); without it the
// image code is compiled out.
// HALF: half lists; HALF_RT: the list form is known at run time (TermArrays::half).
template<int PREC, int G, bool NF, bool NE, bool PER, bool HALF = false, bool HALF_RT = false>
struct PairEval {
    const SysDev* S;
    double4 pi;
    long long s;
    int halfw_hi;               // image_needed
    double crsq, coefc, eps, eps12, inv_debye, abs_cut_sq, qi, inv4pi, epsi, cr;
    float eps12f, epsf, coefcf, invdf, crsqf, wif;
    int kind, power;
    bool half;                  // HALF_RT: half lists
    bool fe;                    // energy-only: the force-and-energy rule of the generic loop
    const double* slot_p1;
    void* force;
    const int* slot_particle;

    __device__ __forceinline__ PairEval(const Arena& a, const TermArrays& t, long long slot, int sys)
        : PairEval(a, t, slot, sys, t.slot_pd[slot]) {}
    // self: the slot's coordinates and parameter, read by the caller
    __device__ __forceinline__ PairEval(const Arena& a, const TermArrays& t, long long slot, int sys, const double4& self)
    {
        s = slot;
        S = &a.sys[sys];
        const GlobalParams& P = S->g[G];
        halfw_hi = PER ? S->halfw_hi : 0x7fffffff;
        pi = self;
        crsq  = P.cutoff_ratio_sq;
        cr    = P.cutoff_ratio;
        kind  = P.kind;
        power = P.power;
        coefc = P.coef_at_cutoff;
        eps   = P.eps;
        eps12 = eps * 12;
        inv_debye = P.inv_debye;
        abs_cut_sq = P.abs_cutoff * P.abs_cutoff;
        qi = pi.w; inv4pi = P.inv4pi;
        slot_p1 = t.slot_p1;
        // second per-slot parameter: LJ-family epsilon, HardCore core radius
        epsi  = (G == G_LJ || (G == G_EXV && kind == EXV_HARD_CORE)) ? t.slot_p1[slot] : 0.0;
        eps12f = (float)eps12; epsf = (float)eps; coefcf = (float)coefc;
        invdf = (float)inv_debye;
        crsqf = (float)crsq; wif = (float)pi.w;
        half = !HALF_RT || t.half != 0;
        fe = !NF && t.fe_energy != 0;
        force = a.force;
        slot_particle = t.slot_particle;
    }

    // The Lennard-Jones family's second parameter of partner q (epsilon):
    // callers request it with the partner's coordinates.
    __device__ __forceinline__ double partner_p1(int q) const {return G == G_LJ ? slot_p1[q] : 0.0;}

    // Half lists (mixed form): the partner's share of the pair, the negated
    // fixed-point components of c r_ij.  Its own evaluation of the pair would
    // take r_ji = -r_ij exactly (an FP64 difference; the minimum image is odd
    // inside the cutoff), the same coefficient (every potential is symmetric
    // in its two parameters, and FP32 sums and products commute) and the same
    // rounding to the grid (round to nearest even is odd), so the integer sum
    // of each particle is the full lists' sum, bit for bit.
    // jp: the partner's particle when the caller has read it with its coordinates
    __device__ __forceinline__ void partner_add(double c, int q, double dx, double dy, double dz, int jp = -1) const
    {
        if constexpr(PREC == P_MIXED && NF && HALF)
        {
            if((HALF_RT && !half) || c == 0.0) {return;}
            const long long x = fx_from_double(c * dx), y = fx_from_double(c * dy), z = fx_from_double(c * dz);
            unsigned long long* f =
                reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + (jp >= 0 ? jp : slot_particle[q]));
            if(x) {atomicAdd(f + 0, (unsigned long long)(-x));}
            if(y) {atomicAdd(f + 1, (unsigned long long)(-y));}
            if(z) {atomicAdd(f + 2, (unsigned long long)(-z));}
        }
    }

    // The same for an FP32 coefficient (Acc::add_c).
    __device__ __forceinline__ void partner_add_c(float c, int q, double dx, double dy, double dz, int jp) const
    {
        if constexpr(PREC == P_MIXED && NF && HALF)
        {
            if((HALF_RT && !half) || c == 0.0f) {return;}
            const double cs = fx_coefficient(c);
            const long long x = fx_product(cs, dx), y = fx_product(cs, dy), z = fx_product(cs, dz);
            unsigned long long* f =
                reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + (jp >= 0 ? jp : slot_particle[q]));
            if(x) {atomicAdd(f + 0, (unsigned long long)(-x));}
            if(y) {atomicAdd(f + 1, (unsigned long long)(-y));}
            if(z) {atomicAdd(f + 2, (unsigned long long)(-z));}
        }
    }

    // WCA, LennardJonesAttractive and UniformLennardJones through the generic
    // pair loop: f = r_ij (f_mag / |r|) with f_mag = potential.derivative(|r|),
    // a pair with f_mag = 0 skipped in the force pass; the energy-only pass
    // (calc_energy) sums potential(|r|) over every listed pair.  Formulas of
    // WCAPotential.hpp:37-58, LennardJonesAttractivePotential.hpp:36-70,
    // UniformLennardJonesPotential.hpp:41-61 (uniform sigma and epsilon are
    // equal per-slot values, which the Lorentz-Berthelot rule keeps as is).
    template<typename T>
    __device__ __forceinline__ static T fam_derivative(int kind, T r, T sigma, T epsilon, T cutoff_ratio)
    {
        if(kind == LJ_WCA)
        {
            if(sigma * T(SIXTH_ROOT_OF_TWO) < r) {return T(0);}
            const T rinv = T(1) / r;
            const T r1s1 = sigma * rinv;
            const T r3s3 = r1s1 * r1s1 * r1s1;
            const T r6s6 = r3s3 * r3s3;
            return T(24) * epsilon * (r6s6 * (T(1) - T(2) * r6s6)) * rinv;
        }
        if(kind == LJ_ATTRACTIVE)
        {
            if(r < sigma * T(SIXTH_ROOT_OF_TWO) || sigma * cutoff_ratio < r) {return T(0);}
            const T rinv = T(1) / r;
            const T sr1 = sigma * rinv;
            const T sr3 = sr1 * sr1 * sr1;
            const T sr6 = sr3 * sr3;
            return T(24) * epsilon * (sr6 - T(2) * sr6 * sr6) * rinv;
        }
        if(sigma * cutoff_ratio < r) {return T(0);}
        const T rinv = T(1) / r;
        const T sr1 = sigma * rinv;
        const T sr3 = sr1 * sr1 * sr1;
        const T sr6 = sr3 * sr3;
        return (epsilon * T(24)) * sr6 * (T(1) - T(2) * sr6) * rinv;
    }
    template<typename T>
    __device__ __forceinline__ static T fam_potential(int kind, T r, T sigma, T epsilon, T cutoff_ratio, T coefc)
    {
        if(kind == LJ_WCA)
        {
            if(sigma * T(SIXTH_ROOT_OF_TWO) < r) {return T(0);}
            const T r1s1 = sigma / r;
            const T r3s3 = r1s1 * r1s1 * r1s1;
            const T r6s6 = r3s3 * r3s3;
            return T(4) * epsilon * (r6s6 * (r6s6 - T(1)) + T(0.25));
        }
        if(kind == LJ_ATTRACTIVE)
        {
            if(r < sigma * T(SIXTH_ROOT_OF_TWO)) {return -epsilon;}
            if(sigma * cutoff_ratio < r) {return T(0);}
            const T sr1 = sigma / r;
            const T sr3 = sr1 * sr1 * sr1;
            const T sr6 = sr3 * sr3;
            return T(4) * epsilon * (sr6 * (sr6 - T(1)) - coefc);
        }
        if(sigma * cutoff_ratio < r) {return T(0);}
        const T sr1 = sigma / r;
        const T sr3 = sr1 * sr1 * sr1;
        const T sr6 = sr3 * sr3;
        return (epsilon * T(4)) * (sr6 * (sr6 - T(1)) - coefc);
    }
    __device__ __forceinline__ void family(int k, double sigma, double epsilon, double l2, double dx,
                                           double dy, double dz, bool count_e, Acc<PREC>& acc,
                                           double& energy, bool& ovf, int q, int jp) const
    {
        using T = typename std::conditional<PREC == P_FP64, double, float>::type;
        if(NF || fe)
        {
            const T rl = PREC == P_FP64 ? T(rsqrt(l2)) : T(rsqrtf((float)l2));
            const T l  = T(l2) * rl;
            const T f_mag = fam_derivative<T>(k, l, T(sigma), T(epsilon), T(cr));
            if(f_mag == T(0)) {return;}
            if(NF) {acc.add((double)(f_mag * rl), dx, dy, dz, ovf); partner_add((double)(f_mag * rl), q, dx, dy, dz, jp);}
            if(count_e) {energy += (double)fam_potential<T>(k, l, T(sigma), T(epsilon), T(cr), T(coefc));}
        }
        else if(count_e)
        {
            const T l = PREC == P_FP64 ? T(sqrt(l2)) : sqrtf((float)l2);
            energy += (double)fam_potential<T>(k, l, T(sigma), T(epsilon), T(cr), T(coefc));
        }
    }

    // InversePower (InversePowerPotential.hpp:38-57; sigma_ij = r_i + r_j)
    // and HardCoreExcludedVolume (HardCoreExcludedVolumePotential.hpp:44-80;
    // sigma_ij = s_i + s_j, R_ij = c_i + c_j) through the generic pair loop
    template<typename T>
    __device__ __forceinline__ T exv_derivative(T r, T sigma, T radius) const
    {
        if(kind == EXV_INVERSE_POWER)
        {
            if(sigma * T(cr) < r) {return T(0);}
            const T rinv = T(1) / r;
            const T d_r = sigma * rinv;
            const T drn = pow(d_r, T(power));
            return T(-power) * T(eps) * drn * rinv;
        }
        if(sigma * T(cr) + radius < r) {return T(0);}
        if(r < radius) {return T(INFINITY);}
        const T gapinv = T(1) / (r - radius);
        const T s1 = sigma * gapinv;
        const T s3 = s1 * s1 * s1;
        const T s6 = s3 * s3;
        return T(-12) * T(eps) * s6 * s6 * gapinv;
    }
    template<typename T>
    __device__ __forceinline__ T exv_potential(T r, T sigma, T radius) const
    {
        if(kind == EXV_INVERSE_POWER)
        {
            if(sigma * T(cr) < r) {return T(0);}
            const T d_r = sigma / r;
            const T drn = pow(d_r, T(power));
            return T(eps) * (drn - T(coefc));
        }
        if(sigma * T(cr) + radius < r) {return T(0);}
        if(r < radius) {return T(INFINITY);}
        const T gap = r - radius;
        const T s1 = sigma / gap;
        const T s3 = s1 * s1 * s1;
        const T s6 = s3 * s3;
        return T(eps) * (s6 * s6 - T(coefc));
    }
    __device__ __forceinline__ void exv_family(double sigma, double radius, double l2, double dx, double dy,
                                               double dz, bool count_e, Acc<PREC>& acc, double& energy,
                                               bool& ovf, int q, int jp) const
    {
        using T = typename std::conditional<PREC == P_FP64, double, float>::type;
        if(NF || fe)
        {
            const T rl = PREC == P_FP64 ? T(rsqrt(l2)) : T(rsqrtf((float)l2));
            const T l  = T(l2) * rl;
            const T f_mag = exv_derivative<T>(l, T(sigma), T(radius));
            if(f_mag == T(0)) {return;}
            if(NF) {acc.add((double)(f_mag * rl), dx, dy, dz, ovf); partner_add((double)(f_mag * rl), q, dx, dy, dz, jp);}
            if(count_e) {energy += (double)exv_potential<T>(l, T(sigma), T(radius));}
        }
        else if(count_e)
        {
            const T l = PREC == P_FP64 ? T(sqrt(l2)) : sqrtf((float)l2);
            energy += (double)exv_potential<T>(l, T(sigma), T(radius));
        }
    }

    // p1j: partner_p1(q)
    __device__ __forceinline__ void operator()(const double4& pj, const double p1j, const int q, Acc<PREC>& acc,
                                               double& energy, bool& ovf, int jp = -1) const
    {
        double dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
        if(PER && image_needed(dx, dy, dz, halfw_hi))
        {
            dx = min_image(dx, S->halfw[0], S->width[0]);
            dy = min_image(dy, S->halfw[1], S->width[1]);
            dz = min_image(dz, S->halfw[2], S->width[2]);
        }
        const double l2 = fma(dz, dz, fma(dy, dy, dx * dx));
        const bool count_e = NE && (s < q);
        if(G == G_EXV)
        {
            if(kind != EXV_PLAIN)
            {
                const double radius = kind == EXV_HARD_CORE ? epsi + slot_p1[q] : 0.0;
                exv_family(pi.w + pj.w, radius, l2, dx, dy, dz, count_e, acc, energy, ovf, q, jp);
                return;
            }
            const double sigma = pi.w + pj.w;
            const double sigma_sq = sigma * sigma;
            const bool in = !(sigma_sq * crsq < l2);
            if constexpr(PREC == P_FP64)
            {
                if(!in) {return;}
                const double rcp = 1.0 / l2;
                const double s2 = sigma_sq * rcp;
                const double s6 = s2 * s2 * s2;
                if(NF) {acc.add(-eps12 * s6 * s6 * rcp, dx, dy, dz, ovf);}
                if(count_e) {energy += eps * (s6 * s6 - coefc);}
            }
            else
            {
                // branch-free: every lane evaluates, pairs outside the
                // cutoff add an exact zero; sigma in FP32 from the two radii
                const float l2f = (float)l2;
                const float rcp = reciprocal(l2f);
                const float sg = wif + (float)pj.w;
                const float s2 = sg * sg * rcp;
                const float s6 = s2 * s2 * s2;
                const float cf = in ? -eps12f * s6 * s6 * rcp : 0.0f;
                if constexpr(NF)
                {
                    acc.add_c(cf, fabsf(cf) * fmaxf(l2f, 1.0f), dx, dy, dz, ovf);
                    partner_add_c(cf, q, dx, dy, dz, jp);
                }
                if(count_e && in) {energy += (double)(epsf * (s6 * s6 - coefcf));}
            }
        }
        else if(G == G_DH)
        {
            const bool in = l2 < abs_cut_sq;
            if constexpr(PREC == P_FP64)
            {
                if(!in) {return;}
                const double qq = (qi * pj.w) * inv4pi;     // symmetric in i, j
                const double rl = rsqrt(l2);
                const double l  = l2 * rl;
                const double ex = exp(-l * inv_debye);
                if(NF) {acc.add(-qq * fma(l, inv_debye, 1.0) * (rl * rl) * ex * rl, dx, dy, dz, ovf);}
                if(count_e) {energy += qq * (ex / l - coefc);}
            }
            else
            {
                // branch-free like ExcludedVolume: outside the cutoff the
                // force is zero; (debye + l) / debye = 1 + l / debye;
                // the charge product stays in FP64 and scales the FP32
                // coefficient of the unit-charge potential
                const double qq = (qi * pj.w) * inv4pi;
                const float l2f = (float)l2;
                const float rl = rsqrt_approx(l2f);
                const float l  = l2f * rl;
                const float ex = exp2_approx(__fmul_rn(l, invdf) * -1.4426950408889634f);
                // an explicit product-sum: every kernel must round alike
                const float cu = in ? -fmaf(l, invdf, 1.0f) * (rl * rl) * rl * ex : 0.0f;
                if constexpr(NF)
                {
                    const float cf = (float)qq * cu;
                    acc.add_c(cf, fabsf(cf) * l, dx, dy, dz, ovf);
                    partner_add_c(cf, q, dx, dy, dz, jp);
                }
                if(count_e && in) {energy += qq * (double)(ex * rl - coefcf);}
            }
        }
        else   // G_LJ
        {
            const double sigma = (pi.w + pj.w) / 2;
            const double epsj = p1j;
            const double epsilon = (epsi == epsj) ? epsi : sqrt(epsi * epsj);
            if(kind != LJ_PLAIN)
            {
                family(kind, sigma, epsilon, l2, dx, dy, dz, count_e, acc, energy, ovf, q, jp);
                return;
            }
            const double sigma_sq = sigma * sigma;
            if(sigma_sq * crsq < l2) {return;}
            if constexpr(PREC == P_FP64)
            {
                const double rcp = 1.0 / l2;
                const double s2 = sigma_sq * rcp;
                const double s6 = s2 * s2 * s2;
                if(NF) {acc.add(24 * epsilon * (s6 - 2 * s6 * s6) * rcp, dx, dy, dz, ovf);}
                if(count_e) {energy += 4 * epsilon * (s6 * s6 - s6 - coefc);}
            }
            else
            {
                const float l2f = (float)l2;
                const float rcp = reciprocal(l2f);
                const float s2 = (float)sigma_sq * rcp;
                const float s6 = s2 * s2 * s2;
                const float ef = (float)epsilon;
                if constexpr(NF)
                {
                    const float cf = 24.0f * ef * fmaf(-2.0f * s6, s6, s6) * rcp;
                    acc.add_c(cf, fabsf(cf) * fmaxf(l2f, 1.0f), dx, dy, dz, ovf);
                    partner_add_c(cf, q, dx, dy, dz, jp);
                }
                if(count_e) {energy += (double)(4.0f * ef * (s6 * s6 - s6 - coefcf));}
            }
        }
    }
};

// A slot's system and the number of partners its force launch walks (0 in a
// frozen system, which keeps its forces): the two loads are independent, the
// system's flag is read once they arrive, and only when the arena has a
// frozen system.
struct SlotHead {
    int sys;
    int n;
};
__device__ __forceinline__ SlotHead slot_head(const Arena& a, const TermArrays& t, long long s)
{
    const int sys = t.slot_sys[s];
    const int n = t.nnb[s];
    return {sys, a.any_frozen && a.sys[sys].frozen ? 0 : n};
}

}  // namespace mjg
