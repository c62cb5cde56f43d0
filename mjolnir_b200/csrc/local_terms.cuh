// The bonded terms' formulas and force accumulators, shared by the bonded
// launch (local.cu) and the multi-step kernel of small arenas (run.cu).
#pragma once
#include "kernels.cuh"

namespace mjg {

// Forces of one block's terms are summed in shared memory over a window of
// WINDOW particles starting at the block's first particle (bonds, angles and
// dihedrals of a chain touch a narrow index range), then added to global
// memory once per particle; a particle outside the window goes to global
// memory directly.
constexpr int SEG = 256;              // particles owned by one block (window start)
constexpr int HALO = 64;              // terms may reach this far past the window
constexpr int WINDOW = SEG + HALO;

// FP64 sums in the plain form.  The mixed form's 64-bit integer sums are kept as
// two 32-bit words each: shared memory adds 32-bit words in one instruction and
// 64-bit ones in a compare-and-swap loop.  The low word's add returns what it
// found, which gives the carry, and the high word is touched only where it
// changes.
template<int PREC> struct WinT;
template<> struct WinT<P_FP64>  {using type = double; static constexpr int words = 1;};
template<> struct WinT<P_MIXED> {using type = unsigned; static constexpr int words = 2;};

template<int PREC>
struct Window {
    using T = typename WinT<PREC>::type;
    static constexpr int SIZE = 3 * WINDOW * WinT<PREC>::words;
    T* w;         // [SIZE] in shared memory; mixed: low words, then high words
    int base;
    __device__ __forceinline__ void add64(int k, long long v)
    {
        unsigned* lo = reinterpret_cast<unsigned*>(w) + k;
        const unsigned l = (unsigned)v;
        const unsigned old = atomicAdd(lo, l);
        const unsigned h = (unsigned)((unsigned long long)v >> 32) + (old + l < l ? 1u : 0u);
        if(h) {atomicAdd(lo + 3 * WINDOW, h);}
    }
    __device__ __forceinline__ void add(void* force, int i, double fx, double fy, double fz)
    {
        const int k = i - base;
        if(k >= 0 && k < WINDOW)
        {
            if(PREC == P_FP64)
            {
                atomicAdd(reinterpret_cast<double*>(w) + 3 * k + 0, fx);
                atomicAdd(reinterpret_cast<double*>(w) + 3 * k + 1, fy);
                atomicAdd(reinterpret_cast<double*>(w) + 3 * k + 2, fz);
            }
            else
            {
                add64(3 * k + 0, fx_from_double(fx));
                add64(3 * k + 1, fx_from_double(fy));
                add64(3 * k + 2, fx_from_double(fz));
            }
            return;
        }
        global_add(force, i, fx, fy, fz);
    }
    // mixed form: a sum of shares already on the grid
    __device__ __forceinline__ void add_fx(void* force, int i, long long x, long long y, long long z)
    {
        const int k = i - base;
        if(k >= 0 && k < WINDOW)
        {
            add64(3 * k + 0, x);
            add64(3 * k + 1, y);
            add64(3 * k + 2, z);
            return;
        }
        global_add_fx(force, i, x, y, z);
    }
    __device__ __forceinline__ static void global_add_fx(void* force, int i, long long x, long long y, long long z)
    {
        unsigned long long* f = reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + i);
        atomicAdd(f + 0, (unsigned long long)x);
        atomicAdd(f + 1, (unsigned long long)y);
        atomicAdd(f + 2, (unsigned long long)z);
    }
    __device__ __forceinline__ static void global_add(void* force, int i, double fx, double fy, double fz)
    {
        if(PREC == P_FP64)
        {
            double* f = reinterpret_cast<double*>(static_cast<double4*>(force) + i);
            atomicAdd(f + 0, fx); atomicAdd(f + 1, fy); atomicAdd(f + 2, fz);
        }
        else
        {
            unsigned long long* f = reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + i);
            atomicAdd(f + 0, (unsigned long long)fx_from_double(fx));
            atomicAdd(f + 1, (unsigned long long)fx_from_double(fy));
            atomicAdd(f + 2, (unsigned long long)fx_from_double(fz));
        }
    }
    __device__ __forceinline__ void flush(void* force, long long n) const
    {
        for(int k = threadIdx.x; k < WINDOW; k += blockDim.x)
        {
            const long long i = (long long)base + k;
            if(i >= n) {break;}
            if(PREC == P_FP64)
            {
                const double* v = reinterpret_cast<const double*>(w) + 3 * k;
                if(v[0] == 0.0 && v[1] == 0.0 && v[2] == 0.0) {continue;}
                double* f = reinterpret_cast<double*>(static_cast<double4*>(force) + i);
                atomicAdd(f + 0, v[0]); atomicAdd(f + 1, v[1]); atomicAdd(f + 2, v[2]);
            }
            else
            {
                const unsigned* v = reinterpret_cast<const unsigned*>(w) + 3 * k;
                unsigned long long* f = reinterpret_cast<unsigned long long*>(static_cast<longlong4*>(force) + i);
#pragma unroll
                for(int c = 0; c < 3; ++c)
                {
                    const unsigned long long x = (unsigned long long)v[3 * WINDOW + c] << 32 | v[c];
                    if(x) {atomicAdd(f + c, x);}
                }
            }
        }
    }
};

__device__ __forceinline__ double3 direction(const SysDev& S, const double4& from, const double4& to)
{
    double3 d = make_double3(to.x - from.x, to.y - from.y, to.z - from.z);
    if(image_needed(d.x, d.y, d.z, S.halfw_hi))
    {
        d.x = min_image(d.x, S.halfw[0], S.width[0]);
        d.y = min_image(d.y, S.halfw[1], S.width[1]);
        d.z = min_image(d.z, S.halfw[2], S.width[2]);
    }
    return d;
}
// Products and sums are joined explicitly below: the joined records and the
// separate terms must round alike, and the compiler joins them differently from
// kernel to kernel.
__device__ __forceinline__ double dot(double3 a, double3 b) {return fma(a.z, b.z, fma(a.y, b.y, __dmul_rn(a.x, b.x)));}
__device__ __forceinline__ double3 cross(double3 a, double3 b)
{
    return make_double3(fma(a.y, b.z, -__dmul_rn(a.z, b.y)), fma(a.z, b.x, -__dmul_rn(a.x, b.z)), fma(a.x, b.y, -__dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double clamp1(double x) {return fmin(fmax(x, -1.0), 1.0);}

__device__ __forceinline__ void reduce_energy(const Arena& a, int sys, bool active, double e, int term)
{
    const unsigned full = 0xffffffffu;
    const int s0 = __shfl_sync(full, sys, 0);
    const bool uniform = __all_sync(full, !active || sys == s0);
    if(uniform)
    {
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) {e += __shfl_xor_sync(full, e, o);}
        if(__any_sync(full, active) && (threadIdx.x & 31) == 0) {atomicAdd(&a.sys[s0].energy[term], e);}
    }
    else if(active)
    {
        atomicAdd(&a.sys[sys].energy[term], e);
    }
}

template<int PREC, bool NF, bool NE, class ACC>
__device__ __forceinline__ void do_bond(const Arena& a, const LocalArrays& l, long long b, bool active,
                                         ACC& W)
{
    const int sys = active ? l.bond_sys[b] : 0;
    double e = 0.0;
    if(active)
    {
        const SysDev& S = a.sys[sys];
        const int i0 = l.bond_idx[2 * b], i1 = l.bond_idx[2 * b + 1];
        const double k = l.bond_k[b], v0 = l.bond_v0[b];
        const double3 d = direction(S, a.pos[i0], a.pos[i1]);      // r1 - r0
        const double len2 = dot(d, d);
        const double rlen = rsqrt(len2);
        const double len  = len2 * rlen;
        const double dv   = len - v0;
        if(NE) {e = k * dv * dv;}
        if(NF)
        {
            const double c = -(2 * k * dv) * rlen;
            W.add(a.force, i0, -d.x * c, -d.y * c, -d.z * c);
            W.add(a.force, i1,  d.x * c,  d.y * c,  d.z * c);
        }
    }
    if(NE) {reduce_energy(a, sys, active, e, T_BOND);}
}

// the reference's formulas for one (active) angle: adds its forces, returns
// its energy (NE)
template<int PREC, bool NF, bool NE, class ACC>
__device__ __forceinline__ double angle_fp64(const Arena& a, const LocalArrays& l, long long b, ACC& W)
{
    double e = 0.0;
    const SysDev& S = a.sys[l.angle_sys[b]];
    {
        const int i0 = l.angle_idx[3 * b], i1 = l.angle_idx[3 * b + 1], i2 = l.angle_idx[3 * b + 2];
        const double k = l.angle_k[b], v0 = l.angle_v0[b];
        const double4 p1 = a.pos[i1];
        const double3 r_ij = direction(S, p1, a.pos[i0]);
        const double3 r_kj = direction(S, p1, a.pos[i2]);
        const double inv_ij = rsqrt(dot(r_ij, r_ij));
        const double inv_kj = rsqrt(dot(r_kj, r_kj));
        const double3 eij = make_double3(r_ij.x * inv_ij, r_ij.y * inv_ij, r_ij.z * inv_ij);
        const double3 ekj = make_double3(r_kj.x * inv_kj, r_kj.y * inv_kj, r_kj.z * inv_kj);
        const double cos_t = clamp1(dot(eij, ekj));
        const double theta = acos(cos_t);
        const double dv = theta - v0;
        if(NE) {e = k * dv * dv;}
        if(NF)
        {
            const double coef = -(2 * k * dv);
            const double sin_t = sin(theta);
            const double cis = coef / fmax(sin_t, 1e-8);          // math/constants.hpp:26
            const double ci = cis * inv_ij, ck = cis * inv_kj;
            const double3 Fi = make_double3(ci * fma(cos_t, eij.x, -ekj.x), ci * fma(cos_t, eij.y, -ekj.y), ci * fma(cos_t, eij.z, -ekj.z));
            const double3 Fk = make_double3(ck * fma(cos_t, ekj.x, -eij.x), ck * fma(cos_t, ekj.y, -eij.y), ck * fma(cos_t, ekj.z, -eij.z));
            W.add(a.force, i0, Fi.x, Fi.y, Fi.z);
            W.add(a.force, i1, -Fi.x - Fk.x, -Fi.y - Fk.y, -Fi.z - Fk.z);
            W.add(a.force, i2, Fk.x, Fk.y, Fk.z);
        }
    }
    return e;
}

template<int PREC, bool NF, bool NE, class ACC>
__device__ __forceinline__ void do_angle(const Arena& a, const LocalArrays& l, long long b, bool active,
                                         ACC& W)
{
    const int sys = active ? l.angle_sys[b] : 0;
    const double e = active ? angle_fp64<PREC, NF, NE>(a, l, b, W) : 0.0;
    if(NE) {reduce_energy(a, sys, active, e, T_ANGLE);}
}

// the reference's formulas for one (active) dihedral: adds its forces,
// returns its energy (NE)
template<int PREC, bool NF, bool NE, class ACC>
__device__ __forceinline__ double dihedral_fp64(const Arena& a, const LocalArrays& l, long long b, ACC& W)
{
    double e = 0.0;
    const SysDev& S = a.sys[l.dihd_sys[b]];
    {
        const int i0 = l.dihd_idx[4 * b], i1 = l.dihd_idx[4 * b + 1];
        const int i2 = l.dihd_idx[4 * b + 2], i3 = l.dihd_idx[4 * b + 3];
        const double K = l.dihd_k[b], v0 = l.dihd_v0[b];
        const double nn = (double)l.dihd_n[b];
        const double4 rj = a.pos[i1], rk = a.pos[i2];
        const double3 r_ij = direction(S, rj, a.pos[i0]);
        const double3 r_kj = direction(S, rj, rk);
        const double3 r_lk = direction(S, rk, a.pos[i3]);
        const double3 r_kl = make_double3(-r_lk.x, -r_lk.y, -r_lk.z);
        const double r_kj_lensq  = dot(r_kj, r_kj);
        const double r_kj_rlen   = rsqrt(r_kj_lensq);
        const double r_kj_rlensq = r_kj_rlen * r_kj_rlen;
        const double r_kj_len    = r_kj_rlen * r_kj_lensq;
        const double3 m = cross(r_ij, r_kj);
        const double3 n = cross(r_kj, r_kl);
        const double m_lensq = dot(m, m);
        const double n_lensq = dot(n, n);
        const double cos_phi = clamp1(dot(m, n) * rsqrt(m_lensq * n_lensq));
        const double phi = copysign(acos(cos_phi), dot(r_ij, n));
        const double dv = phi - v0;
        if(NE) {e = K * (1 + cos(nn * dv));}
        if(NF)
        {
            const double coef = K * nn * sin(nn * dv);                // -dV/dphi
            const double cfi =  coef * r_kj_len / m_lensq;
            const double cfl = -coef * r_kj_len / n_lensq;
            const double3 Fi = make_double3(cfi * m.x, cfi * m.y, cfi * m.z);
            const double3 Fl = make_double3(cfl * n.x, cfl * n.y, cfl * n.z);
            const double cijk = dot(r_ij, r_kj) * r_kj_rlensq;
            const double cjkl = dot(r_kl, r_kj) * r_kj_rlensq;
            W.add(a.force, i0, Fi.x, Fi.y, Fi.z);
            W.add(a.force, i1, fma(cijk - 1.0, Fi.x, -__dmul_rn(cjkl, Fl.x)), fma(cijk - 1.0, Fi.y, -__dmul_rn(cjkl, Fl.y)),
                            fma(cijk - 1.0, Fi.z, -__dmul_rn(cjkl, Fl.z)));
            W.add(a.force, i2, fma(cjkl - 1.0, Fl.x, -__dmul_rn(cijk, Fi.x)), fma(cjkl - 1.0, Fl.y, -__dmul_rn(cijk, Fi.y)),
                            fma(cjkl - 1.0, Fl.z, -__dmul_rn(cijk, Fi.z)));
            W.add(a.force, i3, Fl.x, Fl.y, Fl.z);
        }
    }
    return e;
}

template<int PREC, bool NF, bool NE, class ACC>
__device__ __forceinline__ void do_dihedral(const Arena& a, const LocalArrays& l, long long b, bool active,
                                         ACC& W)
{
    const int sys = active ? l.dihd_sys[b] : 0;
    const double e = active ? dihedral_fp64<PREC, NF, NE>(a, l, b, W) : 0.0;
    if(NE) {reduce_energy(a, sys, active, e, T_DIHEDRAL);}
}

// ----------------------------------------------------------- mixed form
// sin of a bond angle below which an angle or dihedral is evaluated with the
// FP64 formulas instead (ill-conditioned in FP32)
constexpr float ILL_SIN = 0.2f;
// The same terms in FP32 from FP64 displacements: bond stretch via
// (r^2 - v0^2) / (r + v0) with r^2 - v0^2 in FP64, the angle from atan2 of the
// cross and dot products, the dihedral from (cos phi, sin phi) of the normals
// (phi = atan2(|r_kj| r_ij.n, m.n) has the reference's sign convention) and
// cos / sin of n (phi - v0) by the multiple-angle recurrence, so no FP64
// transcendental is evaluated.  Parameters come pre-packed as floats.

__device__ __forceinline__ float3 fdir(const SysDev& S, const double4& from, const double4& to)
{
    const double3 d = direction(S, from, to);
    return make_float3((float)d.x, (float)d.y, (float)d.z);
}
__device__ __forceinline__ float fdot(float3 a, float3 b) {return fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x)));}
__device__ __forceinline__ float3 fcross(float3 a, float3 b)
{
    return make_float3(fmaf(a.y, b.z, -__fmul_rn(a.z, b.y)), fmaf(a.z, b.x, -__fmul_rn(a.x, b.z)), fmaf(a.x, b.y, -__fmul_rn(a.y, b.x)));
}

// minus dV/dr over r of a bond of squared length len2
__device__ __forceinline__ double bond_coefficient(double len2, const float2& kv)
{
    const float lenf = sqrtf((float)len2);
    const float dv = (float)(len2 - (double)kv.y * (double)kv.y) / (lenf + kv.y);
    return (double)(-(2.0f * kv.x * dv) / lenf);
}

// Angle and dihedral forces from FP32 displacements; forces() returns false
// where the geometry needs the FP64 formulas (ILL_SIN).
struct AngleF32 {
    double3 fi, fk;
    __device__ __forceinline__ bool forces(const float3& rij, const float3& rkj, const float2& kv)
    {
        const float inv_ij = rsqrtf(fdot(rij, rij));
        const float inv_kj = rsqrtf(fdot(rkj, rkj));
        const float3 eij = make_float3(rij.x * inv_ij, rij.y * inv_ij, rij.z * inv_ij);
        const float3 ekj = make_float3(rkj.x * inv_kj, rkj.y * inv_kj, rkj.z * inv_kj);
        const float3 cr = fcross(eij, ekj);
        const float sin_t = sqrtf(fdot(cr, cr));
        // within 11.5 degrees of collinear the FP32 cross products and
        // differences of unit vectors lose the force
        if(sin_t < ILL_SIN) {return false;}
        const float cos_t = fdot(eij, ekj);
        const float theta = atan2f(sin_t, cos_t);
        const float dv = theta - kv.y;
        const float cis = -(2.0f * kv.x * dv) / fmaxf(sin_t, 1e-8f);
        const float ci = cis * inv_ij, ck = cis * inv_kj;
        const float cc = fminf(fmaxf(cos_t, -1.0f), 1.0f);
        fi = make_double3(ci * fmaf(cc, eij.x, -ekj.x), ci * fmaf(cc, eij.y, -ekj.y), ci * fmaf(cc, eij.z, -ekj.z));
        fk = make_double3(ck * fmaf(cc, ekj.x, -eij.x), ck * fmaf(cc, ekj.y, -eij.y), ck * fmaf(cc, ekj.z, -eij.z));
        return true;
    }
};

struct DihedralF32 {
    float3 f0, f1, f2, f3;
    // p: {k, cos(n v0), sin(n v0), n}
    __device__ __forceinline__ bool forces(const float3& r_ij, const float3& r_kj, const float3& r_kl, const float4& p)
    {
        const int nn = (int)p.w;
        const float r_kj_lensq  = fdot(r_kj, r_kj);
        const float r_kj_rlen   = rsqrtf(r_kj_lensq);
        const float r_kj_len    = r_kj_rlen * r_kj_lensq;
        const float3 m = fcross(r_ij, r_kj);
        const float3 n = fcross(r_kj, r_kl);
        const float m_lensq = fdot(m, m);
        const float n_lensq = fdot(n, n);
        // a bond angle of the dihedral within 11.5 degrees of collinear: the
        // normals m, n lose their direction in FP32
        if(m_lensq < ILL_SIN * ILL_SIN * fdot(r_ij, r_ij) * r_kj_lensq ||
           n_lensq < ILL_SIN * ILL_SIN * fdot(r_kl, r_kl) * r_kj_lensq)
        {
            return false;
        }
        // (cos phi, sin phi) of the reference's phi = copysign(acos(m.n), r_ij.n)
        const float x = fdot(m, n);
        const float y = r_kj_len * fdot(r_ij, n);
        const float h = rsqrtf(fmaf(y, y, __fmul_rn(x, x)));
        const float c1 = x * h, s1 = y * h;
        float cn = 1.0f, sn = 0.0f;
        const int na = nn < 0 ? -nn : nn;
        for(int q = 0; q < na; ++q)
        {
            const float c2 = fmaf(cn, c1, -__fmul_rn(sn, s1));
            sn = fmaf(sn, c1, __fmul_rn(cn, s1));
            cn = c2;
        }
        if(nn < 0) {sn = -sn;}
        const float sd = fmaf(sn, p.y, -__fmul_rn(cn, p.z));           // sin of n (phi - v0)
        const float coef = p.x * (float)nn * sd;         // -dV/dphi
        const float cfi =  coef * r_kj_len / m_lensq;
        const float cfl = -coef * r_kj_len / n_lensq;
        f0 = make_float3(cfi * m.x, cfi * m.y, cfi * m.z);
        f3 = make_float3(cfl * n.x, cfl * n.y, cfl * n.z);
        const float rl2 = r_kj_rlen * r_kj_rlen;
        const float cijk = fdot(r_ij, r_kj) * rl2;
        const float cjkl = fdot(r_kl, r_kj) * rl2;
        f1 = make_float3(fmaf(cijk - 1.0f, f0.x, -__fmul_rn(cjkl, f3.x)), fmaf(cijk - 1.0f, f0.y, -__fmul_rn(cjkl, f3.y)),
                         fmaf(cijk - 1.0f, f0.z, -__fmul_rn(cjkl, f3.z)));
        f2 = make_float3(fmaf(cjkl - 1.0f, f3.x, -__fmul_rn(cijk, f0.x)), fmaf(cjkl - 1.0f, f3.y, -__fmul_rn(cijk, f0.y)),
                         fmaf(cjkl - 1.0f, f3.z, -__fmul_rn(cijk, f0.z)));
        return true;
    }
};

// one term of the mixed form by itself
template<class ACC>
__device__ __forceinline__ void do_bond_f32(const Arena& a, const LocalArrays& l, long long b, ACC& W)
{
    const SysDev& S = a.sys[l.bond_sys[b]];
    const int i0 = l.bond_idx[2 * b], i1 = l.bond_idx[2 * b + 1];
    const double3 d = direction(S, a.pos[i0], a.pos[i1]);
    const double c = bond_coefficient(dot(d, d), l.bond_kv[b]);
    W.add(a.force, i0, -d.x * c, -d.y * c, -d.z * c);
    W.add(a.force, i1,  d.x * c,  d.y * c,  d.z * c);
}

template<class ACC>
__device__ __forceinline__ void do_angle_f32(const Arena& a, const LocalArrays& l, long long b, ACC& W)
{
    const SysDev& S = a.sys[l.angle_sys[b]];
    const int i0 = l.angle_idx[3 * b], i1 = l.angle_idx[3 * b + 1], i2 = l.angle_idx[3 * b + 2];
    const double4 p1 = a.pos[i1];
    AngleF32 A;
    if(!A.forces(fdir(S, p1, a.pos[i0]), fdir(S, p1, a.pos[i2]), l.angle_kv[b]))
    {
        angle_fp64<P_MIXED, true, false>(a, l, b, W);
        return;
    }
    W.add(a.force, i0, A.fi.x, A.fi.y, A.fi.z);
    W.add(a.force, i1, -A.fi.x - A.fk.x, -A.fi.y - A.fk.y, -A.fi.z - A.fk.z);
    W.add(a.force, i2, A.fk.x, A.fk.y, A.fk.z);
}

template<class ACC>
__device__ __forceinline__ void do_dihedral_f32(const Arena& a, const LocalArrays& l, long long b, ACC& W)
{
    const SysDev& S = a.sys[l.dihd_sys[b]];
    const int i0 = l.dihd_idx[4 * b], i1 = l.dihd_idx[4 * b + 1];
    const int i2 = l.dihd_idx[4 * b + 2], i3 = l.dihd_idx[4 * b + 3];
    const double4 rj = a.pos[i1], rk = a.pos[i2];
    const float3 r_lk = fdir(S, rk, a.pos[i3]);
    DihedralF32 D;
    if(!D.forces(fdir(S, rj, a.pos[i0]), fdir(S, rj, rk), make_float3(-r_lk.x, -r_lk.y, -r_lk.z), l.dihd_p[b]))
    {
        dihedral_fp64<P_MIXED, true, false>(a, l, b, W);
        return;
    }
    W.add(a.force, i0, D.f0.x, D.f0.y, D.f0.z);
    W.add(a.force, i1, D.f1.x, D.f1.y, D.f1.z);
    W.add(a.force, i2, D.f2.x, D.f2.y, D.f2.z);
    W.add(a.force, i3, D.f3.x, D.f3.y, D.f3.z);
}

// ----------------------------------------------------------- joined terms
// A bead chain's bond (i, i+1), angle (i, i+1, i+2) and dihedral (i .. i+3)
// share their leading particles.  A record joins the terms whose particles are
// prefixes of one another (built at commit; a term that joins none is a record
// of its own), so that a step loads four positions instead of nine, takes three
// displacements instead of six, and adds one sum per particle (4) instead of one
// per term and particle (9).  Each term's share is rounded to the fixed-point
// grid by itself and the integers are summed, so the forces are those of the
// separate terms bit for bit.
struct Fx3 {
    long long x = 0, y = 0, z = 0;
    __device__ __forceinline__ void add(double fx, double fy, double fz)
    {
        x += fx_from_double(fx); y += fx_from_double(fy); z += fx_from_double(fz);
    }
};

template<class ACC>
__device__ __forceinline__ void record_mixed(const Arena& a, const LocalArrays& l, const int4& idx, const int4& term, ACC& W)
{
    const SysDev& S = a.sys[term.x];
    // all loads of the record, then the arithmetic
    const double4 p0 = a.pos[idx.x], p1 = a.pos[idx.y];
    const double4 p2 = idx.z >= 0 ? a.pos[idx.z] : p1, p3 = idx.w >= 0 ? a.pos[idx.w] : p1;
    const float2 bkv = term.y >= 0 ? l.bond_kv[term.y] : make_float2(0.0f, 1.0f);
    const float2 akv = term.z >= 0 ? l.angle_kv[term.z] : make_float2(0.0f, 1.0f);
    const float4 dp = term.w >= 0 ? l.dihd_p[term.w] : make_float4(0.0f, 1.0f, 0.0f, 0.0f);
    const double3 d10 = direction(S, p1, p0);
    const float3 r_ij = make_float3((float)d10.x, (float)d10.y, (float)d10.z);
    const float3 r_kj = fdir(S, p1, p2);
    Fx3 f0, f1, f2;
    if(term.w >= 0)
    {
        const float3 r_lk = fdir(S, p2, p3);
        const float3 r_kl = make_float3(-r_lk.x, -r_lk.y, -r_lk.z);
        DihedralF32 D;
        if(!D.forces(r_ij, r_kj, r_kl, dp))
        {
            if constexpr(ACC::DEFER) {W.defer_dihedral(term.w);}
            else                     {dihedral_fp64<P_MIXED, true, false>(a, l, term.w, W);}
        }
        else
        {
            f0.add(D.f0.x, D.f0.y, D.f0.z);
            f1.add(D.f1.x, D.f1.y, D.f1.z);
            f2.add(D.f2.x, D.f2.y, D.f2.z);
            Fx3 f3;
            f3.add(D.f3.x, D.f3.y, D.f3.z);
            W.add_fx(a.force, idx.w, f3.x, f3.y, f3.z);
        }
    }
    if(term.z >= 0)
    {
        AngleF32 A;
        if(!A.forces(r_ij, r_kj, akv))
        {
            if constexpr(ACC::DEFER) {W.defer_angle(term.z);}
            else                     {angle_fp64<P_MIXED, true, false>(a, l, term.z, W);}
        }
        else
        {
            f0.add(A.fi.x, A.fi.y, A.fi.z);
            f1.add(-A.fi.x - A.fk.x, -A.fi.y - A.fk.y, -A.fi.z - A.fk.z);
            f2.add(A.fk.x, A.fk.y, A.fk.z);
        }
    }
    if(idx.z >= 0) {W.add_fx(a.force, idx.z, f2.x, f2.y, f2.z);}
    if(term.y >= 0)
    {
        double3 d = make_double3(-d10.x, -d10.y, -d10.z);
        // a component of exactly half a box: its minimum image is -half a box
        // from either end, not the negated other one
        if(image_needed(d.x, d.y, d.z, S.halfw_hi)) {d = direction(S, a.pos[idx.x], a.pos[idx.y]);}
        const double c = bond_coefficient(dot(d, d), bkv);
        f0.add(-d.x * c, -d.y * c, -d.z * c);
        f1.add(d.x * c, d.y * c, d.z * c);
    }
    W.add_fx(a.force, idx.x, f0.x, f0.y, f0.z);
    W.add_fx(a.force, idx.y, f1.x, f1.y, f1.z);
}

// the forces of record r (mixed form)
template<class ACC>
__device__ __forceinline__ void do_record(const Arena& a, const LocalArrays& l, long long r, ACC& W)
{
    const int4 idx = l.rec_idx[r], term = l.rec_term[r];
    if(a.any_frozen && a.sys[term.x].frozen) {return;}
    record_mixed(a, l, idx, term, W);
}

}  // namespace mjg
