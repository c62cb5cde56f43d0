// One particle's share of an integrator step, shared by the integrator
// launches (integrate.cu) and the multi-step kernel of small arenas (run.cu).
#pragma once
#include "kernels.cuh"

namespace mjg {

template<int PREC>
__device__ __forceinline__ void load_force(const void* force, long long i, double& fx, double& fy, double& fz)
{
    if(PREC == P_FP64)
    {
        const double4 f = static_cast<const double4*>(force)[i];
        fx = f.x; fy = f.y; fz = f.z;
    }
    else
    {
        const longlong4 f = static_cast<const longlong4*>(force)[i];
        fx = fx_to_double(f.x); fy = fx_to_double(f.y); fz = fx_to_double(f.z);
    }
}

template<int PREC>
__device__ __forceinline__ void zero_force(void* force, long long i)
{
    if(PREC == P_FP64) {static_cast<double4*>(force)[i] = make_double4(0, 0, 0, 0);}
    else               {static_cast<longlong4*>(force)[i] = make_longlong4(0, 0, 0, 0);}
}

// The closing half of an UnderdampedLangevin step
// (core/UnderdampedLangevinIntegrator.hpp:252-264): a = f/m + sigma R with the
// noise of counter `ctr`, v += halfdt (1 - gamma halfdt) a.
__device__ __forceinline__ void underdamped_close(const SysDev& S, long long i, double4& v, double4& acc,
                                                  const double4& c, double fx, double fy, double fz,
                                                  unsigned long long ctr)
{
    double r0, r1, r2;
    gaussian3(S.seed, (unsigned long long)(i - S.off), ctr, r0, r1, r2);
    acc.x = __dadd_rn(__dmul_rn(fx, c.x), __dmul_rn(r0, c.z));
    acc.y = __dadd_rn(__dmul_rn(fy, c.x), __dmul_rn(r1, c.z));
    acc.z = __dadd_rn(__dmul_rn(fz, c.x), __dmul_rn(r2, c.z));
    const double halfdt = c.w / 2;
    const double k = __dmul_rn(halfdt, __dsub_rn(1.0, __dmul_rn(c.y, halfdt)));
    v.x = __dadd_rn(v.x, __dmul_rn(k, acc.x));
    v.y = __dadd_rn(v.y, __dmul_rn(k, acc.y));
    v.z = __dadd_rn(v.z, __dmul_rn(k, acc.z));
}

// B-A-O-A of BAOAB (or the first half-kick and drift of velocity Verlet, or
// the first half of an UnderdampedLangevin or G-JF step) of particle i of
// system S at the system's step counter `step`, the refresh of its slot
// coordinates and its force reset; returns its squared displacement.  kick:
// the previous step's closing half is applied first, as separate rounding
// steps, so that consecutive steps of a chunk share one pass.  noise(r0, r1,
// r2) gives the particle's three deviates of this step, force(fx, fy, fz) its
// force.  AUX: the arena holds UnderdampedLangevin or G-JF systems (their
// branches cost registers, and occupancy, in the BAOAB / velocity-Verlet arenas
// that have none).
template<int PREC, bool AUX, class NOISE, class FORCE>
__device__ __forceinline__ double advance_particle(const Arena& a, SysDev& S, long long i, bool kick,
                                                   unsigned long long step, NOISE&& noise, FORCE&& force)
{
    double4 p = a.pos[i];
    double4 v = a.vel[i];
    const double4 c = S.uniform_coef ? S.coef : a.coef[i];     // per integrator: see Arena::coef
    double fx, fy, fz;
    force(fx, fy, fz);
    // the particle's slots and their parameters, requested with its state
    int so[NGLOBAL];
    double sw[NGLOBAL];
#pragma unroll
    for(int g = 0; g < NGLOBAL; ++g)
    {
        so[g] = -1;
        if(a.slot_of[g]) {so[g] = a.slot_of[g][i]; sw[g] = a.slot_w[g][i];}
    }
    const bool uld = AUX && S.integrator == I_UNDERDAMPED;
    if(kick && !uld)
    {
        v.x = __dadd_rn(v.x, __dmul_rn(c.x, fx));
        v.y = __dadd_rn(v.y, __dmul_rn(c.x, fy));
        v.z = __dadd_rn(v.z, __dmul_rn(c.x, fz));
    }
    double dx, dy, dz;
    double4 pn = p;     // g-BAOAB: the new position, moved by its two half drifts
    bool direct = false;
    if(uld)             // core/UnderdampedLangevinIntegrator.hpp:198-221
    {
        double4 acc = a.accel[i];
        if(kick) {underdamped_close(S, i, v, acc, c, fx, fy, fz, step); a.accel[i] = acc;}
        const double dt = c.w, halfdt = dt / 2, halfdt2 = dt * dt / 2;
        const double gdo2 = __dmul_rn(c.y, halfdt);                 // gamma dt / 2
        const double omg  = __dsub_rn(1.0, gdo2);
        const double cv   = __dmul_rn(dt, omg);
        dx = __dadd_rn(__dmul_rn(cv, v.x), __dmul_rn(halfdt2, acc.x));
        dy = __dadd_rn(__dmul_rn(cv, v.y), __dmul_rn(halfdt2, acc.y));
        dz = __dadd_rn(__dmul_rn(cv, v.z), __dmul_rn(halfdt2, acc.z));
        const double sv = __dmul_rn(omg, __dadd_rn(__dmul_rn(omg, omg), gdo2));
        v.x = __dmul_rn(v.x, sv);
        v.y = __dmul_rn(v.y, sv);
        v.z = __dmul_rn(v.z, sv);
        const double sa = __dmul_rn(halfdt, omg);
        v.x = __dadd_rn(v.x, __dmul_rn(sa, acc.x));
        v.y = __dadd_rn(v.y, __dmul_rn(sa, acc.y));
        v.z = __dadd_rn(v.z, __dmul_rn(sa, acc.z));
    }
    else if(AUX && S.integrator == I_GJF)   // core/GJFNVTLangevinIntegrator.hpp:183-204
    {
        double r0, r1, r2;
        noise(r0, r1, r2);
        const double4 x = a.accel[i];                       // {1/2m, b/m, b dt}
        const double b0 = __dmul_rn(r0, c.z), b1 = __dmul_rn(r1, c.z), b2 = __dmul_rn(r2, c.z);
        // dp = (b dt) (v + 1/2m (dt f + beta))
        dx = __dmul_rn(x.z, __dadd_rn(v.x, __dmul_rn(x.x, __dadd_rn(__dmul_rn(c.w, fx), b0))));
        dy = __dmul_rn(x.z, __dadd_rn(v.y, __dmul_rn(x.x, __dadd_rn(__dmul_rn(c.w, fy), b1))));
        dz = __dmul_rn(x.z, __dadd_rn(v.z, __dmul_rn(x.x, __dadd_rn(__dmul_rn(c.w, fz), b2))));
        // v = a (v + (dt/2m) f) + (b/m) beta
        v.x = __dadd_rn(__dmul_rn(c.y, __dadd_rn(v.x, __dmul_rn(c.x, fx))), __dmul_rn(x.y, b0));
        v.y = __dadd_rn(__dmul_rn(c.y, __dadd_rn(v.y, __dmul_rn(c.x, fy))), __dmul_rn(x.y, b1));
        v.z = __dadd_rn(__dmul_rn(c.y, __dadd_rn(v.z, __dmul_rn(c.x, fz))), __dmul_rn(x.y, b2));
    }
    else if(S.integrator == I_BAOAB || S.integrator == I_GBAOAB)
    {
        // g-BAOAB without constraints (gBAOABLangevinIntegrator.hpp:318-420,
        // one correction step): the same B-A-O-A, but each half drift moves
        // the position itself and the displacement is new minus old position
        const bool split = S.integrator == I_GBAOAB;
        double r0, r1, r2;
        noise(r0, r1, r2);
        v.x = __dadd_rn(v.x, __dmul_rn(c.x, fx));          // v += halfdt*rm*f
        v.y = __dadd_rn(v.y, __dmul_rn(c.x, fy));
        v.z = __dadd_rn(v.z, __dmul_rn(c.x, fz));
        dx = __dmul_rn(c.w, v.x);                          // dp  = halfdt*v
        dy = __dmul_rn(c.w, v.y);
        dz = __dmul_rn(c.w, v.z);
        if(split) {pn = make_double4(__dadd_rn(p.x, dx), __dadd_rn(p.y, dy), __dadd_rn(p.z, dz), p.w);}
        v.x = __dmul_rn(v.x, c.y);                         // v  *= exp(-gamma dt)
        v.y = __dmul_rn(v.y, c.y);
        v.z = __dmul_rn(v.z, c.y);
        v.x = __dadd_rn(v.x, __dmul_rn(c.z, r0));          // v  += noise*R
        v.y = __dadd_rn(v.y, __dmul_rn(c.z, r1));
        v.z = __dadd_rn(v.z, __dmul_rn(c.z, r2));
        if(split)
        {
            pn.x = __dadd_rn(pn.x, __dmul_rn(c.w, v.x));
            pn.y = __dadd_rn(pn.y, __dmul_rn(c.w, v.y));
            pn.z = __dadd_rn(pn.z, __dmul_rn(c.w, v.z));
            dx = __dsub_rn(pn.x, p.x);                     // displacement = new - old
            dy = __dsub_rn(pn.y, p.y);
            dz = __dsub_rn(pn.z, p.z);
            direct = true;
        }
        else
        {
            dx = __dadd_rn(dx, __dmul_rn(c.w, v.x));       // dp += halfdt*v
            dy = __dadd_rn(dy, __dmul_rn(c.w, v.y));
            dz = __dadd_rn(dz, __dmul_rn(c.w, v.z));
        }
    }
    else
    {
        v.x = __dadd_rn(v.x, __dmul_rn(c.x, fx));          // v += (halfdt*rm)*f
        v.y = __dadd_rn(v.y, __dmul_rn(c.x, fy));
        v.z = __dadd_rn(v.z, __dmul_rn(c.x, fz));
        dx = __dmul_rn(c.w, v.x);                          // disp = dt*v
        dy = __dmul_rn(c.w, v.y);
        dz = __dmul_rn(c.w, v.z);
    }
    if(direct) {p = pn;}
    else
    {
        p.x = __dadd_rn(p.x, dx);
        p.y = __dadd_rn(p.y, dy);
        p.z = __dadd_rn(p.z, dz);
    }
    if(S.boundary == B_PERIODIC)                           // adjust_position
    {
        if(p.x < S.lower[0]) {p.x = __dadd_rn(p.x, S.width[0]);} else if(p.x >= S.upper[0]) {p.x = __dsub_rn(p.x, S.width[0]);}
        if(p.y < S.lower[1]) {p.y = __dadd_rn(p.y, S.width[1]);} else if(p.y >= S.upper[1]) {p.y = __dsub_rn(p.y, S.width[1]);}
        if(p.z < S.lower[2]) {p.z = __dadd_rn(p.z, S.width[2]);} else if(p.z >= S.upper[2]) {p.z = __dsub_rn(p.z, S.width[2]);}
    }
    a.pos[i] = p;
    a.vel[i] = v;
    // the pair kernels read coordinates in slot order: keep every term's
    // copy current (a rebuild later in the step renumbers its systems'
    // slots and rewrites them)
#pragma unroll
    for(int g = 0; g < NGLOBAL; ++g)
    {
        if(so[g] >= 0) {a.slot_pd[g][so[g]] = make_double4(p.x, p.y, p.z, sw[g]);}   // whole 32 B
    }
    zero_force<PREC>(a.force, i);
    double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if(!(d2 == d2) || d2 > 1e300) {atomicOr(&S.status, ST_NONFINITE); d2 = 0.0;}
    return d2;
}

// The closing half of the last step of a chunk: v += (halfdt/m) f (BAOAB,
// velocity Verlet, G-JF) or the UnderdampedLangevin closing
__device__ __forceinline__ void close_particle(const Arena& a, const SysDev& S, long long i, unsigned long long step,
                                               double fx, double fy, double fz)
{
    double4 v = a.vel[i];
    if(S.integrator == I_UNDERDAMPED)
    {
        double4 acc = a.accel[i];
        underdamped_close(S, i, v, acc, S.uniform_coef ? S.coef : a.coef[i], fx, fy, fz, step);
        a.accel[i] = acc;
        a.vel[i] = v;
        return;
    }
    const double c = S.uniform_coef ? S.coef.x : a.coef[i].x;
    v.x = __dadd_rn(v.x, __dmul_rn(c, fx));
    v.y = __dadd_rn(v.y, __dmul_rn(c, fy));
    v.z = __dadd_rn(v.z, __dmul_rn(c, fz));
    a.vel[i] = v;
}

}  // namespace mjg
