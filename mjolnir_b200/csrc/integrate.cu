// BAOAB Langevin and velocity-Verlet updates (core/BAOABLangevinIntegrator.hpp
// :170-240, core/VelocityVerletIntegrator.hpp:90-135), the Verlet-skin
// bookkeeping of reduce_margin (core/PeriodicGridCellList.hpp:100-110), and
// the host<->arena layout conversions.
//
// One thread per particle over every system of the arena; a particle finds its
// system's box, seed and step through psys.  Arithmetic is FP64 with explicit
// round-to-nearest products and sums, in the reference's operation order.
#include "integrate.cuh"

namespace mjg {

namespace {

constexpr int TPB = 256;

// advance_particle over every particle of the arena, with the per-system
// largest squared displacement.  KICK: with the previous step's closing half.
template<int PREC, bool KICK, bool AUX>
__global__ void __launch_bounds__(TPB) k_integrate_first(Arena a)
{
    const long long i = (long long)blockIdx.x * TPB + threadIdx.x;
    const bool active = i < a.n;
    int s = active ? a.psys[i] : 0;
    double d2 = 0.0;
    if(active && !a.sys[s].frozen)
    {
        SysDev& S = a.sys[s];
        d2 = advance_particle<PREC, AUX>(a, S, i, KICK, S.step, [&](double& r0, double& r1, double& r2) {
            gaussian3(S.seed, (unsigned long long)(i - S.off), S.step, r0, r1, r2);
        }, [&](double& fx, double& fy, double& fz) {load_force<PREC>(a.force, i, fx, fy, fz);});
    }
    // per-system maximum: warp-level when the warp sits in one system
    const unsigned full = 0xffffffffu;
    const int s0 = __shfl_sync(full, s, 0);
    const bool uniform = __all_sync(full, !active || s == s0);
    if(uniform)
    {
        double m = d2;
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) {m = fmax(m, __shfl_xor_sync(full, m, o));}
        const bool any = __any_sync(full, active);
        if(any && (threadIdx.x & 31) == 0)
        {
            atomicMax(&a.sys[s0].max_disp2, (unsigned long long)__double_as_longlong(m));
        }
    }
    else if(active)
    {
        atomicMax(&a.sys[s].max_disp2, (unsigned long long)__double_as_longlong(d2));
    }
}

// reduce_margin(2 sqrt(max|dp|^2)) for every global term of every system;
// a term whose skin is used up is flagged for a rebuild.  Also advances the
// noise step counter.
__global__ void k_margin(Arena a, int* any0, int* any1, int* any2, RebuildGate gate)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s >= a.nsys) {return;}
    SysDev& S = a.sys[s];
    if(S.frozen) {return;}
    const double d = 2 * sqrt(__longlong_as_double((long long)S.max_disp2));
    S.max_disp2 = 0ull;
    S.step += 1ull;
    int* any[3] = {any0, any1, any2};
    for(int g = 0; g < NGLOBAL; ++g)
    {
        GlobalParams& G = S.g[g];
        if(!G.on) {continue;}
        G.current_margin = __dsub_rn(G.current_margin, d);
        if(G.current_margin < 0)
        {
            G.rebuild = 1;
            if(any[g]) {atomicOr(any[g], 1);}
            if(gate.on[g]) {cudaGraphSetConditional(gate.handle[g], 1u);}   // the term's rebuild runs
        }
    }
}

// closing half of the last step of a chunk
template<int PREC>
__global__ void __launch_bounds__(TPB) k_integrate_last(Arena a)
{
    const long long i = (long long)blockIdx.x * TPB + threadIdx.x;
    if(i >= a.n) {return;}
    const SysDev& S = a.sys[a.psys[i]];
    if(S.frozen) {return;}
    double fx, fy, fz;
    load_force<PREC>(a.force, i, fx, fy, fz);
    close_particle(a, S, i, S.step, fx, fy, fz);
}

// UnderdampedLangevinIntegrator::initialize (:160-181): a = f/m + sigma R,
// with the noise counter at the system's current step (a resumed system gets
// the acceleration the uninterrupted run had)
template<int PREC>
__global__ void k_init_accel(Arena a, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k >= count) {return;}
    const long long i = first + k;
    const SysDev& S = a.sys[a.psys[i]];
    if(S.integrator != I_UNDERDAMPED) {return;}
    double fx, fy, fz;
    load_force<PREC>(a.force, i, fx, fy, fz);
    const double4 c = S.uniform_coef ? S.coef : a.coef[i];
    double r0, r1, r2;
    gaussian3(S.seed, (unsigned long long)(i - S.off), S.step, r0, r1, r2);
    a.accel[i] = make_double4(__dadd_rn(__dmul_rn(fx, c.x), __dmul_rn(r0, c.z)),
                              __dadd_rn(__dmul_rn(fy, c.x), __dmul_rn(r1, c.z)),
                              __dadd_rn(__dmul_rn(fz, c.x), __dmul_rn(r2, c.z)), 0.0);
}

template<int PREC>
__global__ void k_zero_force(Arena a)
{
    const long long i = (long long)blockIdx.x * TPB + threadIdx.x;
    if(i < a.n && !a.sys[a.psys[i]].frozen) {zero_force<PREC>(a.force, i);}
}

__global__ void k_unpack(Arena a, const double* src_pos, const double* src_vel, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k >= count) {return;}
    const long long i = first + k;
    if(src_pos) {a.pos[i] = make_double4(src_pos[3*k], src_pos[3*k+1], src_pos[3*k+2], 0.0);}
    if(src_vel) {a.vel[i] = make_double4(src_vel[3*k], src_vel[3*k+1], src_vel[3*k+2], 0.0);}
}

template<int PREC>
__global__ void k_pack(Arena a, double* dst, int what, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k >= count) {return;}
    const long long i = first + k;
    double x, y, z;
    if(what == 0)      {const double4 p = a.pos[i]; x = p.x; y = p.y; z = p.z;}
    else if(what == 1) {const double4 v = a.vel[i]; x = v.x; y = v.y; z = v.z;}
    else if(what == 3) {const double4 q = a.accel ? a.accel[i] : make_double4(0, 0, 0, 0); x = q.x; y = q.y; z = q.z;}
    else               {load_force<PREC>(a.force, i, x, y, z);}
    dst[3*k] = x; dst[3*k+1] = y; dst[3*k+2] = z;
}

template<int PREC>
__global__ void k_set_force(Arena a, const double* src, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k >= count) {return;}
    const long long i = first + k;
    if(PREC == P_FP64)
    {
        static_cast<double4*>(a.force)[i] = make_double4(src[3*k], src[3*k+1], src[3*k+2], 0.0);
    }
    else
    {
        static_cast<longlong4*>(a.force)[i] = make_longlong4(fx_from_double(src[3*k]),
            fx_from_double(src[3*k+1]), fx_from_double(src[3*k+2]), 0);
    }
}

__global__ void k_set_noise(Arena a, const double* src, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k < count) {a.coef[first + k].z = src[k];}
}

__global__ void k_clear_energy(Arena a)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if(s >= a.nsys) {return;}
    for(int t = 0; t < NTERMS; ++t) {a.sys[s].energy[t] = 0.0;}
}

inline unsigned blocks(long long n) {return (unsigned)((n + TPB - 1) / TPB);}

}  // namespace

void launch_integrate_first(const Arena& a, cudaStream_t s, bool kick)
{
    if(a.n == 0) {return;}
    const bool aux = a.accel != nullptr;
    const int nb = (int)blocks(a.n);
    if(a.precision == P_FP64)
    {
        if(aux) {if(kick) {k_integrate_first<P_FP64, true,  true ><<<nb, TPB, 0, s>>>(a);}
                 else     {k_integrate_first<P_FP64, false, true ><<<nb, TPB, 0, s>>>(a);}}
        else    {if(kick) {k_integrate_first<P_FP64, true,  false><<<nb, TPB, 0, s>>>(a);}
                 else     {k_integrate_first<P_FP64, false, false><<<nb, TPB, 0, s>>>(a);}}
    }
    else
    {
        if(aux) {if(kick) {k_integrate_first<P_MIXED, true,  true ><<<nb, TPB, 0, s>>>(a);}
                 else     {k_integrate_first<P_MIXED, false, true ><<<nb, TPB, 0, s>>>(a);}}
        else    {if(kick) {k_integrate_first<P_MIXED, true,  false><<<nb, TPB, 0, s>>>(a);}
                 else     {k_integrate_first<P_MIXED, false, false><<<nb, TPB, 0, s>>>(a);}}
    }
    note_launches(1);
}

void launch_margin(const Arena& a, TermArrays* t, cudaStream_t s, const RebuildGate& gate)
{
    if(a.nsys == 0) {return;}
    k_margin<<<(a.nsys + 127) / 128, 128, 0, s>>>(a,
        t[0].on ? t[0].any_rebuild : nullptr, t[1].on ? t[1].any_rebuild : nullptr,
        t[2].on ? t[2].any_rebuild : nullptr, gate);
    note_launches(1);
}

__global__ void k_set_accel(Arena a, const double* src, long long first, long long count)
{
    const long long k = (long long)blockIdx.x * TPB + threadIdx.x;
    if(k < count) {a.accel[first + k] = make_double4(src[3 * k], src[3 * k + 1], src[3 * k + 2], 0.0);}
}

void launch_set_accel(const Arena& a, const double* src, long long first, long long count, cudaStream_t s)
{
    if(count == 0 || !a.accel) {return;}
    k_set_accel<<<blocks(count), TPB, 0, s>>>(a, src, first, count);
    note_launches(1);
}

void launch_init_accel(const Arena& a, long long first, long long count, cudaStream_t s)
{
    if(count == 0 || !a.accel) {return;}
    if(a.precision == P_FP64) {k_init_accel<P_FP64><<<blocks(count), TPB, 0, s>>>(a, first, count);}
    else                      {k_init_accel<P_MIXED><<<blocks(count), TPB, 0, s>>>(a, first, count);}
    note_launches(1);
}

void launch_integrate_last(const Arena& a, cudaStream_t s)
{
    if(a.n == 0) {return;}
    if(a.precision == P_FP64) {k_integrate_last<P_FP64><<<blocks(a.n), TPB, 0, s>>>(a);}
    else                      {k_integrate_last<P_MIXED><<<blocks(a.n), TPB, 0, s>>>(a);}
    note_launches(1);
}

void launch_zero_force(const Arena& a, cudaStream_t s)
{
    if(a.n == 0) {return;}
    if(a.precision == P_FP64) {k_zero_force<P_FP64><<<blocks(a.n), TPB, 0, s>>>(a);}
    else                      {k_zero_force<P_MIXED><<<blocks(a.n), TPB, 0, s>>>(a);}
    note_launches(1);
}

void launch_unpack_state(const Arena& a, const double* src_pos, const double* src_vel,
                         long long first, long long count, cudaStream_t s)
{
    if(count == 0) {return;}
    k_unpack<<<blocks(count), TPB, 0, s>>>(a, src_pos, src_vel, first, count);
    note_launches(1);
}

void launch_pack_state(const Arena& a, double* dst, int what, long long first, long long count,
                       cudaStream_t s)
{
    if(count == 0) {return;}
    if(a.precision == P_FP64) {k_pack<P_FP64><<<blocks(count), TPB, 0, s>>>(a, dst, what, first, count);}
    else                      {k_pack<P_MIXED><<<blocks(count), TPB, 0, s>>>(a, dst, what, first, count);}
    note_launches(1);
}

void launch_clear_energy(const Arena& a, cudaStream_t s)
{
    if(a.nsys == 0) {return;}
    k_clear_energy<<<(a.nsys + 127) / 128, 128, 0, s>>>(a);
    note_launches(1);
}

// reads `n` int4 words and keeps one word of the result (only when it takes
// an impossible value), so that every line read stays clean in L2
__global__ void k_read_sweep(const int4* __restrict__ p, long long n, int* sink)
{
    int acc = 0;
    for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
        k += (long long)gridDim.x * blockDim.x)
    {
        const int4 w = __ldcg(p + k);
        acc ^= w.x ^ w.y ^ w.z ^ w.w;
    }
    if(acc == 0x7fffffff && sink) {*sink = acc;}
}

void launch_read_sweep(const void* p, size_t bytes, int* sink, cudaStream_t s)
{
    const long long n = (long long)(bytes / sizeof(int4));
    if(n == 0) {return;}
    k_read_sweep<<<148 * 8, 256, 0, s>>>(static_cast<const int4*>(p), n, sink);
    note_launches(1);
}

void launch_set_noise(const Arena& a, const double* noise, long long first, long long count,
                      cudaStream_t s)
{
    if(count == 0) {return;}
    k_set_noise<<<blocks(count), TPB, 0, s>>>(a, noise, first, count);
    note_launches(1);
}

void launch_set_force(const Arena& a, const double* src, long long first, long long count,
                      cudaStream_t s)
{
    if(count == 0) {return;}
    if(a.precision == P_FP64) {k_set_force<P_FP64><<<blocks(count), TPB, 0, s>>>(a, src, first, count);}
    else                      {k_set_force<P_MIXED><<<blocks(count), TPB, 0, s>>>(a, src, first, count);}
    note_launches(1);
}

}  // namespace mjg
