// ExcludedVolume forces of one system held by the caller in device memory,
// without any device allocation (mjg_exv_force_noalloc in mjolnir_b200.h).
//
// Who needs this: code that runs where cudaMalloc is not available to it --
// inside a host that owns all device memory itself (a framework with its own
// pool, an embedding that forbids allocation after start-up) -- cannot create
// an mjg_context, whose arena is allocated at mjg_commit.  This entry point
// needs nothing but the caller's input and output buffers: the cell list it
// builds lives in a fixed, file-scope device array that every GPU loading the
// library holds until the process exits.
//
// The force is the ExcludedVolume pair sum over all particle pairs within
// sigma_ij * cutoff_ratio (sigma_ij = r_i + r_j), every particle taking part
// and no pair excluded, evaluated in FP64 with the reference's expressions
// (forcefield/global/GlobalPairExcludedVolumeInteraction.hpp:148-195); it is
// the same quantity mjg_term_force returns for MJG_TERM_EXV of a system with
// no ignore rules.  Each particle walks its 27 neighbouring cells (no Verlet
// margin), so its force is written once, without atomics.
#include "../../include/mjolnir_b200.h"
#include "common.cuh"

#include <cstdio>
#include <mutex>

namespace mjg {
namespace {

constexpr int NA_MAX_PARTICLES = 65536;
constexpr int NA_MAX_CELLS     = 65536;
constexpr int NA_TPB           = 256;
constexpr int NA_BLOCKS        = 64;      // blocks of the radius pass
constexpr int NA_SCAN          = 1024;    // cells per block of the scan
constexpr int NA_LANES         = 8;       // lanes per particle of the force pass

// header: [0] dims x, [1] dims y, [2] dims z, [3] hashed
struct NaScratch {
    int      header[8];
    double   inv_w;
    double   max_radius[NA_BLOCKS];       // of each block's share
    int      count[NA_MAX_CELLS];
    int      start[NA_MAX_CELLS + 1];
    unsigned place[NA_MAX_PARTICLES];     // cell, and rank within it, 16 bits each
    int      order[NA_MAX_PARTICLES];
};

// The one scratch area of this entry point (about 1 MiB per device).  In host
// code this name is only a stand-in; kernels receive the device address that
// cudaGetSymbolAddress returns.
static __device__ __align__(256) NaScratch g_na_scratch;

struct NaBox {
    int periodic;
    double lower[3], width[3], halfw[3];
};

// The five launches of a call are a few microseconds of latency each: every one
// spreads its work over the GPU (one block that took the largest radius, cleared
// 65,536 cells and scanned them took 60 us of a call's 150).

// largest radius of each block's share, counters to zero
__global__ void __launch_bounds__(NA_TPB) k_na_radius(NaScratch* sc, long long n, const double* radius, double* energy)
{
    __shared__ double red[NA_TPB / 32];
    const int t = blockIdx.x * NA_TPB + threadIdx.x;
    double m = 0.0;
    for(long long i = t; i < n; i += NA_BLOCKS * NA_TPB) {m = fmax(m, radius[i]);}
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));}
    if((threadIdx.x & 31) == 0) {red[threadIdx.x >> 5] = m;}
    // the previous call's contents must not leak into this one
    for(int c = t; c < NA_MAX_CELLS; c += NA_BLOCKS * NA_TPB) {sc->count[c] = 0;}
    if(t == 0) {*energy = 0.0;}
    __syncthreads();
    if(threadIdx.x == 0)
    {
        for(int k = 1; k < NA_TPB / 32; ++k) {m = fmax(m, red[k]);}
        sc->max_radius[blockIdx.x] = m;
    }
}

// grid shape from the largest radius, by every block of the binning for itself
__device__ __forceinline__ void na_grid(const NaScratch* sc, long long n, double cutoff_ratio, const NaBox& box,
                                        int (&header)[4], double& inv_w)
{
    double mr = 0.0;
    for(int k = 0; k < NA_BLOCKS; ++k) {mr = fmax(mr, sc->max_radius[k]);}
    const double rc = mr * 2 * cutoff_ratio;       // ExcludedVolumePotential::max_cutoff
    int d[3];
    if(box.periodic)
    {
        for(int x = 0; x < 3; ++x)
        {
            const double c = rc > 0 ? floor(box.width[x] / rc) : 3.0;
            d[x] = (int)fmin(fmax(c, 3.0), 64.0);   // at least 3, cells at least rc wide
        }
        while((long long)d[0] * d[1] * d[2] > NA_MAX_CELLS)
        {
            int b = 0;
            for(int x = 1; x < 3; ++x) {if(d[x] > d[b]) {b = x;}}
            d[b] -= 1;
        }
        inv_w = 0.0;
    }
    else
    {
        // unbounded space: cells rc wide hashed modulo a small grid
        int dd = (int)ceil(cbrt((double)n));
        dd = dd < 3 ? 3 : (dd > 32 ? 32 : dd);
        d[0] = d[1] = d[2] = dd;
        inv_w = rc > 0 ? 1.0 / (rc * (1 + 1e-9)) : 0.0;
    }
    header[0] = d[0]; header[1] = d[1]; header[2] = d[2];
    header[3] = box.periodic ? 0 : 1;
}

__device__ __forceinline__ int na_coord(const int* header, double inv_w, const NaBox& box, double x, int axis)
{
    const int d = header[axis];
    if(box.periodic)
    {
        // wrapped: a particle a little outside [lower, upper) lands in the
        // cell its periodic image occupies, next to its image neighbours
        long long c = (long long)floor((x - box.lower[axis]) / (box.width[axis] / d)) % d;
        return (int)(c < 0 ? c + d : c);
    }
    long long c = (long long)floor(x * inv_w) % d;
    return (int)(c < 0 ? c + d : c);
}

// cell of each particle and its place in the cell
__global__ void __launch_bounds__(NA_TPB) k_na_bin(NaScratch* sc, long long n, const double* pos, double cutoff_ratio, NaBox box)
{
    __shared__ int header[4];
    __shared__ double inv_w;
    if(threadIdx.x == 0)
    {
        int h[4];
        double w;
        na_grid(sc, n, cutoff_ratio, box, h, w);
        for(int k = 0; k < 4; ++k) {header[k] = h[k];}
        inv_w = w;
        if(blockIdx.x == 0)
        {
            for(int k = 0; k < 4; ++k) {sc->header[k] = h[k];}
            sc->inv_w = w;
        }
    }
    __syncthreads();
    const long long i = (long long)blockIdx.x * NA_TPB + threadIdx.x;
    if(i >= n) {return;}
    const int c = na_coord(header, inv_w, box, pos[3 * i], 0) + header[0] * (na_coord(header, inv_w, box, pos[3 * i + 1], 1) +
                  header[1] * na_coord(header, inv_w, box, pos[3 * i + 2], 2));
    sc->place[i] = (unsigned)c << 16 | (unsigned)atomicAdd(&sc->count[c], 1);
}

// exclusive scan of the cell counts, one block per NA_SCAN cells: a block adds up
// the counts before its own cells itself (at most 256 KB from L2), so the blocks
// need not wait for one another
__global__ void __launch_bounds__(NA_SCAN) k_na_scan(NaScratch* sc)
{
    __shared__ int tot[32];
    __shared__ int base;
    const int ncell = sc->header[0] * sc->header[1] * sc->header[2];
    const int first = blockIdx.x * NA_SCAN;
    if(first >= ncell) {return;}
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int before = 0;
    for(int c = threadIdx.x; c < first; c += NA_SCAN) {before += sc->count[c];}
    before = __reduce_add_sync(0xffffffffu, before);
    const int c = first + threadIdx.x;
    const int v = c < ncell ? sc->count[c] : 0;
    int incl = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if(lane >= o) {incl += y;}
    }
    if(threadIdx.x == 0) {base = 0;}
    if(lane == 31) {tot[w] = incl;}
    __syncthreads();
    if(lane == 0 && before) {atomicAdd(&base, before);}
    __syncthreads();
    int run = base;
    for(int k = 0; k < w; ++k) {run += tot[k];}
    if(c < ncell) {sc->start[c] = run + incl - v;}
    if(c == ncell - 1) {sc->start[ncell] = run + incl;}
}

__global__ void __launch_bounds__(NA_TPB) k_na_scatter(NaScratch* sc, long long n)
{
    const long long i = (long long)blockIdx.x * NA_TPB + threadIdx.x;
    if(i >= n) {return;}
    const unsigned p = sc->place[i];
    sc->order[sc->start[p >> 16] + (int)(p & 0xffffu)] = (int)i;
}

// Forces, NA_LANES lanes per particle, particles in cell order (neighbouring
// groups read the same partners).  The 27 cells around a particle are nine rows
// along x, each one range of the cell order or two where it wraps; the lanes
// look the at most 18 ranges up together and then walk their concatenation, so
// a particle's candidates (41 in the bead fluid) are a few loads deep instead of
// one serial chain through 27 cells.
constexpr int NA_RANGES = 18;
__global__ void __launch_bounds__(NA_TPB) k_na_force(const NaScratch* sc, long long n, const double* pos, const double* radius,
                           double eps, double cutoff_ratio, NaBox box, double* force, double* energy)
{
    constexpr int GROUPS = NA_TPB / NA_LANES;
    __shared__ int s_begin[GROUPS][NA_RANGES];
    __shared__ int s_excl[GROUPS][NA_RANGES + 1];
    const unsigned full = 0xffffffffu;
    const int grp = threadIdx.x / NA_LANES, gl = threadIdx.x % NA_LANES;
    int* const begin = s_begin[grp];
    int* const excl = s_excl[grp];
    const long long slot = (long long)blockIdx.x * GROUPS + grp;
    const bool valid = slot < n;
    double e = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
    int i = 0;
    double xi = 0.0, yi = 0.0, zi = 0.0, ri = 0.0;
    if(valid)
    {
        i = sc->order[slot];
        xi = pos[3 * i]; yi = pos[3 * i + 1]; zi = pos[3 * i + 2]; ri = radius[i];
        const int cell = (int)(sc->place[i] >> 16);
        const int nx = sc->header[0], ny = sc->header[1], nz = sc->header[2];
        const int cx = cell % nx, cy = cell / nx % ny, cz = cell / (nx * ny);
        for(int j = gl; j < 9; j += NA_LANES)
        {
            const int y = (cy + j % 3 - 1 + ny) % ny, z = (cz + j / 3 - 1 + nz) % nz;
            const int row = nx * (y + ny * z);
            int lo = cx - 1, hi = cx + 1, hi1 = -1;      // the second range is [0, hi1]
            if(lo < 0)        {lo = hi = nx - 1; hi1 = cx + 1;}
            else if(hi >= nx) {hi = nx - 1; hi1 = 0;}
            begin[2 * j] = sc->start[row + lo];
            excl[2 * j] = sc->start[row + hi + 1] - begin[2 * j];
            begin[2 * j + 1] = sc->start[row];
            excl[2 * j + 1] = sc->start[row + hi1 + 1] - begin[2 * j + 1];
        }
    }
    __syncwarp();
    if(valid && gl == 0)
    {
        int run = 0;
        for(int k = 0; k < NA_RANGES; ++k)
        {
            const int c = excl[k];
            excl[k] = run;
            run += c;
        }
        excl[NA_RANGES] = run;
    }
    __syncwarp();
    if(valid)
    {
        const double crsq = cutoff_ratio * cutoff_ratio;
        const double coef_at_cutoff = pow(1.0 / cutoff_ratio, 12);   // ExcludedVolumePotential.hpp:44-48
        const double eps12 = eps * 12;
        const int total = excl[NA_RANGES];
        int at = 0;
        auto candidate = [&](int k) {
            if(k >= total) {return i;}               // none: the particle itself, which is dropped
            while(at < NA_RANGES - 1 && excl[at + 1] <= k) {++at;}
            return sc->order[begin[at] + (k - excl[at])];
        };
        // the next candidate's coordinates are requested before the current pair is evaluated
        int j = candidate(gl);
        double xj = pos[3 * j], yj = pos[3 * j + 1], zj = pos[3 * j + 2], rj = radius[j];
        for(int k = gl; k < total; k += NA_LANES)
        {
            const int jn = candidate(k + NA_LANES);
            const double xn = pos[3 * jn], yn = pos[3 * jn + 1], zn = pos[3 * jn + 2], rn = radius[jn];
            if(j != i)
            {
                double ddx = xj - xi, ddy = yj - yi, ddz = zj - zi;
                if(box.periodic)
                {
                    ddx = min_image(ddx, box.halfw[0], box.width[0]);
                    ddy = min_image(ddy, box.halfw[1], box.width[1]);
                    ddz = min_image(ddz, box.halfw[2], box.width[2]);
                }
                const double l_sq = ddx * ddx + ddy * ddy + ddz * ddz;
                const double sigma = ri + rj;
                const double sigma_sq = sigma * sigma;
                if(!(sigma_sq * crsq < l_sq))
                {
                    const double rcp = 1.0 / l_sq;
                    const double s2 = sigma_sq * rcp;
                    const double s6 = s2 * s2 * s2;
                    const double cf = -eps12 * s6 * s6 * rcp;
                    fx += ddx * cf; fy += ddy * cf; fz += ddz * cf;
                    if(i < j) {e += eps * (s6 * s6 - coef_at_cutoff);}
                }
            }
            j = jn;
            xj = xn; yj = yn; zj = zn; rj = rn;
        }
    }
#pragma unroll
    for(int o = NA_LANES / 2; o > 0; o >>= 1)
    {
        fx += __shfl_xor_sync(full, fx, o);
        fy += __shfl_xor_sync(full, fy, o);
        fz += __shfl_xor_sync(full, fz, o);
    }
    if(valid && gl == 0) {force[3 * i] = fx; force[3 * i + 1] = fy; force[3 * i + 2] = fz;}
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {e += __shfl_xor_sync(full, e, o);}
    if((threadIdx.x & 31) == 0 && e != 0.0) {atomicAdd(energy, e);}
}

// Device address of the scratch array, looked up once per CUDA context: the
// address belongs to the context that was current at the lookup, and a device
// reset (cudaDeviceReset, or a host framework resetting the primary context)
// makes a new context in which the array has a new address.  The current
// context is read through the driver's cuCtxGetCurrent, found at run time so
// that the library does not link against the driver.
std::mutex g_na_mutex;
struct NaSlot {
    void* ctx;
    NaScratch* ptr;
};
NaSlot g_na_slots[64] = {};
int g_na_nslots = 0;
using CtxGetCurrent = int (*)(void**);
CtxGetCurrent g_ctx_get_current = nullptr;

// the current context (nullptr when none is current or the driver does not
// say); called with g_na_mutex held
void* current_context()
{
    if(!g_ctx_get_current)
    {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if(cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q) != cudaSuccess ||
           q != cudaDriverEntryPointSuccess || !fn)
        {
            cudaGetLastError();
            return nullptr;
        }
        g_ctx_get_current = reinterpret_cast<CtxGetCurrent>(fn);
    }
    void* ctx = nullptr;
    return g_ctx_get_current(&ctx) == 0 ? ctx : nullptr;
}

}  // namespace
}  // namespace mjg

using namespace mjg;

extern "C" MJG_API int mjg_exv_force_noalloc(int64_t n, int boundary, const double* lower,
                                             const double* upper, const double* pos,
                                             const double* radius, double epsilon,
                                             double cutoff_ratio, double* force, double* energy,
                                             void* stream)
{
    if(n <= 0 || !pos || !radius || !force || !energy || !(cutoff_ratio > 0)) {return MJG_EINVAL;}
    if(n > NA_MAX_PARTICLES)
    {
        std::fprintf(stderr, "mjg_exv_force_noalloc: %lld particles exceed the limit of %d\n",
                     (long long)n, NA_MAX_PARTICLES);
        return MJG_EINVAL;
    }
    if(boundary != MJG_UNLIMITED && boundary != MJG_PERIODIC_CUBOID) {return MJG_EINVAL;}
    NaBox box{};
    box.periodic = boundary == MJG_PERIODIC_CUBOID;
    if(box.periodic)
    {
        if(!lower || !upper) {return MJG_EINVAL;}
        for(int x = 0; x < 3; ++x)
        {
            box.lower[x] = lower[x];
            box.width[x] = upper[x] - lower[x];
            box.halfw[x] = box.width[x] / 2;
            if(!(box.width[x] > 0)) {return MJG_EINVAL;}
        }
    }
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess || dev < 0) {cudaGetLastError(); return MJG_ECUDA;}
    NaScratch* sc = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_na_mutex);
        // the first call in a context (the first on a device, or the first
        // after a reset) has the runtime make the device's primary context
        // current (cudaSetDevice initialises it), then looks the array's
        // address up in it; without a context handle the address is looked
        // up on every call
        if(cudaSetDevice(dev) != cudaSuccess) {cudaGetLastError(); return MJG_ECUDA;}
        void* ctx = current_context();
        for(int k = 0; k < g_na_nslots && ctx; ++k)
        {
            if(g_na_slots[k].ctx == ctx) {sc = g_na_slots[k].ptr; break;}
        }
        if(!sc)
        {
            void* p = nullptr;
            if(cudaGetSymbolAddress(&p, g_na_scratch) != cudaSuccess || !p)
            {
                cudaGetLastError();
                return MJG_ECUDA;
            }
            sc = static_cast<NaScratch*>(p);
            if(ctx)
            {
                // keep at most 64 contexts; the oldest entry gives way
                if(g_na_nslots < 64) {++g_na_nslots;}
                for(int k = g_na_nslots - 1; k > 0; --k) {g_na_slots[k] = g_na_slots[k - 1];}
                g_na_slots[0] = NaSlot{ctx, sc};
            }
        }
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned nb = (unsigned)((n + NA_TPB - 1) / NA_TPB);
    const unsigned nf = (unsigned)((n * NA_LANES + NA_TPB - 1) / NA_TPB);
    k_na_radius <<<NA_BLOCKS, NA_TPB, 0, s>>>(sc, n, radius, energy);
    k_na_bin    <<<nb, NA_TPB, 0, s>>>(sc, n, pos, cutoff_ratio, box);
    k_na_scan   <<<NA_MAX_CELLS / NA_SCAN, NA_SCAN, 0, s>>>(sc);
    k_na_scatter<<<nb, NA_TPB, 0, s>>>(sc, n);
    k_na_force  <<<nf, NA_TPB, 0, s>>>(sc, n, pos, radius, epsilon, cutoff_ratio, box, force, energy);
    return cudaGetLastError() == cudaSuccess ? MJG_OK : MJG_ECUDA;
}
