// Device functions of the pair evaluation against CUDA's own: the largest
// distance in units in the last place and the number of differing results, over
// every mantissa of a range of exponents (tests/test_gpu_fast_math.py).
#include "pair_eval.cuh"

namespace mjg {
void note_launches(int) {}
}

struct Result {
    unsigned long long differ;       // results that are not the reference's float
    unsigned long long beyond;       // results further than one unit in the last place from it
    double worst;                    // largest relative error against FP64
};

namespace {

__device__ int ulps(float a, float b)
{
    return abs(__float_as_int(a) - __float_as_int(b));          // one sign
}

template<class F>
__global__ void scan(int first_exp, int exps, Result* out, F f)
{
    unsigned long long differ = 0, beyond = 0;
    double worst = 0.0;
    const long long n = (long long)exps << 23;
    for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    {
        const float x = __int_as_float((int)((first_exp + 127 + (k >> 23)) << 23 | (k & 0x7fffff)));
        float got, ref;
        double exact;
        f(x, got, ref, exact);
        const int u = ulps(got, ref);
        differ += u != 0;
        beyond += u > 1;
        worst = fmax(worst, fabs((double)got - exact) / fabs(exact));
    }
    atomicAdd(&out->differ, differ);
    atomicAdd(&out->beyond, beyond);
    atomicMax(reinterpret_cast<unsigned long long*>(&out->worst), (unsigned long long)__double_as_longlong(worst));
}

struct Reciprocal {
    __device__ void operator()(float x, float& got, float& ref, double& exact) const
    {
        got = mjg::reciprocal(x); ref = __frcp_rn(x); exact = 1.0 / (double)x;
    }
};
struct Rsqrt {
    __device__ void operator()(float x, float& got, float& ref, double& exact) const
    {
        got = mjg::rsqrt_approx(x); ref = rsqrtf(x); exact = rsqrt((double)x);
    }
};
// exp(-x) as DebyeHuckel takes it
struct Exp {
    __device__ void operator()(float x, float& got, float& ref, double& exact) const
    {
        got = mjg::exp2_approx(x * -1.4426950408889634f); ref = __expf(-x); exact = exp(-(double)x);
    }
};

}  // namespace

extern "C" __attribute__((visibility("default"))) int fast_math_scan(int which, int first_exp, int exps, Result* host)
{
    Result* d = nullptr;
    if(cudaMalloc(&d, sizeof(Result)) != cudaSuccess) {return 1;}
    cudaMemset(d, 0, sizeof(Result));
    if(which == 0)      {scan<<<148 * 8, 256>>>(first_exp, exps, d, Reciprocal{});}
    else if(which == 1) {scan<<<148 * 8, 256>>>(first_exp, exps, d, Rsqrt{});}
    else                {scan<<<148 * 8, 256>>>(first_exp, exps, d, Exp{});}
    const bool ok = cudaMemcpy(host, d, sizeof(Result), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(d);
    return ok ? 0 : 1;
}
