// The elementary functions of the FP64 pair kernels, one call per element, for test_gpu_pair_math.py.
#include "pairs.cuh"

// the two functions of the library that the headers refer to
namespace sphgb {
char gCudaError[256];
void setCudaError(cudaError_t, const char*) {}
bool reclaimPairMemory(const DBuf*) { return false; }
}  // namespace sphgb

using namespace sphgb;

// what 0: a / b; 1: e^-a; 2 and 3: the Atwood weights of particles with densities a, b, logarithms la, lb and
// volumes xa, xb, as the forward pass and as the adjoint form them
__global__ void pairMath(int what, const double* a, const double* b, const double* rho, const double* lnxm,
                         const double* xm, const double4* tab, double* o0, double* o1, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (what == 0) o0[t] = quotient(a[t], b[t]);
    else if (what == 1) o0[t] = expNegSmall(a[t], tab);
    else if (what == 2)
        atwoodWeights(rho, lnxm, tab, t, n + t, float(rho[t]), float(rho[n + t]), xm[t], xm[n + t], o0[t], o1[t]);
    else {
        const AtwoodRamp w = atwoodRamp(tab, rho[t], rho[n + t], lnxm[t], lnxm[n + t], xm[t], xm[n + t]);
        o0[t] = w.am;
        o1[t] = w.bm;
    }
}

extern "C" int pair_math(int what, const double* a, const double* b, const double* rho, const double* lnxm,
                         const double* xm, const double* tab, double* o0, double* o1, int n)
{
    pairMath<<<(n + 127) / 128, 128>>>(what, a, b, rho, lnxm, xm, reinterpret_cast<const double4*>(tab), o0, o1, n);
    return int(cudaDeviceSynchronize());
}
