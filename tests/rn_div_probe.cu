// Calls every quotient of rn_div.cuh beside the compiler's division, an operand pair
// per thread (test_gpu_rn_div.py). out[0]: the method, out[1]: `/`, ok: good guard.
#include <cstddef>

#include "rn_div.cuh"

using namespace hevi;

template <typename R>
__global__ void probe(int what, const R *a, const R *b, R *got, R *want, unsigned char *ok, size_t n)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rn::Guard<R> g;
    if (what == 0) { // div, its own reciprocal
        got[i] = rn::div<true>(g, a[i], b[i]);
        want[i] = a[i] / b[i];
    } else if (what == 1) { // div with a shared reciprocal
        const R y = rn::recip<true>(g, b[i]);
        got[i] = rn::div<true>(g, a[i], b[i], y);
        want[i] = a[i] / b[i];
    } else if (what == 2) { // either sign, own fallback
        got[i] = rn::quotient_mag(a[i], b[i]);
        want[i] = a[i] / b[i];
    } else if (what == 3) {
        got[i] = rn::sixth(a[i]);
        want[i] = a[i] / R(6.0);
    } else {
        got[i] = rn::third(a[i]);
        want[i] = a[i] / R(3.0);
    }
    ok[i] = !g.bad();
}

extern "C" int rn_probe(int is_double, int what, const void *a, const void *b, void *got, void *want,
                        unsigned char *ok, size_t n)
{
    const unsigned nb = (unsigned)((n + 255) / 256);
    if (is_double)
        probe<double><<<nb, 256>>>(what, (const double *)a, (const double *)b, (double *)got, (double *)want, ok, n);
    else
        probe<float><<<nb, 256>>>(what, (const float *)a, (const float *)b, (float *)got, (float *)want, ok, n);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
