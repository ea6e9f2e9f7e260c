// The division policies of exact_div.cuh on arrays, for test_division_device_gpu.py.
#include "../../vanguard_b200/csrc/exact_div.cuh"

using namespace vg;

namespace {

// one quotient per element through each policy; ok: the shared policy's range flag
__global__ void quotients(const double* a, const double* b, long n, double* shared, double* ieee,
                          unsigned char* ok) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        SharedDiv s;
        shared[i] = s.by(b[i])(a[i]);
        ok[i] = s.ok();
        IeeeDiv c;
        ieee[i] = c.by(b[i])(a[i]);
    }
}
__global__ void thirds(const double* a, long n, double* shared, unsigned char* ok) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        SharedDiv s;
        shared[i] = s.third(a[i]);
        ok[i] = s.ok();
    }
}
// the limiters' quotients, whose operands' ranges the caller knows
__global__ void knowns(const double* a, const double* b, long n, double* q) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        q[i] = SharedDiv::known(a[i], b[i]);
}
__global__ void positives(const double* a, const double* b, long n, double* q, unsigned char* ok, unsigned char* below) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        SharedDiv s;
        q[i] = s.by(b[i]).positive(a[i]);
        ok[i] = s.ok();
        SharedDiv t;
        t.note_below(a[i]);
        below[i] = t.ok();
    }
}
__global__ void reciprocals(const double* b, long n, double* approximation, double* y) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        double r;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b[i]));
        approximation[i] = r;
        y[i] = SharedDiv::reciprocal(b[i]);
    }
}

}  // namespace

extern "C" {

int probe_quotients(const double* a, const double* b, long n, double* shared, double* ieee,
                    unsigned char* ok) {
    quotients<<<1184, 256>>>(a, b, n, shared, ieee, ok);
    return (int)cudaDeviceSynchronize();
}
int probe_thirds(const double* a, long n, double* shared, unsigned char* ok) {
    thirds<<<1184, 256>>>(a, n, shared, ok);
    return (int)cudaDeviceSynchronize();
}
int probe_knowns(const double* a, const double* b, long n, double* q) {
    knowns<<<1184, 256>>>(a, b, n, q);
    return (int)cudaDeviceSynchronize();
}
int probe_positives(const double* a, const double* b, long n, double* q, unsigned char* ok, unsigned char* below) {
    positives<<<1184, 256>>>(a, b, n, q, ok, below);
    return (int)cudaDeviceSynchronize();
}
int probe_reciprocals(const double* b, long n, double* approximation, double* y) {
    reciprocals<<<1184, 256>>>(b, n, approximation, y);
    return (int)cudaDeviceSynchronize();
}

}  // extern "C"
