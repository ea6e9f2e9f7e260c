// The HPR model's two forms (with p_inf, and without: Plain) on arrays of conserved vectors, for test_hpr_forms_gpu.py.
#include "../../vanguard_b200/csrc/physics_hpr.cuh"

using namespace vg;

namespace {

template <class M, class D>
__device__ void evaluate(const double* U, const typename M::P& q, double* out, D& dv) {
    M::template flux<0>(U, q, out, dv);
    M::template flux<1>(U, q, out + 17, dv);
    M::source(U, q, out + 34, dv);
}
// out: [form][component][cell]; forms: general and plain with the compiler's division, plain with the shared one (ok: in range)
__global__ void forms(const double* U, const double* prm, long n, double* out, unsigned char* ok) {
    using G = HPRModel<false>;
    using P = G::Plain;
    const G::P qg = G::params(prm, 0.0);
    const P::P qp = P::params(prm, 0.0);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        double u[17], o[51];
        for (int v = 0; v < 17; v++) u[v] = U[v * n + i];
        IeeeDiv c;
        evaluate<G>(u, qg, o, c);
        for (int v = 0; v < 51; v++) out[v * n + i] = o[v];
        evaluate<P>(u, qp, o, c);
        for (int v = 0; v < 51; v++) out[(51 + v) * n + i] = o[v];
        SharedDiv s;
        evaluate<P>(u, qp, o, s);
        for (int v = 0; v < 51; v++) out[(102 + v) * n + i] = o[v];
        ok[i] = s.ok();
    }
}

}  // namespace

extern "C" int probe_forms(const double* U, const double* prm, long n, double* out, unsigned char* ok) {
    forms<<<592, 128>>>(U, prm, n, out, ok);
    return (int)cudaDeviceSynchronize();
}
