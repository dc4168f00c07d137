// Device helpers called on their own, for test_gpu_device_units.py: compiled
// there with the library's flags and loaded with ctypes.  Every function
// returns the CUDA error of its calls (0: none); arrays are host memory.

#include "../include/fcc_user_terms.h"

namespace fcc_user {
// sqrt(R'^2 + R''^2): not differentiable on a circle, where both vanish
struct Kink {
    static constexpr int M = 1;
    template <class T>
    FCC_HD static void q(T, T dR, T ddR, T, T, T* out) {
        out[0] = sqrt(dR * dR + ddR * ddR);
    }
    template <class T>
    FCC_HD static void dq(T, T dR, T ddR, T, T, T (*out)[3]) {
        const T s = sqrt(dR * dR + ddR * ddR);
        out[0][0] = T(0);
        out[0][1] = dR / s;
        out[0][2] = ddR / s;
    }
};
}  // namespace fcc_user

// the table the kernels dispatch on, with one term more
#undef FCC_USER_BODY_TERMS
#define FCC_USER_BODY_TERMS(X) X(0, Bending) X(1, ShapeIndexElasticity) X(2, Kink)

#include "../fouriercontourcells.jl_b200/csrc/fcc_kernels.cuh"

#include <vector>

using namespace fcc;

namespace {
template <class V>
struct Dev {  // a host array's copy on the device
    V* p = nullptr;
    size_t n;
    cudaError_t e;
    Dev(const V* h, size_t n_) : n(n_) {
        e = cudaMalloc(&p, n * sizeof(V));
        if (e == cudaSuccess) e = cudaMemcpy(p, h, n * sizeof(V), cudaMemcpyHostToDevice);
    }
    ~Dev() { cudaFree(p); }
    cudaError_t back(V* h) { return cudaMemcpy(h, p, n * sizeof(V), cudaMemcpyDeviceToHost); }
};
#define TRY(x)                                 \
    do {                                       \
        const cudaError_t e_ = (x);            \
        if (e_ != cudaSuccess) return (int)e_; \
    } while (0)

// Node gradients that body term 2 adds on one warp of 4 bodies, 5 slots a lane
__global__ void k_user_gradients(SimDesc<double>* P, int nth, const double* R, const double* R1, const double* R2,
                                 double w, double* GR, double* GD, double* GDD) {
    const int t = threadIdx.x, l = t & 7;
    double r[5], r1[5], r2[5], gr[5], gd[5], gdd[5];
    unsigned vmask = 0;
    for (int s = 0; s < 5; ++s) {
        const bool v = l + 8 * s < nth;
        vmask |= v ? 1u << s : 0u;
        r[s] = v ? R[5 * t + s] : 0.0;  // beyond the contour as the force evaluation leaves them
        r1[s] = v ? R1[5 * t + s] : 0.0;
        r2[s] = v ? R2[5 * t + s] : 0.0;
        gr[s] = gd[s] = gdd[s] = 0.0;
    }
    UserBody<double> u;
    u.integrals<8, 5>(*P, 0, vmask, r, r1, r2, P->dphi);
    for (int k = 0; k < MUT; ++k)
        for (int j = 0; j < fcc_user::MAX_M; ++j) u.w[k][j] = w;
    u.gradients(*P, 0, vmask, r, r1, r2, gr, gd, gdd);
    for (int s = 0; s < 5; ++s) GR[5 * t + s] = gr[s], GD[5 * t + s] = gd[s], GDD[5 * t + s] = gdd[s];
}
__global__ void k_roots(const double* x, int n, double* inv, double* root) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    inv[i] = rsqrt_normal(x[i]);
    root[i] = sqrt_normal(x[i]);
}
}  // namespace

extern "C" int unit_roots(const double* x, int n, double* inv, double* root) {
    Dev<double> dx(x, n), di(inv, n), dr(root, n);
    for (cudaError_t e : {dx.e, di.e, dr.e}) TRY(e);
    k_roots<<<(n + 255) / 256, 256>>>(dx.p, n, di.p, dr.p);
    TRY(cudaGetLastError());
    TRY(di.back(inv));
    return (int)dr.back(root);
}

// k_init of n bodies in a grid of `cells` cells; count[cells] and total[ranges]
// as the launch finds and leaves them
extern "C" int unit_init_counts(int n, int cells, int* count, int* total) {
    SimDesc<double> h{};
    h.K = KM;
    h.n = n;
    h.ncells = cells;
    for (int t = 0; t < MT; ++t) h.kmax[t] = KM;
    const std::vector<double> zero((size_t)n * RECW, 0.0), one(n, 1.0);
    const std::vector<int> izero(n, 0);
    Dev<SimDesc<double>> P(&h, 1);
    Dev<double> rec0(zero.data(), (size_t)n * RECW), rec1(zero.data(), (size_t)n * RECW),
        coef(zero.data(), (size_t)n * NCM), in(zero.data(), (size_t)n * NCM), x(zero.data(), n), r0(one.data(), n);
    Dev<int> sim_of(izero.data(), n), w(izero.data(), n), c(count, cells), t(total, (cells + SCAN_RANGE - 1) / SCAN_RANGE);
    for (cudaError_t e : {P.e, rec0.e, rec1.e, coef.e, in.e, x.e, r0.e, sim_of.e, w.e, c.e, t.e}) TRY(e);
    DevPtrs<double> d{};
    d.sims = P.p;
    d.nsims = 1;
    d.Ntot = n;
    d.Ctot = cells;
    d.sim_of = sim_of.p;
    d.rec0 = rec0.p;
    d.rec1 = rec1.p;
    d.coef = coef.p;
    d.R0 = r0.p;
    d.ccount = c.p;
    d.ctot = t.p;
    k_init<double><<<(n + INIT_BODIES - 1) / INIT_BODIES, INIT_BLOCK, init_smem_bytes(NCM)>>>(
        d, 0, 0, n, x.p, x.p, x.p, in.p, NCM, KM, w.p, nullptr, nullptr);
    TRY(cudaGetLastError());
    TRY(c.back(count));
    return (int)t.back(total);
}

extern "C" int unit_user_gradients(int nth, const double* R, const double* R1, const double* R2, double w, double* GR,
                                   double* GD, double* GDD) {
    SimDesc<double> h{};
    h.nth = nth;
    h.dphi = 6.283185307179586 / nth;
    h.nub = 1;
    h.ub_id[0] = 2;
    h.ub_mask[0] = 1;
    Dev<SimDesc<double>> P(&h, 1);
    Dev<double> r(R, 160), r1(R1, 160), r2(R2, 160), gr(GR, 160), gd(GD, 160), gdd(GDD, 160);
    for (cudaError_t e : {P.e, r.e, r1.e, r2.e, gr.e, gd.e, gdd.e}) TRY(e);
    k_user_gradients<<<1, 32>>>(P.p, nth, r.p, r1.p, r2.p, w, gr.p, gd.p, gdd.p);
    TRY(cudaGetLastError());
    TRY(gr.back(GR));
    TRY(gd.back(GD));
    return (int)gdd.back(GDD);
}
