// GE quantities of interest on the device (sm_103a): values and pointwise
// error estimates for the QoI-bounded retrieval drivers.
//
// Values: V_TOT = |V|, T = P / (D R), C = sqrt(gamma R T), Mach = V_TOT / C,
// PT = P (1 + (gamma - 1) / 2 Mach^2)^(7/2), mu = mu_r (T / T_r)^(3/2)
// (T_r + S) / (T + S), in double as qoi_utils.hpp:135-165 computes them;
// the reference's pow(x, 7) and pow(x, 3) are multiplication chains here.
// Estimates (qoi_utils.hpp:18-98): |V_TOT~ - V_TOT| <= sqrt-rule(V^2,
// sum_f square-rule(V_f, eb_f)) as halving_Vtot.cpp:38-45 forms it, and
// |T~ - T| <= division-rule(P, D, eb_P, eb_D) / R (0 where the rule gives no
// bound, as the reference does). The FP64 pipe bounds both kernels, and three
// quarters of its work were four divisions and four roots a point (values; two
// and two for the estimates): they are made of integer operations (exact64.cuh)
// with the same bits, comparisons too, and so are as many products as balance
// the two kinds of pipe: three of the values' fourteen, six of the estimates'
// ten. 257^3 points: values 2574 -> 704 us, 633 with the products (three more
// 681, six more 740), estimates 1951 -> 840, 656 with them (none of them 840,
// three 747, nine 649); DRAM floor 224 and 143 us. One thread per point,
// streaming; the
// maxima over the field are reduced with 64-bit atomicMax on the (non-
// negative) doubles' bit patterns.
#include "common.cuh"
#include "exact64.cuh"
#include "kernels.cuh"

namespace prodm {
namespace {

struct Ge {
    static constexpr double R = 287.1, gamma = 1.4, mu_r = 1.716e-5, T_r = 273.15, S = 110.4;
};

// uncontracted, operation by operation as the host evaluates the rules; eb2 = eb * eb
__device__ __forceinline__ double bx2(double x, double eb, double eb2) {
    return __dadd_rn(mul_exact(twice_abs(x), eb), eb2);
}
__device__ __forceinline__ double bsqrt(double x, double eb) {   // x, eb >= +0 or NaN
    const bool zero = bits64(x) == 0;
    double r = sqrt_exact(zero ? eb : x);
    if (zero) return r;
    if (above(x, eb)) r = __dadd_rn(sqrt_exact(__dsub_rn(x, eb)), r);
    return div_exact(eb, r);
}
__device__ __forceinline__ double bdiv(double x, double y, double ebx, double eby) {   // eby >= +0 or NaN
    const double ay = fabs(y);
    if (above(ay, eby))   // (y (y - eby), or for y < 0 y (y + eby))
        return div_exact(__dadd_rn(__dmul_rn(fabs(x), eby), __dmul_rn(ay, ebx)), __dmul_rn(ay, __dsub_rn(ay, eby)));
    return 0;
}

__global__ void k_qoi_values(const double* __restrict__ vx, const double* __restrict__ vy,
                             const double* __restrict__ vz, const double* __restrict__ p,
                             const double* __restrict__ d, uint64_t n, double* __restrict__ vtot,
                             double* __restrict__ temp, double* __restrict__ cs, double* __restrict__ mach,
                             double* __restrict__ pt, double* __restrict__ mu) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double v2 = __dadd_rn(__dadd_rn(__dmul_rn(vx[i], vx[i]), __dmul_rn(vy[i], vy[i])), __dmul_rn(vz[i], vz[i]));
        const double v = sqrt_exact(v2);
        const double t = div_exact(p[i], mul_exact(d[i], Ge::R));
        const double c = sqrt_exact(mul_exact(__dmul_rn(Ge::gamma, Ge::R), t));
        const double m = div_exact(v, c);
        const double mt = __dadd_rn(1.0, __dmul_rn(__dmul_rn((Ge::gamma - 1) / 2, m), m));
        // x^7 and x^3 by multiplication chains instead of pow (GB300's FP64
        // pipe is slow; the chains stay within a few units in the last place)
        const double mt2 = __dmul_rn(mt, mt), mt4 = __dmul_rn(mt2, mt2);
        const double ptv = mul_exact(p[i], sqrt_exact(__dmul_rn(__dmul_rn(mt4, mt2), mt)));
        const double trs = div_exact(Ge::T_r + Ge::S, __dadd_rn(t, Ge::S));
        const double tr = div_exact(t, Ge::T_r);
        const double tt3 = sqrt_exact(__dmul_rn(__dmul_rn(tr, tr), tr));
        vtot[i] = v;
        temp[i] = t;
        cs[i] = c;
        mach[i] = m;
        pt[i] = ptv;
        mu[i] = __dmul_rn(__dmul_rn(Ge::mu_r, tt3), trs);
    }
}

__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
    atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

// the larger of e and m, m where e is NaN; both >= +0 otherwise
__device__ __forceinline__ double max_of(double e, double m) {
    return bits64(e) <= kInfBits ? __longlong_as_double((long long)max_key(bits64(e), bits64(m))) : m;
}

__global__ void k_qoi_bounds(const double* __restrict__ vx, const double* __restrict__ vy,
                             const double* __restrict__ vz, const double* __restrict__ p,
                             const double* __restrict__ d, uint64_t n, double ebx, double eby, double ebz, double ebp,
                             double ebd, double* __restrict__ bv, double* __restrict__ bt, double* __restrict__ mx) {
    double mv = 0, mt = 0;
    ebd += 0.0;   // (-0 to +0)
    const double ebx2 = __dmul_rn(ebx, ebx), eby2 = __dmul_rn(eby, eby), ebz2 = __dmul_rn(ebz, ebz);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (vx) {
            const double x = vx[i], y = vy[i], z = vz[i];
            const double e2 = __dadd_rn(__dadd_rn(bx2(x, ebx, ebx2), bx2(y, eby, eby2)), bx2(z, ebz, ebz2));
            const double v2 = __dadd_rn(__dadd_rn(mul_exact(x, x), mul_exact(y, y)), mul_exact(z, z));
            const double e = bsqrt(v2, e2);
            if (bv) bv[i] = e;
            mv = max_of(e, mv);
        }
        if (p) {
            const double e = __dmul_rn(1.0 / Ge::R, bdiv(p[i], d[i], ebp, ebd));
            if (bt) bt[i] = e;
            mt = max_of(e, mt);
        }
    }
    if (mx) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, mv, o), ot = __shfl_xor_sync(0xffffffffu, mt, o);
            mv = max_of(ov, mv);
            mt = max_of(ot, mt);
        }
        if ((threadIdx.x & 31) == 0) {
            atomic_max_nonneg(mx, mv);
            atomic_max_nonneg(mx + 1, mt);
        }
    }
}

}  // namespace
}  // namespace prodm

using namespace prodm;

extern "C" {

int prodm_qoi_ge_values(int dtype, const void* vx, const void* vy, const void* vz, const void* p, const void* d,
                        uint64_t n, void* vtot, void* temp, void* c, void* mach, void* pt, void* mu, void* stream) {
    if (dtype != PRODM_F64) return fail(PRODM_EUNSUPPORTED, "prodm_qoi_ge_values: fp64 fields only");
    if (!vx || !vy || !vz || !p || !d || !vtot || !temp || !c || !mach || !pt || !mu)
        return fail(PRODM_EINVAL, "prodm_qoi_ge_values: NULL pointer");
    if (n == 0) return PRODM_OK;
    k_qoi_values<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        (const double*)vx, (const double*)vy, (const double*)vz, (const double*)p, (const double*)d, n,
        (double*)vtot, (double*)temp, (double*)c, (double*)mach, (double*)pt, (double*)mu);
    PRODM_CHECK_LAUNCH("k_qoi_values");
    return PRODM_OK;
}

int prodm_qoi_ge_bounds(int dtype, const void* vx, const void* vy, const void* vz, const void* p, const void* d,
                        uint64_t n, double eb_vx, double eb_vy, double eb_vz, double eb_p, double eb_d,
                        double* bound_vtot, double* bound_t, double* max_bounds, void* stream) {
    if (dtype != PRODM_F64) return fail(PRODM_EUNSUPPORTED, "prodm_qoi_ge_bounds: fp64 fields only");
    const bool v = vx && vy && vz, t = p && d;
    if (!v && !t) return fail(PRODM_EINVAL, "prodm_qoi_ge_bounds: give the velocity fields, or P and D");
    if ((vx || vy || vz) && !v) return fail(PRODM_EINVAL, "prodm_qoi_ge_bounds: all three velocity fields are needed");
    if ((p || d) && !t) return fail(PRODM_EINVAL, "prodm_qoi_ge_bounds: P and D are needed together");
    if (eb_vx < 0 || eb_vy < 0 || eb_vz < 0 || eb_p < 0 || eb_d < 0)
        return fail(PRODM_EINVAL, "prodm_qoi_ge_bounds: error bounds must be non-negative");
    cudaStream_t st = (cudaStream_t)stream;
    if (max_bounds) PRODM_CUDA(cudaMemsetAsync(max_bounds, 0, 2 * sizeof(double), st));
    if (n == 0) return PRODM_OK;
    k_qoi_bounds<<<grid_for(n, 256), 256, 0, st>>>(
        v ? (const double*)vx : nullptr, (const double*)vy, (const double*)vz, t ? (const double*)p : nullptr,
        (const double*)d, n, eb_vx, eb_vy, eb_vz, eb_p, eb_d, bound_vtot, bound_t, max_bounds);
    PRODM_CHECK_LAUNCH("k_qoi_bounds");
    return PRODM_OK;
}

}  // extern "C"
