// Adjoint of the hierarchical recomposition (sm_103a).
//
// The retrieval's recomposition is a linear map R from the packed level
// coefficients (level 0 box, then box(l) \ box(l-1) of every level in
// interleaved order, the layout of the device coefficient buffer) to the
// natural-order field. One level is
//   V(x) = C(c)                     at the coarse node x = fine(c)
//   V(x) = coef(x) + sum_corners w C at every other node (w = 2^-#odd dims)
// so its transpose, applied to a field gradient G, is
//   g_coef(x) = G(x)                                    (a gather by rank)
//   g_C(c)    = sum_{d in {-1,0,1}^3} 2^-|d| G(fine(c) + d)
// where each nonzero offset must land on an odd (non-coarse) node, whose
// interpolation then has fine(c) as one of its corners. Each output is
// written by exactly one thread, in a fixed summation order, so the result
// is deterministic. Levels run fine -> coarse through two ping-pong boxes.
#include "common.cuh"
#include "kernels.cuh"
#include "rows.cuh"

namespace prodm {

namespace {

// Both outputs of one level in one pass: a warp takes coarse columns c = 32 g +
// lane of the coarse rows (i, b) for kPatchSteps consecutive b. The 27-point
// sum is taken dim by dim: a fine row's h = G(even) + (G(left odd) + G(right
// odd)) / 2, three rows along dim 1 (the odd ones between b and b + 1 carry
// over), then three along dim 0. The rows x0 = fine(i) and the odd one behind
// it also leave their coefficient gradients; the odd one before it belongs to
// i - 1. The lone columns of a row (even node only) are taken by the lanes
// that hold them, or by items of their own where the last group has no lane
// left (a lane per b). Each step's loads are issued a step ahead of their use.
// One pass reads the level about 1.5 times (the odd rows of dim 0 twice, from
// L2) and needs no 64-bit divisions per node: 257^3 fp32, finest level 139 us
// with a thread per node in two passes, 33 us this way.
__host__ __device__ inline uint32_t adj_groups(uint32_t P) { return P ? (P + 31) >> 5 : 0; }
// items: per (i, strip) the column groups; then, where columns are left over,
// per i ceil(C1 / 32) items of 32 rows
__host__ __device__ inline uint64_t adj_items(const Box& F, const Box& C, uint64_t& body) {
    const uint32_t groups = adj_groups(F.n[2] - C.n[2]);
    body = (uint64_t)C.n[0] * ((C.n[1] + kPatchSteps - 1) / kPatchSteps) * groups;
    return body + (32 * groups < C.n[2] ? (uint64_t)C.n[0] * ((C.n[1] + 31) / 32) : 0);
}

__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// The sum at the coarse node *p with each of the up to 27 values weighted before
// it is added, node by node: for where the dim-by-dim sum, whose pairs are added
// before they are halved, is not finite. have: odd nodes before (even bits) and
// behind (odd bits) it, dims 0, 1, 2.
template <class T>
__device__ __noinline__ T adj_sum_ordered(const T* __restrict__ p, int64_t s0, int64_t s1, uint32_t have) {
    T acc = 0;
    for (int a = 0; a < 3; a++) {
        if (a && !(have >> (a - 1) & 1u)) continue;
        for (int b = 0; b < 3; b++) {
            if (b && !(have >> (b + 1) & 1u)) continue;
            for (int c = 0; c < 3; c++) {
                if (c && !(have >> (c + 3) & 1u)) continue;
                const T w = (a ? (T)0.5 : (T)1) * (b ? (T)0.5 : (T)1) * (c ? (T)0.5 : (T)1);
                const int64_t at = (a ? 2 * a - 3 : 0) * s0 + (b ? 2 * b - 3 : 0) * s1 + (c ? 2 * c - 3 : 0);
                acc += w * p[at];
            }
        }
    }
    return acc;
}

template <class T, bool COEF>
__device__ __forceinline__ void adj_patch_item(const T* __restrict__ g, const Box& F, const Box& C,
                                               T* __restrict__ gcoef, T* __restrict__ gc, uint64_t item, uint32_t lane) {
    const uint32_t C1 = C.n[1], C2 = C.n[2], O0 = F.n[0] - C.n[0], O1 = F.n[1] - C1, P = F.n[2] - C2;
    const uint32_t groups = adj_groups(P), nstrip = (C1 + kPatchSteps - 1) / kPatchSteps;
    const uint32_t c = 32 * (uint32_t)(item % groups) + lane;
    const uint64_t r = item / groups;
    const uint32_t i = (uint32_t)(r / nstrip), b0 = (uint32_t)(r % nstrip) * kPatchSteps;
    const uint32_t b1 = min(b0 + kPatchSteps, C1);
    const bool ld = c < C2, pair = c < P, first = lane == 0 && c > 0;
    const uint64_t s0 = (uint64_t)F.n[1] * F.n[2], s1 = F.n[2];
    const uint32_t xc = min(2 * c, F.n[2] - 1);
    const bool before = i >= 1 && i - 1 < O0, behind = i < O0;   // odd rows of dim 0 on either side
    const T* mid = g + (uint64_t)min(2 * i, F.n[0] - 1) * s0;
    struct Row { T e, o, l; };   // even node, odd node behind it, (lane 0) odd node before it
    auto load = [&](const T* plane, bool on, uint32_t x1, Row& w) {
        const T* p = plane + (uint64_t)x1 * s1 + xc;
        w.e = on && ld ? __ldg(p) : (T)0;
        w.o = on && pair ? __ldg(p + 1) : (T)0;
        w.l = on && first ? __ldg(p - 1) : (T)0;
    };
    auto sum = [&](const Row& w) {
        T l = __shfl_up_sync(0xffffffffu, w.o, 1);
        if (lane == 0) l = w.l;
        return w.e + (T)0.5 * (l + w.o);
    };
    struct Step { Row me, mo, ae, ao, be, bo; };   // rows x1 = fine(b), 2b + 1 of the three planes
    auto load_step = [&](uint32_t b, Step& s) {
        const uint32_t x1 = min(2 * b, F.n[1] - 1);
        const bool odd = b < O1;
        load(mid, true, x1, s.me);
        load(mid, odd, x1 + 1, s.mo);
        load(mid - s0, before, x1, s.ae);
        load(mid - s0, before && odd, x1 + 1, s.ao);
        load(mid + s0, behind, x1, s.be);
        load(mid + s0, behind && odd, x1 + 1, s.bo);
    };
    T lm = 0, la = 0, lb = 0;   // sums of the odd rows 2b - 1
    if (b0 >= 1 && b0 - 1 < O1) {
        Row w;
        load(mid, true, 2 * b0 - 1, w);
        lm = sum(w);
        load(mid - s0, before, 2 * b0 - 1, w);
        la = sum(w);
        load(mid + s0, behind, 2 * b0 - 1, w);
        lb = sum(w);
    }
    Step S;
    load_step(b0, S);
    bool bad = false;
    for (uint32_t b = b0; b < b1; b++) {
        Step N = S;
        if (b + 1 < b1) load_step(b + 1, N);
        const T hm = sum(S.me), om = sum(S.mo), ha = sum(S.ae), oa = sum(S.ao), hb = sum(S.be), ob = sum(S.bo);
        const T m = hm + (T)0.5 * (lm + om), a = ha + (T)0.5 * (la + oa), d = hb + (T)0.5 * (lb + ob);
        const T v = m + (T)0.5 * (a + d);
        if (ld) gc[((uint64_t)i * C1 + b) * C2 + c] = v;
        bad |= not_finite(v);
        if (COEF) {
            const bool odd = b < O1;
            const uint64_t r00 = level_rank(i, b, C2, F, C);   // even-even row: odd nodes only
            if (pair) gcoef[r00 + c] = S.me.o;
            if (odd) {
                T* q = gcoef + level_rank(i, C1 + b, 0, F, C);
                if (ld) q[c] = S.mo.e;
                if (pair) q[C2 + c] = S.mo.o;
            }
            if (behind) {
                T* q = gcoef + level_rank(C.n[0] + i, b, 0, F, C);
                if (ld) q[c] = S.be.e;
                if (pair) q[C2 + c] = S.be.o;
                if (odd) {
                    q = gcoef + level_rank(C.n[0] + i, C1 + b, 0, F, C);
                    if (ld) q[c] = S.bo.e;
                    if (pair) q[C2 + c] = S.bo.o;
                }
            }
        }
        lm = om;
        la = oa;
        lb = ob;
        S = N;
    }
    if (bad && ld)
        for (uint32_t b = b0; b < b1; b++) {
            T* v = gc + ((uint64_t)i * C1 + b) * C2 + c;
            if (not_finite(*v))
                *v = adj_sum_ordered(mid + (uint64_t)min(2 * b, F.n[1] - 1) * s1 + xc, (int64_t)s0, (int64_t)s1,
                                     (uint32_t)before | behind << 1 | (b >= 1 && b - 1 < O1) << 2 | (b < O1) << 3 |
                                         (c >= 1 && c - 1 < P) << 4 | (uint32_t)pair << 5);
        }
}

// the columns behind the groups (no odd node behind them): a lane per b
template <class T, bool COEF>
__device__ __forceinline__ void adj_lone_item(const T* __restrict__ g, const Box& F, const Box& C,
                                              T* __restrict__ gcoef, T* __restrict__ gc, uint64_t item, uint32_t lane) {
    const uint32_t C1 = C.n[1], C2 = C.n[2], O0 = F.n[0] - C.n[0], O1 = F.n[1] - C1, P = F.n[2] - C2;
    const uint32_t nb = (C1 + 31) / 32, i = (uint32_t)(item / nb), b = (uint32_t)(item % nb) * 32 + lane;
    if (b >= C1) return;
    const uint64_t s0 = (uint64_t)F.n[1] * F.n[2], s1 = F.n[2];
    const uint32_t x1 = min(2 * b, F.n[1] - 1);
    const bool before = i >= 1 && i - 1 < O0, behind = i < O0, odd = b < O1, left = b >= 1 && b - 1 < O1;
    const T* mid = g + (uint64_t)min(2 * i, F.n[0] - 1) * s0;
    for (uint32_t c = 32 * adj_groups(P); c < C2; c++) {
        const uint32_t xc = min(2 * c, F.n[2] - 1);
        const bool lo = c >= 1 && c - 1 < P;   // the odd node before it
        auto row = [&](const T* plane, bool on, uint32_t y) {
            if (!on) return (T)0;
            const T* p = plane + (uint64_t)y * s1 + xc;
            return p[0] + (T)0.5 * (lo ? p[-1] : (T)0);
        };
        auto three = [&](const T* plane, bool on) {
            return row(plane, on, x1) + (T)0.5 * (row(plane, on && left, x1 - 1) + row(plane, on && odd, x1 + 1));
        };
        const T m = three(mid, true), a = three(mid - s0, before), d = three(mid + s0, behind);
        T v = m + (T)0.5 * (a + d);
        if (not_finite(v))
            v = adj_sum_ordered(mid + (uint64_t)x1 * s1 + xc, (int64_t)s0, (int64_t)s1,
                                (uint32_t)before | behind << 1 | left << 2 | odd << 3 | lo << 4);
        gc[((uint64_t)i * C1 + b) * C2 + c] = v;
        if (COEF) {
            const T* p = mid + (uint64_t)x1 * s1 + xc;
            if (odd) gcoef[level_rank(i, C1 + b, 0, F, C) + c] = p[s1];
            if (behind) {
                gcoef[level_rank(C.n[0] + i, b, 0, F, C) + c] = p[s0];
                if (odd) gcoef[level_rank(C.n[0] + i, C1 + b, 0, F, C) + c] = p[s0 + s1];
            }
        }
    }
}

// (one-warp blocks: 257^3 fp32 31.9 us for the finest level, 33.8 in blocks of eight)
template <class T, bool COEF>
__global__ void __launch_bounds__(32, 16) k_adj_level(const T* __restrict__ g, Box F, Box C, T* __restrict__ gcoef,
                                                      T* __restrict__ gc) {
    pdl_wait();   // the gradient comes from the previous launch
    pdl_release();
    uint64_t body;
    const uint64_t items = adj_items(F, C, body);
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint64_t w = (uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < items; w += (uint64_t)gridDim.x * wpb) {
        if (w < body) adj_patch_item<T, COEF>(g, F, C, gcoef, gc, w, lane);
        else adj_lone_item<T, COEF>(g, F, C, gcoef, gc, w - body, lane);
    }
}

template <class T, bool COEF>
int launch_adj_level(const T* g, const Box& F, const Box& C, T* gcoef, T* gc, cudaStream_t st) {
    uint64_t body;
    const uint64_t need = adj_items(F, C, body);
    const unsigned grid = persistent_grid_for((const void*)k_adj_level<T, COEF>, 32, 0, need, need);
    count_launch();
    const cudaError_t e = launch_chain(true, k_adj_level<T, COEF>, dim3(grid), dim3(32), 0, st, g, F, C, gcoef, gc);
    if (e != cudaSuccess) return cuda_status(e, "k_adj_level");
    return PRODM_OK;
}

// ---------------------------------------------------------------------------
// Orthogonal basis. Its recomposition of one level first removes the L2
// correction from the coarse box, C' = C - Q f (f: the level's coefficients on
// the fine box, zero at the coarse-box nodes; Q = Q0 Q1 Q2, one line operator
// per dim, Qd = Mc^-1 R Mf: fine P1 mass matrix, restriction with weights 1
// and 1/2, coarse mass-matrix solve), then interpolates as the hierarchical
// basis. So its transpose takes g_C = g_C' and g_f = g_f(hier) - Q^T g_C',
// Q^T = Q2^T Q1^T Q0^T with Qd^T = Mf R^T Mc^-1 (both mass matrices are
// symmetric): per dim, a tridiagonal solve on the coarse lines, then the
// interpolation (R^T) and the fine mass matrix on the fine lines.
// ---------------------------------------------------------------------------

// the lines of a box along dim d: line li -> (p, q) over the two other dims,
// consecutive li on the faster one (coalesced across a warp)
__device__ __forceinline__ void line_origin(const Box& S, int d, uint64_t li, uint64_t& off_s, const Box& D,
                                            uint64_t& off_d) {
    const int o1 = d == 0 ? 1 : 0, o2 = d == 2 ? 1 : 2;
    const uint64_t ss[3] = {(uint64_t)S.n[1] * S.n[2], S.n[2], 1};
    const uint64_t ds[3] = {(uint64_t)D.n[1] * D.n[2], D.n[2], 1};
    const uint32_t q = (uint32_t)(li % S.n[o2]);
    const uint32_t p = (uint32_t)(li / S.n[o2]);
    off_s = p * ss[o1] + q * ss[o2];
    off_d = p * ds[o1] + q * ds[o2];
}

// u = Mc^-1 y along dim d of box S (coarse length S.n[d]); Thomas factors
// cp / lo_w / inv_den as the forward correction's; u may be y (in place)
template <class T>
__global__ void k_adj_solve(const T* y, Box S, int d, T* u, const T* __restrict__ cp,
                            const T* __restrict__ lo_w, const T* __restrict__ inv_den) {
    const uint32_t nc = S.n[d];
    const uint64_t st = d == 0 ? (uint64_t)S.n[1] * S.n[2] : d == 1 ? S.n[2] : 1;
    const uint64_t lines = S.size() / nc;
    for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < lines;
         li += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t os, od;
        line_origin(S, d, li, os, S, od);
        const T* yl = y + os;
        T* ul = u + os;
        T prev = 0;
        for (uint32_t m = 0; m < nc; m++) {
            const T b = yl[m * st];
            const T dp = (m == 0) ? b * inv_den[0] : (b - lo_w[m] * prev) * inv_den[m];
            ul[m * st] = dp;
            prev = dp;
        }
        T z = ul[(uint64_t)(nc - 1) * st];
        for (uint32_t m = nc - 1; m-- > 0;) {
            z = ul[m * st] - cp[m] * z;
            ul[m * st] = z;
        }
    }
}

// w = Mf R^T u along dim d: u on box S (coarse length nc along d), w on box D
// (fine length nf). v = R^T u is u at the coarse nodes and the mean of the two
// coarse neighbours at the others; w(x) = dg(x) v(x) + (v(x-1) + v(x+1)) / 6
// (dg = 1/3 at the ends, else 2/3; v = 0 outside). One pass with a window.
template <class T>
__global__ void k_adj_spread(const T* __restrict__ u, Box S, int d, T* __restrict__ w, Box D) {
    const uint32_t nc = S.n[d], nf = D.n[d];
    const uint64_t ss = d == 0 ? (uint64_t)S.n[1] * S.n[2] : d == 1 ? S.n[2] : 1;
    const uint64_t ds = d == 0 ? (uint64_t)D.n[1] * D.n[2] : d == 1 ? D.n[2] : 1;
    const uint64_t lines = S.size() / nc;
    for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < lines;
         li += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t os, od;
        line_origin(S, d, li, os, D, od);
        const T* ul = u + os;
        T* wl = w + od;
        if (nc == nf) {   // no coarse subset along this dim: the operator is the identity
            for (uint32_t x = 0; x < nf; x++) wl[x * ds] = ul[x * ss];
            continue;
        }
        auto v_at = [&](uint32_t x) -> T {   // R^T u at fine node x (0 <= x < nf)
            if (is_coarse(x, nf)) return ul[(uint64_t)reord(x, nf, nc) * ss];
            return (T)0.5 * ul[(uint64_t)reord(x - 1, nf, nc) * ss] + (T)0.5 * ul[(uint64_t)reord(x + 1, nf, nc) * ss];
        };
        T vl = 0, vx = v_at(0);
        for (uint32_t x = 0; x < nf; x++) {
            const T vr = x + 1 < nf ? v_at(x + 1) : (T)0;
            const T dg = (x == 0 || x == nf - 1) ? (T)1 / 3 : (T)2 / 3;
            wl[x * ds] = dg * vx + (vl + vr) / 6;
            vl = vx;
            vx = vr;
        }
    }
}

// gradient of the level-l coefficients with the correction's share removed:
// gcoef(rank(x)) = G(x) - W(x) at every fine node outside the coarse box
template <class T>
__global__ void k_adj_coef_minus(const T* __restrict__ g, const T* __restrict__ wv, Box F, Box C,
                                 T* __restrict__ gcoef) {
    const uint64_t N = F.size();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t x2 = (uint32_t)(i % F.n[2]);
        const uint64_t r = i / F.n[2];
        const uint32_t x1 = (uint32_t)(r % F.n[1]), x0 = (uint32_t)(r / F.n[1]);
        const bool c0 = is_coarse(x0, F.n[0]), c1 = is_coarse(x1, F.n[1]), c2 = is_coarse(x2, F.n[2]);
        if (c0 && c1 && c2) continue;
        const uint64_t rank = level_rank(reord(x0, F.n[0], C.n[0]), reord(x1, F.n[1], C.n[1]),
                                         reord(x2, F.n[2], C.n[2]), F, C);
        gcoef[rank] = g[i] - wv[i];
    }
}

}  // namespace

// transpose of one orthogonal recomposition level: g (box F) -> gcoef (packed
// level coefficients) and gcoarse (box C). tabs[d]: Thomas factors of dim d;
// scratch: boxes (n0, c1, c2), (n0, n1, c2), F and one C box.
template <class T>
int launch_recompose_adjoint_level_orth(const T* g, const Box& F, const Box& C, T* gcoef, T* gcoarse,
                                        const T* const tabs[3], T* s_a, T* s_b, T* s_w, T* s_u, cudaStream_t st) {
    const int th = 256;
    const int rc = launch_adj_level<T, false>(g, F, C, nullptr, gcoarse, st);
    if (rc) return rc;
    // Q0^T, Q1^T, Q2^T: C -> (n0, c1, c2) -> (n0, n1, c2) -> F
    Box a = C;
    const T* src = gcoarse;
    T* outs[3] = {s_a, s_b, s_w};
    for (int d = 0; d < 3; d++) {
        Box b = a;
        b.n[d] = F.n[d];
        const uint32_t nc = a.n[d];
        const uint64_t lines = a.size() / nc;
        if (nc != F.n[d]) {   // in place on the previous scratch box; gcoarse itself stays (it is g_C)
            const T* tab = tabs[d];
            T* u = d == 0 ? s_u : const_cast<T*>(src);
            k_adj_solve<T><<<grid_for(lines, th, 16), th, 0, st>>>(src, a, d, u, tab, tab + nc, tab + 2 * nc);
            PRODM_CHECK_LAUNCH("k_adj_solve");
            src = u;
        }
        k_adj_spread<T><<<grid_for(lines, th, 16), th, 0, st>>>(src, a, d, outs[d], b);
        PRODM_CHECK_LAUNCH("k_adj_spread");
        src = outs[d];
        a = b;
    }
    k_adj_coef_minus<T><<<grid_for(F.size(), th), th, 0, st>>>(g, s_w, F, C, gcoef);
    PRODM_CHECK_LAUNCH("k_adj_coef_minus");
    return PRODM_OK;
}

template int launch_recompose_adjoint_level_orth<float>(const float*, const Box&, const Box&, float*, float*,
                                                        const float* const[3], float*, float*, float*, float*,
                                                        cudaStream_t);
template int launch_recompose_adjoint_level_orth<double>(const double*, const Box&, const Box&, double*, double*,
                                                         const double* const[3], double*, double*, double*, double*,
                                                         cudaStream_t);

template <class T>
int launch_recompose_adjoint_level(const T* g, const Box& F, const Box& C, T* gcoef, T* gcoarse, cudaStream_t st) {
    return launch_adj_level<T, true>(g, F, C, gcoef, gcoarse, st);
}

template int launch_recompose_adjoint_level<float>(const float*, const Box&, const Box&, float*, float*, cudaStream_t);
template int launch_recompose_adjoint_level<double>(const double*, const Box&, const Box&, double*, double*,
                                                    cudaStream_t);

}  // namespace prodm
