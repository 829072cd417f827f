// MGARD multilevel decomposition / recomposition kernels (sm_103a).
//
// One level maps the nodal values on a fine box F to
//   * coefficients c(x) = u(x) - (multilinear interpolant of the coarse nodal
//     values)(x) at every non-coarse node, and
//   * the coarse nodal values (orthogonal basis: plus the L2-projection
//     correction z = (M_c^-1 P^T M_f)^{(x)3} c, solved per dim with Thomas).
// Per dim the coarse nodes are the even indices below n-1 plus n-1
// ((n >> 1) + 1 of them, RefactorUtils.hpp:21-34). The reference obtains this
// transform from MGARDx (MGARD.hpp:14-66); MGARDx is not part of the reference
// tree, so the arithmetic here follows the published MGARD method.
//
// Two layouts are supported:
//  * packed   -- level coefficients in interleaved order (the order
//                DirectInterleaver.hpp:23-31 produces) plus a compact coarse
//                box; used by the device-resident pipeline, which never
//                materialises the in-place layout;
//  * in place -- the reference layout: the level box of a strided array,
//                reordered per dim so that coarse nodes come first
//                (DecomposerInterface.hpp:14-16).
#include <cstdlib>

#include "common.cuh"
#include "kernels.cuh"
#include "rows.cuh"

namespace prodm {

namespace {

// Multilinear interpolation at fine node (x0,x1,x2) from its corner values,
// dims averaged with dim 0 outermost (the oracle uses the same order).
template <class T, class Get>
__device__ __forceinline__ T interp(int mask, Get at) {
    auto avg = [&](T a, T b) { return avg_rn(a, b); };
    switch (mask) {
        case 1: return avg(at(-1, 0, 0), at(1, 0, 0));
        case 2: return avg(at(0, -1, 0), at(0, 1, 0));
        case 4: return avg(at(0, 0, -1), at(0, 0, 1));
        case 3: return avg(avg(at(-1, -1, 0), at(-1, 1, 0)), avg(at(1, -1, 0), at(1, 1, 0)));
        case 5: return avg(avg(at(-1, 0, -1), at(-1, 0, 1)), avg(at(1, 0, -1), at(1, 0, 1)));
        case 6: return avg(avg(at(0, -1, -1), at(0, -1, 1)), avg(at(0, 1, -1), at(0, 1, 1)));
        case 7: {
            T a = avg(avg(at(-1, -1, -1), at(-1, -1, 1)), avg(at(-1, 1, -1), at(-1, 1, 1)));
            T b = avg(avg(at(1, -1, -1), at(1, -1, 1)), avg(at(1, 1, -1), at(1, 1, 1)));
            return avg(a, b);
        }
        default: return (T)0;
    }
}

// ---------------------------------------------------------------------------
// forward level by elements: in = compact natural-order fine box; out = its
// reordered positions (strides o0, o1, 1), coarse values in the corner
// fnat (optional): natural-order coefficient field, zero at coarse nodes
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_decompose_level(const T* __restrict__ in, Box F, Box C, T* __restrict__ out, uint64_t o0, uint64_t o1,
                                  T* __restrict__ fnat) {
    const uint64_t total = F.size(), s0 = (uint64_t)F.n[1] * F.n[2], s1 = F.n[2];
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, F, x0, x1, x2);
        const T* p = in + idx;
        T v = *p;
        int mask = (is_coarse(x0, F.n[0]) ? 0 : 1) | (is_coarse(x1, F.n[1]) ? 0 : 2) | (is_coarse(x2, F.n[2]) ? 0 : 4);
        uint32_t r0 = reord(x0, F.n[0], C.n[0]), r1 = reord(x1, F.n[1], C.n[1]), r2 = reord(x2, F.n[2], C.n[2]);
        if (mask) {
            auto at = [&](int d0, int d1, int d2) -> T { return __ldg(p + (int64_t)d0 * (int64_t)s0 + (int64_t)d1 * (int64_t)s1 + d2); };
            v = sub_rn(v, interp<T>(mask, at));
        }
        out[r0 * o0 + r1 * o1 + r2] = v;
        if (fnat) fnat[idx] = mask ? v : (T)0;
    }
}

// ---------------------------------------------------------------------------
// inverse level by elements: rin = compact reordered copy of the level box, its
// coarse corner nodal values (already corrected for the orthogonal basis) ->
// natural-order fine box
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_recompose_level(const T* __restrict__ rin, Box F, Box C, T* __restrict__ out, uint64_t s0,
                                  uint64_t s1) {
    const uint64_t total = F.size(), fs0 = (uint64_t)F.n[1] * F.n[2], fs1 = F.n[2];
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, F, x0, x1, x2);
        int mask = (is_coarse(x0, F.n[0]) ? 0 : 1) | (is_coarse(x1, F.n[1]) ? 0 : 2) | (is_coarse(x2, F.n[2]) ? 0 : 4);
        // coarse-index coordinates of the "low" corner
        uint32_t c0 = (mask & 1) ? (x0 >> 1) : reord(x0, F.n[0], C.n[0]);
        uint32_t c1 = (mask & 2) ? (x1 >> 1) : reord(x1, F.n[1], C.n[1]);
        uint32_t c2 = (mask & 4) ? (x2 >> 1) : reord(x2, F.n[2], C.n[2]);
        const T* cb = rin + c0 * fs0 + c1 * fs1 + c2;
        T v;
        if (mask == 0) {
            v = *cb;
        } else {
            // corner offsets: -1 -> low corner (0), +1 -> next coarse node (1)
            auto at = [&](int d0, int d1, int d2) -> T {
                return __ldg(cb + (d0 > 0 ? fs0 : 0) + (d1 > 0 ? fs1 : 0) + (d2 > 0 ? 1 : 0));
            };
            uint32_t r0 = reord(x0, F.n[0], C.n[0]), r1 = reord(x1, F.n[1], C.n[1]), r2 = reord(x2, F.n[2], C.n[2]);
            v = add_rn(rin[r0 * fs0 + r1 * fs1 + r2], interp<T>(mask, at));
        }
        out[x0 * s0 + x1 * s1 + x2] = v;
    }
}

// ---------------------------------------------------------------------------
// Row-parallel forms used by the device pipeline (packed layout). One CTA
// walks fine rows (x0, x1); threads stride along x2, so loads and stores are
// coalesced and there is no per-element 64-bit division. Same arithmetic
// (and the same uncontracted operation order) as the generic kernels.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) k_decompose_rows(const T* __restrict__ in, uint64_t s0, uint64_t s1, Box F, Box C,
                                                        T* __restrict__ coef, T* __restrict__ coarse,
                                                        T* __restrict__ fnat, typename KeyOf<T>::type* maxkey_level,
                                                        typename KeyOf<T>::type* maxkey_coarse) {
    using K = typename KeyOf<T>::type;
    pdl_wait();   // the level's input comes from the previous launch
    pdl_release();
    K mk = 0, mc = 0;
    const uint32_t rows = F.n[0] * F.n[1];
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint32_t row = blockIdx.x * wpb + (threadIdx.x >> 5); row < rows; row += gridDim.x * wpb)
        decompose_row_any<T>(in, s0, s1, F, C, coef, coarse, fnat, row, lane, mk, mc);
    if (maxkey_level) {
        mk = warp_max_key(mk);
        if ((threadIdx.x & 31) == 0 && mk) atomicMax(maxkey_level, mk);
    }
    if (maxkey_coarse) {
        mc = warp_max_key(mc);
        if ((threadIdx.x & 31) == 0 && mc) atomicMax(maxkey_coarse, mc);
    }
}

// Patch items are long (8 steps) and alike, so they run in one-warp blocks: as
// many warps an SM as the registers allow, each replaced when it ends, where a
// block of eight warps waits for the last of them. 513 x 257 x 257 fp64 finest
// recomposition 192 -> 171 us (64 threads 173, 128 177), decomposition 195 -> 172;
// fp32 about 1 %.
constexpr int kPatchThreads = 32;
template <class T>
constexpr int kPatchBlocks = sizeof(T) == 4 ? 24 : 16;
// patch form (no natural-order copy): one
// warp item = coarse columns 32g .. 32g + 31 of a 2 x 2 kPatchSteps strip of
// fine rows (decompose_patch_item)
template <class T, int PLANE>
__global__ void __launch_bounds__(kPatchThreads, kPatchBlocks<T>) k_decompose_patch(const T* __restrict__ in, uint64_t s0, uint64_t s1, Box F,
                                                         Box C, T* __restrict__ coef, T* __restrict__ coarse,
                                                         typename KeyOf<T>::type* maxkey_level,
                                                         typename KeyOf<T>::type* maxkey_coarse) {
    using K = typename KeyOf<T>::type;
    pdl_wait();   // the level's input comes from the previous launch
    pdl_release();
    K mk = 0, mc = 0;
    const uint64_t items = patch_items(F, C);
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint64_t w = (uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < items; w += (uint64_t)gridDim.x * wpb)
        decompose_patch_item<T, PLANE>(in, s0, s1, F, C, coef, coarse, w, lane, mk, mc);
    if (maxkey_level) {
        mk = warp_max_key(mk);
        if (lane == 0 && mk) atomicMax(maxkey_level, mk);
    }
    if (maxkey_coarse) {
        mc = warp_max_key(mc);
        if (lane == 0 && mc) atomicMax(maxkey_coarse, mc);
    }
}

// patch form of the recomposition (recompose_patch_item), same items as k_decompose_patch
template <class T, int PLANE>
__global__ void __launch_bounds__(kPatchThreads, kPatchBlocks<T>) k_recompose_patch(const T* __restrict__ coarse,
                                                                                  const T* __restrict__ coef, Box F,
                                                                                  Box C, T* __restrict__ out,
                                                                                  uint64_t s0, uint64_t s1) {
    pdl_wait();   // the coarse box and the coefficients come from the previous launches
    pdl_release();
    const uint64_t items = patch_items(F, C);
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint64_t w = (uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < items; w += (uint64_t)gridDim.x * wpb)
        recompose_patch_item<T, PLANE>(coarse, coef, F, C, out, s0, s1, w, lane);
}

// in-place forms of the two (the reordered box instead of packed coefficients)
template <class T>
__global__ void __launch_bounds__(kPatchThreads, kPatchBlocks<T>) k_decompose_patch_inplace(const T* __restrict__ in, Box F,
                                                                                          Box C, T* __restrict__ out,
                                                                                          uint64_t o0, uint64_t o1) {
    typename KeyOf<T>::type mk = 0, mc = 0;
    const uint64_t items = patch_items(F, C);
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint64_t w = (uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < items; w += (uint64_t)gridDim.x * wpb)
        decompose_patch_item<T, 0, true>(in, (uint64_t)F.n[1] * F.n[2], F.n[2], F, C, out, nullptr, w, lane, mk, mc, o0, o1);
}
template <class T>
__global__ void __launch_bounds__(kPatchThreads, kPatchBlocks<T>) k_recompose_patch_inplace(const T* __restrict__ rin, Box F,
                                                                                          Box C, T* __restrict__ out,
                                                                                          uint64_t s0, uint64_t s1) {
    const uint64_t items = patch_items(F, C);
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint64_t w = (uint64_t)blockIdx.x * wpb + (threadIdx.x >> 5); w < items; w += (uint64_t)gridDim.x * wpb)
        recompose_patch_item<T, 0, true>(rin, rin, F, C, out, s0, s1, w, lane);
}

template <class T>
__global__ void __launch_bounds__(256) k_recompose_rows(const T* __restrict__ coarse, const T* __restrict__ coef, Box F,
                                                        Box C, T* __restrict__ out, uint64_t s0, uint64_t s1) {
    pdl_wait();   // the coarse box and the coefficients come from the previous launches
    pdl_release();
    const uint32_t rows = F.n[0] * F.n[1];
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint32_t row = blockIdx.x * wpb + (threadIdx.x >> 5); row < rows; row += gridDim.x * wpb)
        recompose_row_any<T>(coarse, coef, F, C, out, s0, s1, row, lane);
}

// copy a box between strided arrays
template <class T>
__global__ void k_copy_box(const T* __restrict__ src, uint64_t a0, uint64_t a1, Box B, T* __restrict__ dst, uint64_t b0,
                           uint64_t b1) {
    const uint64_t total = B.size();
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, B, x0, x1, x2);
        dst[x0 * b0 + x1 * b1 + x2] = src[x0 * a0 + x1 * a1 + x2];
    }
}

// n values from src to dst by one warp, four in flight per lane
template <class T>
__device__ __forceinline__ void warp_copy(const T* __restrict__ src, T* __restrict__ dst, uint32_t n, uint32_t lane) {
    constexpr int U = 4;
    for (uint32_t x0 = lane; x0 < n; x0 += 32 * U) {
        T v[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (x0 + 32 * u < n) v[u] = src[x0 + 32 * u];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (x0 + 32 * u < n) dst[x0 + 32 * u] = v[u];
    }
}
// the same copy with a warp per row: the coordinates once per row
template <class T>
__global__ void __launch_bounds__(256) k_copy_rows(const T* __restrict__ src, uint64_t a0, uint64_t a1, Box B,
                                                   T* __restrict__ dst, uint64_t b0, uint64_t b1) {
    const uint64_t rows = (uint64_t)B.n[0] * B.n[1], wpb = blockDim.x >> 5;
    for (uint64_t r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
        const uint32_t x0 = (uint32_t)(r / B.n[1]), x1 = (uint32_t)(r - (uint64_t)x0 * B.n[1]);
        warp_copy(src + x0 * a0 + x1 * a1, dst + x0 * b0 + x1 * b1, B.n[2], threadIdx.x & 31);
    }
}

// packed coefficients -> natural-order fine field, zeros at coarse nodes
template <class T>
__global__ void k_coef_to_natural(const T* __restrict__ coef, Box F, Box C, T* __restrict__ fnat) {
    const uint64_t total = F.size();
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, F, x0, x1, x2);
        bool c = is_coarse(x0, F.n[0]) && is_coarse(x1, F.n[1]) && is_coarse(x2, F.n[2]);
        T v = (T)0;
        if (!c) {
            uint32_t r0 = reord(x0, F.n[0], C.n[0]), r1 = reord(x1, F.n[1], C.n[1]), r2 = reord(x2, F.n[2], C.n[2]);
            v = coef[level_rank(r0, r1, r2, F, C)];
        }
        fnat[idx] = v;
    }
}

// in-place reordered level box (compact copy) -> natural coefficient field
template <class T>
__global__ void k_reordered_to_natural(const T* __restrict__ rin, Box F, Box C, T* __restrict__ fnat) {
    const uint64_t total = F.size();
    const uint64_t fs0 = (uint64_t)F.n[1] * F.n[2], fs1 = F.n[2];
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, F, x0, x1, x2);
        bool c = is_coarse(x0, F.n[0]) && is_coarse(x1, F.n[1]) && is_coarse(x2, F.n[2]);
        T v = (T)0;
        if (!c) {
            uint32_t r0 = reord(x0, F.n[0], C.n[0]), r1 = reord(x1, F.n[1], C.n[1]), r2 = reord(x2, F.n[2], C.n[2]);
            v = rin[r0 * fs0 + r1 * fs1 + r2];
        }
        fnat[idx] = v;
    }
}

// Right-hand side of the coarse projection at coarse node m of a line of nf
// fine values: b = (M_f s)[c] + 1/2 (M_f s)[c-1] + 1/2 (M_f s)[c+1] with c
// its fine position, the neighbours only when they are not coarse nodes, and
// (M_f s)[x] = dg(x) s[x] + (s[x-1] + s[x+1]) / 6 (P1 mass matrix, dg = 1/3 at
// the ends, else 2/3; s = 0 outside the line). Window: the fine values at
// c-2 .. c+2. For double data an interior node takes the same sum regrouped as
// one 5-point stencil, 5/6 s[c] + 1/2 (s[c-1] + s[c+1]) + 1/12 (s[c-2] + s[c+2]),
// a third of the FP64 operations; float keeps the term order above.
// INTERIOR: the caller knows that c is an even position in [2, nf - 3]. HALVE:
// halve by the exponent instead of an FP64 operation.
template <class W, bool INTERIOR = false, bool HALVE = false>
__device__ __forceinline__ W l2_rhs(W sm2, W sm1, W s0, W s1, W s2, uint32_t c, uint32_t nf) {
    // fused multiply-adds are written out: which product of a sum the compiler
    // fuses depends on the code around it
    if (sizeof(W) == 8 && (INTERIOR || (c >= 2 && c + 3 <= nf && (c & 1u) == 0)))
        return fma((W)(1.0 / 12.0), sm2 + s2, fma((W)(5.0 / 6.0), s0, HALVE ? (W)half_rn(sm1 + s1) : (W)0.5 * (sm1 + s1)));
    auto mf = [&](W l, W x, W r, uint32_t pos) {
        const W dg = (!INTERIOR && (pos == 0 || pos == nf - 1)) ? (W)1 / 3 : (W)2 / 3;
        return fma(dg, x, (l + r) / 6);
    };
    W b = mf(sm1, s0, s1, c);
    if (INTERIOR || (c > 0 && !is_coarse(c - 1, nf))) b = fma((W)0.5, mf(sm2, sm1, s0, c - 1), b);
    if (INTERIOR || (c + 1 < nf && !is_coarse(c + 1, nf))) b = fma((W)0.5, mf(s0, s1, s2, c + 1), b);
    return b;
}

// One dim of the L2 projection: dst = M_c^-1 P^T M_f src along dim d.
// Thread per line (consecutive threads on consecutive lines of the two
// faster dims, so every access is coalesced across a warp); the fine values
// stream through a 5-value window, the forward sweep stores d'_m in dst, the
// backward sweep substitutes in place. cp / lo_w / inv_den: Thomas factors of
// the coarse mass matrix (length nc, in W). A line is a chain of dependent
// FP64 operations (64 cycles each) whose loads are known in advance, so they
// are issued kLineAhead nodes ahead in both sweeps: with one node ahead, and
// none in the backward sweep, the dim-1 and dim-0 passes of 513 x 513 x 257
// took 414 and 260 us, with four and eight and the right-hand sides of four
// nodes ahead of their chain 325 and 168 us, 272 and 150 with the halving of
// the right-hand side done on the exponent, and 248 and 131 in one-warp blocks
// with twelve nodes back (eight 252 and 135; blocks of two warps 255 and 148;
// FP64 floor 189 and 95).
constexpr int kLineAhead = 4, kLineBack = 12;
template <class T, class W>
__global__ void __launch_bounds__(32, 16) k_l2_line(const T* __restrict__ src, Box S, int d, T* dst, Box D,
                                                 const W* __restrict__ cp, const W* __restrict__ lo_w,
                                                 const W* __restrict__ inv_den) {
    pdl_wait();
    pdl_release();
    const uint32_t nf = S.n[d], nc = D.n[d];
    const int o1 = d == 0 ? 1 : 0, o2 = d == 2 ? 1 : 2;
    const auto stride = [](const Box& B, int k) { return k == 2 ? 1ull : k == 1 ? B.n[2] : (uint64_t)B.n[1] * B.n[2]; };
    const uint64_t st = stride(S, d), dt = stride(D, d);
    const uint64_t lines = (uint64_t)S.n[o1] * S.n[o2];
    for (uint64_t li = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; li < lines;
         li += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t q = (uint32_t)(li % S.n[o2]);
        uint32_t p = (uint32_t)(li / S.n[o2]);
        const T* sl = src + p * stride(S, o1) + q * stride(S, o2);
        T* dl = dst + p * stride(D, o1) + q * stride(D, o2);
        if (nf == nc) {
            for (uint32_t x = 0; x < nf; x++) dl[x * dt] = sl[x * st];
            continue;
        }
        auto at = [&](int64_t x) -> W { return (x >= 0 && x < (int64_t)nf) ? (W)__ldg(sl + x * st) : (W)0; };
        // regular coarse nodes sit at c = 2m; with an even nf the last one is nf - 1
        const uint32_t nreg = (nf & 1u) ? nc : nc - 1;
        W sm2 = 0, sm1 = 0, s0 = at(0), prev = 0;
        W nx[2 * kLineAhead];   // the fine values behind the next node
#pragma unroll
        for (int u = 0; u < 2 * kLineAhead; u++) nx[u] = at(1 + u);
        for (uint32_t m0 = 0; m0 < nreg; m0 += kLineAhead) {
            W w[2 * kLineAhead + 3] = {sm2, sm1, s0};   // the values 2 m0 - 2 .. 2 (m0 + kLineAhead)
#pragma unroll
            for (int u = 0; u < 2 * kLineAhead; u++) {
                w[3 + u] = nx[u];
                nx[u] = at(2 * (int64_t)(m0 + kLineAhead) + 1 + u);
            }
            if (m0 && 2 * (m0 + kLineAhead - 1) + 3 <= nf) {
                W b[kLineAhead], lo[kLineAhead], inv[kLineAhead];
#pragma unroll
                for (int u = 0; u < kLineAhead; u++) {
                    lo[u] = lo_w[m0 + u];
                    inv[u] = inv_den[m0 + u];
                    b[u] = l2_rhs<W, true, true>(w[2 * u], w[2 * u + 1], w[2 * u + 2], w[2 * u + 3], w[2 * u + 4], 2 * (m0 + u), nf);
                }
#pragma unroll
                for (int u = 0; u < kLineAhead; u++) {
                    prev = fma(-lo[u], prev, b[u]) * inv[u];
                    dl[(m0 + u) * dt] = (T)prev;
                }
            } else {
#pragma unroll
                for (int u = 0; u < kLineAhead; u++) {
                    const uint32_t m = m0 + u;
                    if (m < nreg) {
                        const W b = l2_rhs<W>(w[2 * u], w[2 * u + 1], w[2 * u + 2], w[2 * u + 3], w[2 * u + 4], 2 * m, nf);
                        prev = (m == 0) ? b * inv_den[0] : fma(-lo_w[m], prev, b) * inv_den[m];
                        dl[m * dt] = (T)prev;
                    }
                }
            }
            sm2 = w[2 * kLineAhead];
            sm1 = w[2 * kLineAhead + 1];
            s0 = w[2 * kLineAhead + 2];
        }
        if (nreg < nc) {   // even nf: the last coarse node is the last fine node
            const uint32_t c = nf - 1, m = nc - 1;
            const W b = l2_rhs<W>(at((int64_t)c - 2), at((int64_t)c - 1), at(c), (W)0, (W)0, c, nf);
            prev = fma(-lo_w[m], prev, b) * inv_den[m];
            dl[m * dt] = (T)prev;
        }
        W z = (W)(T)prev;   // d' of the last node
        W r[kLineBack];     // d' of the nodes m0, m0 - 1, ..
#pragma unroll
        for (int u = 0; u < kLineBack; u++) r[u] = (int)nc - 2 - u >= 0 ? (W)dl[(uint64_t)(nc - 2 - u) * dt] : (W)0;
        for (int m0 = (int)nc - 2; m0 >= 0; m0 -= kLineBack) {
            W f[kLineBack], v[kLineBack];
#pragma unroll
            for (int u = 0; u < kLineBack; u++) {
                v[u] = r[u];
                f[u] = cp[max(m0 - u, 0)];
                r[u] = m0 - u >= kLineBack ? (W)dl[(uint64_t)(m0 - u - kLineBack) * dt] : (W)0;
            }
#pragma unroll
            for (int u = 0; u < kLineBack; u++)
                if (m0 - u >= 0) {
                    z = fma(-f[u], z, v[u]);
                    dl[(uint64_t)(m0 - u) * dt] = (T)z;
                }
        }
    }
}

// The dim-2 (contiguous) pass of the L2 projection, one warp per 32 rows of F
// and lane r on row r. The FP64 pipe bounds it (eight operations a node, 431 us
// at 513 x 513 x 257), as long as the loads do not hold its warps up: a ring of
// tiles of 8 coarse nodes (of a row in packed coefficients the even and
// the odd values are two contiguous runs, of a natural row one) is filled by
// cp.async while earlier tiles are swept. A tile's values and Thomas factors
// are read first, then its eight right-hand sides, which do not depend on each
// other, then the chain of the forward step. d' leaves through the tile's slot
// in runs of 8 and comes back the same way, from the end, for the backward
// sweep, or stays in shared memory (KEPT), and the rows leave as one run. More
// warps an SM count for more than a deeper ring (4.4 KB a tile): 513 x 513 x 257
// fp64 585 us with two tiles, 601 with three, 612 with four (955 us with
// 16-column tiles loaded, swept and stored in turn); KEPT 257 x 257 x 129 95 us
// with three, 103 with two, 115 with four.
// PACKED: the rows are read straight from the level's packed coefficients
// (coarse nodes of rows inside the coarse box are zero), so no natural-order
// copy is needed; else from a natural field.
constexpr int kRowsTile = 8, kRowsLd = 2 * kRowsTile + 1;
constexpr int kL2RowsKeep = 200 * 1024;   // shared memory that rows may stay in
constexpr int l2_ring(bool kept) { return kept ? 3 : 2; }   // tiles
template <class T>
inline size_t l2_rows_smem(uint32_t nc, bool kept) {
    return ((size_t)(kept ? 32 * (nc | 1u) : 0) + (size_t)l2_ring(kept) * 32 * kRowsLd) * sizeof(T);
}
template <class T>
__device__ __forceinline__ void cp_async_value(T* dst, const T* src, bool on) {   // zero when off
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = on ? (int)sizeof(T) : 0;
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_close() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_left() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <class T, bool PACKED, bool KEPT>
__global__ void __launch_bounds__(32) k_l2_rows(const T* __restrict__ src, Box F, Box C, T* dst,
                                                const T* __restrict__ cp, const T* __restrict__ lo_w,
                                                const T* __restrict__ inv_den) {
    extern __shared__ __align__(16) unsigned char l2_smem[];
    constexpr int kRowsRing = l2_ring(KEPT);
    const int lane = threadIdx.x, col = lane & 7;
    const uint32_t nf = F.n[2], nc = coarse_len(nf), P = nf - nc;
    const uint32_t ld = nc | 1u;
    T* ring = reinterpret_cast<T*>(l2_smem);     // [kRowsRing][32][kRowsLd]
    T* rows = ring + kRowsRing * 32 * kRowsLd;   // KEPT: [32][ld]
    const uint64_t lines = (uint64_t)F.n[0] * F.n[1], l0 = (uint64_t)blockIdx.x * 32;
    const int nl = (int)min((uint64_t)32, lines - l0);
    T* out = dst + l0 * nc;   // the warp's rows are consecutive in dst
    pdl_wait();
    pdl_release();
    // this lane's row: where its even and odd values start (of a row inside
    // the coarse box only the odd ones are there, the even ones are zero)
    uint64_t ebase = 0, obase = 0;
    bool cc = false;
    if (lane < nl) {
        const uint64_t li = l0 + lane;
        if (PACKED) {
            const uint32_t x0 = (uint32_t)(li / F.n[1]), x1 = (uint32_t)(li - (uint64_t)x0 * F.n[1]);
            const uint32_t r0 = reord(x0, F.n[0], C.n[0]), r1 = reord(x1, F.n[1], C.n[1]);
            cc = r0 < C.n[0] && r1 < C.n[1];
            ebase = level_rank(r0, r1, cc ? C.n[2] : 0u, F, C);
            obase = cc ? ebase : ebase + nc;
        } else {
            ebase = obase = li * nf;
        }
    }
    if (nc == nf) {   // no coarse subset along this dim: the projection is the identity
        if (lane < nl)
            for (uint32_t j = 0; j < nf; j++) out[(uint64_t)lane * nc + j] = cc ? (T)0 : src[ebase + j];
        return;
    }
    // tile t: the even and, behind them, the odd values of the nodes 8 t .. 8 t + 7
    auto fetch = [&](uint32_t t) {
        const uint32_t m = t * kRowsTile + col;
        T* tile = ring + (t % kRowsRing) * 32 * kRowsLd;
        if (t * kRowsTile < nc + 1) {
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += 4) {   // four rows per turn, eight lanes a run
                const int r = r0 + (lane >> 3);
                const uint64_t eb = __shfl_sync(0xffffffffu, ebase, r), ob = __shfl_sync(0xffffffffu, obase, r);
                const bool zero = __shfl_sync(0xffffffffu, (int)cc, r), on = r < nl;
                const bool e = on && m < nc && !zero, o = on && m < P;
                const uint64_t ei = eb + (PACKED ? m : min(2 * m, nf - 1)), oi = ob + (PACKED ? m : 2 * m + 1);
                cp_async_value(tile + r * kRowsLd + col, e ? src + ei : src, e);
                cp_async_value(tile + r * kRowsLd + kRowsTile + col, o ? src + oi : src, o);
            }
        }
        cp_async_close();
    };
#pragma unroll
    for (int t = 0; t < kRowsRing - 1; t++) fetch(t);
    T* own = rows + lane * ld;
    // Node m needs the even value of node m + 1, which may lie in the next
    // tile, so tile t brings the nodes 8 t - 1 .. 8 t + 6. Carried over: the
    // last two even values and the last three odd ones.
    T em1 = 0, e0 = 0, om2 = 0, om1 = 0, o0 = 0, prev = 0;
    for (uint32_t t = 0; t * kRowsTile < nc + 1; t++) {
        fetch(t + kRowsRing - 1);
        cp_async_left<kRowsRing - 1>();
        __syncwarp();
        T* tile = ring + (t % kRowsRing) * 32 * kRowsLd + lane * kRowsLd;
        T ev[kRowsTile + 2] = {em1, e0}, od[kRowsTile + 3] = {om2, om1, o0}, dp[kRowsTile];
#pragma unroll
        for (int u = 0; u < kRowsTile; u++) {
            ev[2 + u] = tile[u];
            od[3 + u] = tile[kRowsTile + u];
        }
        const int j0 = (int)(t * kRowsTile) - 1;
        if (t && 2 * (uint32_t)(j0 + kRowsTile - 1) + 3 <= nf) {
            T lo[kRowsTile], inv[kRowsTile];
#pragma unroll
            for (int u = 0; u < kRowsTile; u++) {
                lo[u] = lo_w[j0 + u];
                inv[u] = inv_den[j0 + u];
                dp[u] = l2_rhs<T, true>(ev[u], od[1 + u], ev[1 + u], od[2 + u], ev[2 + u], 2 * (j0 + u), nf);
            }
#pragma unroll
            for (int u = 0; u < kRowsTile; u++) dp[u] = prev = fma(-lo[u], prev, dp[u]) * inv[u];
        } else {
#pragma unroll
            for (int u = 0; u < kRowsTile; u++) {
                const int j = j0 + u;
                if (j >= 0 && j < (int)nc) {
                    const bool lastone = j == (int)nc - 1;
                    T sm2 = ev[u], sm1 = od[1 + u], s1 = od[2 + u], s2 = ev[2 + u];
                    if (lastone) s1 = s2 = 0;
                    if (!(nf & 1u)) {   // the last two nodes sit side by side
                        if (lastone) { sm2 = od[u]; sm1 = ev[u]; }
                        else if (j == (int)nc - 2) { s1 = ev[2 + u]; s2 = 0; }
                    }
                    const T b = l2_rhs<T>(sm2, sm1, ev[1 + u], s1, s2, lastone ? nf - 1 : 2 * j, nf);
                    prev = j == 0 ? b * inv_den[0] : fma(-lo_w[j], prev, b) * inv_den[j];
                }
                dp[u] = prev;
            }
        }
#pragma unroll
        for (int u = 0; u < kRowsTile; u++) {
            if constexpr (KEPT) {
                if (j0 + u >= 0 && j0 + u < (int)nc) own[j0 + u] = dp[u];
            } else {
                tile[u] = dp[u];   // (its own row, read above)
            }
        }
        __syncwarp();
        if constexpr (!KEPT) {
            const int j = j0 + col;
            const T* all = ring + (t % kRowsRing) * 32 * kRowsLd;
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += 4) {
                const int r = r0 + (lane >> 3);
                if (r < nl && j >= 0 && j < (int)nc) out[(uint64_t)r * nc + j] = all[r * kRowsLd + col];
            }
            __syncwarp();   // the slot is free for the fetch after next
        }
        em1 = ev[kRowsTile];
        e0 = ev[kRowsTile + 1];
        om2 = od[kRowsTile];
        om1 = od[kRowsTile + 1];
        o0 = od[kRowsTile + 2];
    }
    // backward substitution, eight nodes at a time from the end
    T z = prev;
    auto back = [&](T* v, int m0) {   // the nodes m0 .. m0 + 7 in v[0 .. 7]
        T x[kRowsTile], f[kRowsTile];
#pragma unroll
        for (int u = 0; u < kRowsTile; u++) {
            x[u] = m0 + u < (int)nc ? v[u] : (T)0;
            f[u] = cp[min(m0 + u, (int)nc - 1)];
        }
#pragma unroll
        for (int u = kRowsTile - 1; u >= 0; u--)
            if (m0 + u < (int)nc - 1) v[u] = z = fma(-f[u], z, x[u]);
    };
    const int top = ((int)nc - 1) & ~(kRowsTile - 1);
    if constexpr (KEPT) {
        for (int m0 = top; m0 >= 0; m0 -= kRowsTile) back(own + m0, m0);
        __syncwarp();
        for (uint32_t j = lane; j < nc; j += 32)
#pragma unroll 8
            for (int r = 0; r < nl; r++) out[(uint64_t)r * nc + j] = rows[r * ld + j];
    } else {
        auto fetch_back = [&](int i) {   // the i-th tile from the end
            const int m = top - i * kRowsTile + col;
            T* tile = ring + (i % kRowsRing) * 32 * kRowsLd;
            if (top - i * kRowsTile >= 0) {
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 4) {
                    const int r = r0 + (lane >> 3);
                    const bool on = r < nl && m < (int)nc;
                    cp_async_value(tile + r * kRowsLd + col, on ? out + (uint64_t)r * nc + m : out, on);
                }
            }
            cp_async_close();
        };
#pragma unroll
        for (int i = 0; i < kRowsRing - 1; i++) fetch_back(i);
        for (int i = 0; i * kRowsTile <= top; i++) {
            fetch_back(i + kRowsRing - 1);
            cp_async_left<kRowsRing - 1>();
            __syncwarp();
            T* all = ring + (i % kRowsRing) * 32 * kRowsLd;
            const int m0 = top - i * kRowsTile;
            back(all + lane * kRowsLd, m0);
            __syncwarp();
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += 4) {
                const int r = r0 + (lane >> 3);
                if (r < nl && m0 + col < (int)nc) out[(uint64_t)r * nc + m0 + col] = all[r * kRowsLd + col];
            }
            __syncwarp();
        }
    }
}

// dst[i] += sign * z[i] over a compact box written into a strided box
template <class T>
__global__ void k_add_box(T* __restrict__ dst, uint64_t b0, uint64_t b1, const T* __restrict__ z, Box B, T sign) {
    pdl_wait();
    pdl_release();
    const uint64_t total = B.size();
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, B, x0, x1, x2);
        dst[x0 * b0 + x1 * b1 + x2] += sign * z[idx];
    }
}

// DirectInterleaver gather/scatter over box(fine) \ box(coarse).
template <class T, bool GATHER>
__global__ void k_interleave(T* __restrict__ data, uint64_t s0, uint64_t s1, Box F, Box C, T* __restrict__ buf) {
    const uint64_t total = F.size();
    for (uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x0, x1, x2;
        split3(idx, F, x0, x1, x2);
        if (x0 < C.n[0] && x1 < C.n[1] && x2 < C.n[2]) continue;
        uint64_t r = level_rank(x0, x1, x2, F, C);
        if (GATHER) buf[r] = data[x0 * s0 + x1 * s1 + x2];
        else data[x0 * s0 + x1 * s1 + x2] = buf[r];
    }
}

// the same with a warp per row, whose values outside the coarse box are one run of ranks
template <class T, bool GATHER>
__global__ void __launch_bounds__(256) k_interleave_rows(T* __restrict__ data, uint64_t s0, uint64_t s1, Box F, Box C,
                                                         T* __restrict__ buf) {
    const uint64_t rows = (uint64_t)F.n[0] * F.n[1], wpb = blockDim.x >> 5;
    for (uint64_t r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
        const uint32_t x0 = (uint32_t)(r / F.n[1]), x1 = (uint32_t)(r - (uint64_t)x0 * F.n[1]);
        bool cc;
        T* run = buf + row_rank_base(x0, x1, F, C, cc);
        const uint32_t from = cc ? C.n[2] : 0u;
        T* row = data + x0 * s0 + x1 * s1 + from;
        warp_copy<T>(GATHER ? row : run, GATHER ? run : row, F.n[2] - from, threadIdx.x & 31);
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// one warp per row, four warps per CTA (f64 recompositions of 513 x 257 x 257's
// small levels 86 us, with eight 90 and with one 92; fp32 1 % from eight, with
// two 10 % slower); enough CTAs for full occupancy
constexpr unsigned kRowThreads = 128;
// PRODM_DECOMPOSE_PATCH=0 keeps every level on the row kernels (decomposition and
// recomposition; read per launch)
bool decompose_patch_enabled() {
    const char* v = getenv("PRODM_DECOMPOSE_PATCH");
    return !(v && v[0] == '0');
}
// Copies and interleaving go by rows, a warp each, where a row has at least a
// warp's width of values and there are rows for every SM (else by elements).
// 150 x 257 x 301 fp32: copy 16 us by rows, 39 by elements; interleaving 13 and
// 48 us (DRAM floor 14).
inline bool walk_rows(const Box& B) { return B.n[2] >= 32 && (uint64_t)B.n[0] * B.n[1] >= 8ull * kSMs; }
unsigned row_grid(uint64_t rows, unsigned th) {
    const uint64_t wpb = th / 32;
    uint64_t need = (rows + wpb - 1) / wpb;
    uint64_t cap = (uint64_t)device_sms() * 8 * 4 * (256 / th);
    uint64_t g = need < cap ? need : cap;
    return (unsigned)(g ? g : 1);
}

template <class T>
int launch_decompose_level_packed(const T* in, uint64_t s0, uint64_t s1, const Box& F, const Box& C, T* coef, T* coarse,
                                  T* fnat, void* maxkey_level, void* maxkey_coarse, cudaStream_t st) {
    using K = typename KeyOf<T>::type;
    const unsigned th = kRowThreads;
    count_launch();
    if (!fnat && patch_level(F, C) && decompose_patch_enabled()) {
        const auto kernel = F.n[0] == 1 ? k_decompose_patch<T, kPlaneAhead> : k_decompose_patch<T, 0>;
        const cudaError_t e = launch_chain(true, kernel, dim3(row_grid(patch_items(F, C), kPatchThreads)), dim3(kPatchThreads), 0,
                                           st, in, s0, s1, F, C, coef, coarse, (K*)maxkey_level, (K*)maxkey_coarse);
        if (e != cudaSuccess) return cuda_status(e, "k_decompose_patch");
        return PRODM_OK;
    }
    const cudaError_t e = launch_chain(true, k_decompose_rows<T>, dim3(row_grid((uint64_t)F.n[0] * F.n[1], th)), dim3(th),
                                       0, st, in, s0, s1, F, C, coef, coarse, fnat, (K*)maxkey_level, (K*)maxkey_coarse);
    if (e != cudaSuccess) return cuda_status(e, "k_decompose_rows");
    return PRODM_OK;
}

template <class T>
int launch_decompose_level_inplace(const T* in, const Box& F, const Box& C, T* out, uint64_t o0, uint64_t o1, T* fnat,
                                   cudaStream_t st) {
    const int th = 256;
    if (!fnat && patch_level(F, C) && decompose_patch_enabled()) {   // 150 x 257 x 301 fp32: 18.7 us, by elements 81
        k_decompose_patch_inplace<T><<<row_grid(patch_items(F, C), kPatchThreads), kPatchThreads, 0, st>>>(in, F, C, out, o0, o1);
        PRODM_CHECK_LAUNCH("k_decompose_patch_inplace");
        return PRODM_OK;
    }
    k_decompose_level<T><<<grid_for(F.size(), th), th, 0, st>>>(in, F, C, out, o0, o1, fnat);
    PRODM_CHECK_LAUNCH("k_decompose_level");
    return PRODM_OK;
}

template <class T>
int launch_recompose_level_packed(const T* coarse, const T* coef, const Box& F, const Box& C, T* out, uint64_t s0,
                                  uint64_t s1, cudaStream_t st, bool pdl) {
    const unsigned th = kRowThreads;
    count_launch();
    if (patch_level(F, C) && decompose_patch_enabled()) {
        const auto kernel = F.n[0] == 1 ? k_recompose_patch<T, kPlaneAhead> : k_recompose_patch<T, 0>;
        const cudaError_t e = launch_chain(pdl, kernel, dim3(row_grid(patch_items(F, C), kPatchThreads)), dim3(kPatchThreads), 0,
                                           st, coarse, coef, F, C, out, s0, s1);
        if (e != cudaSuccess) return cuda_status(e, "k_recompose_patch");
        return PRODM_OK;
    }
    const cudaError_t e = launch_chain(pdl, k_recompose_rows<T>, dim3(row_grid((uint64_t)F.n[0] * F.n[1], th)), dim3(th),
                                       0, st, coarse, coef, F, C, out, s0, s1);
    if (e != cudaSuccess) return cuda_status(e, "k_recompose_rows");
    return PRODM_OK;
}

template <class T>
int launch_recompose_level_inplace(const T* rin, const Box& F, const Box& C, T* out, uint64_t s0, uint64_t s1,
                                   cudaStream_t st) {
    const int th = 256;
    if (patch_level(F, C) && decompose_patch_enabled()) {   // 150 x 257 x 301 fp32: 18.3 us, by elements 76
        k_recompose_patch_inplace<T><<<row_grid(patch_items(F, C), kPatchThreads), kPatchThreads, 0, st>>>(rin, F, C, out, s0, s1);
        PRODM_CHECK_LAUNCH("k_recompose_patch_inplace");
        return PRODM_OK;
    }
    k_recompose_level<T><<<grid_for(F.size(), th), th, 0, st>>>(rin, F, C, out, s0, s1);
    PRODM_CHECK_LAUNCH("k_recompose_level");
    return PRODM_OK;
}

template <class T>
int launch_copy_box(const T* src, uint64_t a0, uint64_t a1, const Box& B, T* dst, uint64_t b0, uint64_t b1,
                    cudaStream_t st) {
    const int th = 256;
    if (walk_rows(B)) {
        k_copy_rows<T><<<row_grid((uint64_t)B.n[0] * B.n[1], th), th, 0, st>>>(src, a0, a1, B, dst, b0, b1);
        PRODM_CHECK_LAUNCH("k_copy_rows");
        return PRODM_OK;
    }
    k_copy_box<T><<<grid_for(B.size(), th), th, 0, st>>>(src, a0, a1, B, dst, b0, b1);
    PRODM_CHECK_LAUNCH("k_copy_box");
    return PRODM_OK;
}

template <class T>
int launch_coef_to_natural(const T* coef, const Box& F, const Box& C, T* fnat, cudaStream_t st) {
    const int th = 256;
    k_coef_to_natural<T><<<grid_for(F.size(), th), th, 0, st>>>(coef, F, C, fnat);
    PRODM_CHECK_LAUNCH("k_coef_to_natural");
    return PRODM_OK;
}

template <class T>
int launch_reordered_to_natural(const T* rin, const Box& F, const Box& C, T* fnat, cudaStream_t st) {
    const int th = 256;
    k_reordered_to_natural<T><<<grid_for(F.size(), th), th, 0, st>>>(rin, F, C, fnat);
    PRODM_CHECK_LAUNCH("k_reordered_to_natural");
    return PRODM_OK;
}

// Thomas factors of the coarse mass matrix of a dim with n fine nodes.
// layout in tab: [cp(nc) | lo(nc) | inv_den(nc)]
template <class W>
void mass_factors(uint32_t n, W* tab) {
    uint32_t nc = coarse_len(n);
    W* cp = tab;
    W* lo = tab + nc;
    W* inv = tab + 2 * nc;
    double prev_cp = 0;
    for (uint32_t m = 0; m < nc; m++) {
        double hl = m > 0 ? (double)(fine_of_coarse(m, n, nc) - fine_of_coarse(m - 1, n, nc)) : 0.0;
        double hr = m + 1 < nc ? (double)(fine_of_coarse(m + 1, n, nc) - fine_of_coarse(m, n, nc)) : 0.0;
        double dg = (hl + hr) / 3, up = hr / 6, low = hl / 6;
        double den = m == 0 ? dg : dg - low * prev_cp;
        double c = up / den;
        cp[m] = (W)c;
        lo[m] = (W)low;
        inv[m] = (W)(1.0 / den);
        prev_cp = c;
    }
}
template void mass_factors<float>(uint32_t, float*);
template void mass_factors<double>(uint32_t, double*);

// z (compact C box) = L2 projection of the natural coefficient field (F box):
// from fnat, or (coef != nullptr) straight from the level's packed
// coefficients (coarse box C). tabs[d] = device Thomas factors for dim d;
// t1/t2 scratch boxes. The contiguous dim goes first through the staged row
// kernel, the two strided dims through the line kernel (coalesced there).
template <class T>
int launch_l2_correction(const T* fnat, const Box& F, T* t1, T* t2, T* z, const T* const tabs[3], cudaStream_t st,
                         const T* coef, const Box* C) {
    const int th = 32;
    Box a = F;
    T* bufs[3] = {t1, t2, z};
    {
        const uint32_t nc = coarse_len(F.n[2]);
        const T* tab = tabs[2];
        const uint64_t lines = (uint64_t)F.n[0] * F.n[1];
        const dim3 grid((unsigned)((lines + 31) / 32));
        // Keep d' on chip while that leaves six warps an SM (36 KB; 257 x 257 x 129
        // fp64 at 34 KB: level 332 us against 360), or where all warps are
        // resident at once anyway (129 x 129 x 257: 179 against 271); at 50 KB and
        // 54 warps an SM (513 x 513 x 257) it is 2030 against 1797.
        const size_t keep = l2_rows_smem<T>(nc, true);
        const bool kept = keep <= 36 * 1024 ||
                          (keep <= (size_t)kL2RowsKeep && (uint64_t)(227 * 1024 / (keep + 1024)) * kSMs >= grid.x);
        const size_t smem = l2_rows_smem<T>(nc, kept);
        const auto kernel = coef ? (kept ? k_l2_rows<T, true, true> : k_l2_rows<T, true, false>)
                                 : (kept ? k_l2_rows<T, false, true> : k_l2_rows<T, false, false>);
        cudaError_t e;
        // (the most any call needs, not this call's: another thread may launch the kernel in between)
        if (smem > 48 * 1024 && (e = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          kL2RowsKeep)) != cudaSuccess)
            return cuda_status(e, "cudaFuncSetAttribute");
        count_launch();
        // not launched ahead: its one-warp blocks would gather on the SMs that
        // the kernel before leaves room on (65 x 65 x 2049: level 1178 us, 587 so)
        e = launch_chain(false, kernel, grid, dim3(32), smem, st, coef ? coef : fnat, F, coef ? *C : F, t1, tab, tab + nc,
                         tab + 2 * nc);
        if (e != cudaSuccess) return cuda_status(e, "k_l2_rows");
        a.n[2] = nc;
    }
    const T* src = t1;
    for (int k = 1, d = 1; d >= 0; d--, k++) {
        Box b = a;
        b.n[d] = coarse_len(a.n[d]);
        uint64_t lines = a.size() / a.n[d];
        uint32_t nc = b.n[d];
        const T* tab = tabs[d];
        count_launch();
        const cudaError_t e = launch_chain(true, k_l2_line<T, T>, dim3(grid_for(lines, th, 16)), dim3(th), 0, st, src, a, d,
                                           bufs[k], b, tab, tab + nc, tab + 2 * nc);
        if (e != cudaSuccess) return cuda_status(e, "k_l2_line");
        src = bufs[k];
        a = b;
    }
    return PRODM_OK;
}

template <class T>
int launch_add_box(T* dst, uint64_t b0, uint64_t b1, const T* z, const Box& B, T sign, cudaStream_t st) {
    const int th = 256;
    count_launch();
    const cudaError_t e = launch_chain(true, k_add_box<T>, dim3(grid_for(B.size(), th)), dim3(th), 0, st, dst, b0, b1, z, B,
                                       sign);
    if (e != cudaSuccess) return cuda_status(e, "k_add_box");
    return PRODM_OK;
}

template <class T>
int launch_interleave(T* data, uint64_t s0, uint64_t s1, const Box& F, const Box& C, T* buf, bool gather,
                      cudaStream_t st) {
    const int th = 256;
    if (walk_rows(F)) {
        const unsigned grid = row_grid((uint64_t)F.n[0] * F.n[1], th);
        if (gather) k_interleave_rows<T, true><<<grid, th, 0, st>>>(data, s0, s1, F, C, buf);
        else k_interleave_rows<T, false><<<grid, th, 0, st>>>(data, s0, s1, F, C, buf);
        PRODM_CHECK_LAUNCH("k_interleave_rows");
        return PRODM_OK;
    }
    if (gather) k_interleave<T, true><<<grid_for(F.size(), th), th, 0, st>>>(data, s0, s1, F, C, buf);
    else k_interleave<T, false><<<grid_for(F.size(), th), th, 0, st>>>(data, s0, s1, F, C, buf);
    PRODM_CHECK_LAUNCH("k_interleave");
    return PRODM_OK;
}

#define INST(T)                                                                                                     \
    template int launch_decompose_level_packed<T>(const T*, uint64_t, uint64_t, const Box&, const Box&, T*, T*, T*, \
                                                  void*, void*, cudaStream_t);                                      \
    template int launch_decompose_level_inplace<T>(const T*, const Box&, const Box&, T*, uint64_t, uint64_t, T*,    \
                                                   cudaStream_t);                                                   \
    template int launch_recompose_level_packed<T>(const T*, const T*, const Box&, const Box&, T*, uint64_t,         \
                                                  uint64_t, cudaStream_t, bool);                                    \
    template int launch_recompose_level_inplace<T>(const T*, const Box&, const Box&, T*, uint64_t, uint64_t,        \
                                                   cudaStream_t);                                                   \
    template int launch_copy_box<T>(const T*, uint64_t, uint64_t, const Box&, T*, uint64_t, uint64_t, cudaStream_t); \
    template int launch_coef_to_natural<T>(const T*, const Box&, const Box&, T*, cudaStream_t);                     \
    template int launch_reordered_to_natural<T>(const T*, const Box&, const Box&, T*, cudaStream_t);                \
    template int launch_l2_correction<T>(const T*, const Box&, T*, T*, T*, const T* const[3], cudaStream_t,      \
                                         const T*, const Box*);                                                     \
    template int launch_add_box<T>(T*, uint64_t, uint64_t, const T*, const Box&, T, cudaStream_t);                  \
    template int launch_interleave<T>(T*, uint64_t, uint64_t, const Box&, const Box&, T*, bool, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace prodm
