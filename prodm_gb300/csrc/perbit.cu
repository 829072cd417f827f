// Per-bit bitplane format on the device (sm_103a): PerBitBPEncoder
// (PerBitBPEncoder.hpp:7-146 encode, :290-383 progressive_decode).
//
// Reference stream format: one bit stream per plane, bits packed from the
// least significant end of 64-bit words. Element i writes, in plane p, bit
// (B-1-p) of its fixed-point magnitude and, right after its first 1 bit, its
// sign. Where a bit of plane p sits therefore depends on how many earlier
// elements had their first 1 bit in plane p: a stream can only be parsed with
// the planes before it.
//
// Device layout ("rows"): the level's elements in groups of 32; row p (p < B)
// holds one 32-bit word per group whose bit j is bit (B-1-p) of element
// 32g+j's magnitude; row B holds the sign words (bit j set: element negative
// and nonzero); row B+1 (parsed streams only) the elements that have no 1 bit
// in the planes parsed so far. Every row starts on a 16-byte boundary. In this
// layout decoding is a transpose per group and needs no parse; the reference
// stream sizes (ceil((n + first-ones in p) / 64) * 8 bytes) are computed at
// encode time, and pb_pack writes the reference streams on export.
#include "common.cuh"
#include "kernels.cuh"
#include "nbcodec.cuh"

namespace prodm {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int PB_WARPS = 8;
constexpr int PB_GPW = 16;                        // groups per warp per chunk
constexpr int PB_CHUNK = PB_WARPS * PB_GPW;       // groups per CTA chunk
constexpr int PB_LD = PB_CHUNK + 1;               // padded tile row

template <class T>
__device__ __forceinline__ int pb_exp(const typename KeyOf<T>::type* maxkey, int exp_arg) {
    return maxkey ? frexp_exp(key_to_val(*maxkey, T())) : exp_arg;
}

// Fixed-point magnitude of one value, |trunc(ldexp(v, k))| with k = B - exp
// (PerBitBPEncoder.hpp:100-104). The scaling is exact (the result stays
// below 2^B), so the truncated magnitude is floor(|v| * 2^k): for doubles it
// is taken from the exponent and mantissa bits with integer operations
// (GB300's FP64 pipe is slow); for floats by one multiplication with an exact
// power of two where that is a normal float, else ldexpf.
__device__ __forceinline__ uint64_t pb_mag(double v, int k, bool, float) { return fixed_mag(v, k); }
__device__ __forceinline__ uint32_t pb_mag(float v, int k, bool fast, float sc) {
    return (uint32_t)fabsf(fast ? v * sc : ldexpf(v, k));
}
__device__ __forceinline__ bool pb_neg(double v) { return __double_as_longlong(v) < 0; }
__device__ __forceinline__ bool pb_neg(float v) { return v < 0.f; }

// ldexp((T)acc, s) (PerBitBPEncoder.hpp:343). For doubles with every result
// normal (fast: -1022 <= s <= 960), acc is rounded once to 53 bits (nearest,
// ties to even, as the conversion does) and the exponent field written
// directly; otherwise, and for floats, the conversion and an exact scaling.
__device__ __forceinline__ double pb_value(uint64_t acc, int s, bool fast, float) {
    return fast ? fixed_value(acc, s) : ldexp((double)acc, s);
}
__device__ __forceinline__ float pb_value(uint32_t acc, int s, bool fast, float sc) {
    return fast ? (float)acc * sc : ldexpf((float)acc, s);
}
__device__ __forceinline__ double pb_negate(double v) {
    return __longlong_as_double(__double_as_longlong(v) ^ (long long)0x8000000000000000ull);
}
__device__ __forceinline__ float pb_negate(float v) { return -v; }
__device__ __forceinline__ bool pb_value_fast(double*, int s) { return fixed_value_normal(s); }
__device__ __forceinline__ bool pb_value_fast(float*, int s) { return pow2_normal(s); }

__device__ __forceinline__ uint32_t valid_mask(int nvalid) { return nvalid >= 32 ? FULL : ((1u << nvalid) - 1u); }

// The encoder and the decoder take the chunks of all levels of a field in one
// launch (PbSet, one segment per level), so that the small levels' few chunks
// run beside the large one's instead of one launch after the other
// (513 x 257 x 257 fp64, 60 planes: encode 331 us in 14 launches, 203 us in 2;
// decode 184 us per retrieval in 7, 125 us in one).
template <class T>
__device__ __forceinline__ int pb_seg(const PbSet<T>& set, uint32_t c) {
    int l = 0;
    while (l + 1 < set.n && c >= set.seg[l + 1].chunk0) l++;
    return l;
}

// ---------------------------------------------------------------------------
// encode: values -> rows 0..B (magnitude planes + signs) and, per plane, the
// number of elements whose first 1 bit is in that plane
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) k_pb_encode(const __grid_constant__ PbSet<T> set, uint32_t total, int B) {
    using FP = typename Traits<T>::FP;
    extern __shared__ uint32_t tile[];   // (B + 1) rows x PB_LD
    __shared__ uint32_t cnt[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    pdl_release();
    for (int k = threadIdx.x; k < 64; k += blockDim.x) cnt[k] = 0;
    int cur = -1;
    auto flush = [&]() {   // the level's counts; every thread calls it
        __syncthreads();
        if (cur >= 0)
            for (int p = threadIdx.x; p < B; p += blockDim.x)
                if (cnt[p]) {
                    atomicAdd(&set.seg[cur].counts[p], cnt[p]);
                    cnt[p] = 0;
                }
        __syncthreads();
    };
    for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
        const int l = pb_seg(set, c);
        if (l != cur) {
            flush();
            cur = l;
        }
        const PbSeg<T>& q = set.seg[l];
        const T* __restrict__ x = q.x;
        const uint64_t n = q.n, ng = (n + 31) / 32, g0 = (uint64_t)(c - q.chunk0) * PB_CHUNK;
        const int exp = pb_exp<T>(q.key, q.exp);
        const int ks = B - exp;
        const bool fast = pow2_normal(ks);
        const float sc = fast ? pow2f(ks) : 1.f;
#pragma unroll 2
        for (int j = 0; j < PB_GPW; j++) {
            const int gl = warp * PB_GPW + j;
            const uint64_t i = (g0 + gl) * 32 + lane;
            const T v = i < n ? __ldcs(x + i) : (T)0;
            const FP m = pb_mag(v, ks, fast, sc);
            const uint32_t sgn = __ballot_sync(FULL, pb_neg(v) && m != 0);
            // a value's first 1 bit is its most significant one: count the
            // group's values per msb (one shared atomic per distinct msb)
            const int msb = m ? (int)(8 * sizeof(FP)) - 1 - (sizeof(T) == 8 ? __clzll((long long)m) : __clz((int)m))
                              : -1;
            const unsigned same = __match_any_sync(FULL, msb);
            if (msb >= 0 && lane == __ffs(same) - 1) atomicAdd(&cnt[B - 1 - msb], (uint32_t)__popc(same));
            const uint32_t lo = transpose32((uint32_t)m, lane);          // lane k: bit k of the 32 magnitudes
            const uint32_t hi = sizeof(T) == 8 ? transpose32((uint32_t)((uint64_t)m >> 32), lane) : 0u;
            if (lane < B) tile[(B - 1 - lane) * PB_LD + gl] = lo;
            if (sizeof(T) == 8 && lane + 32 < B) tile[(B - 33 - lane) * PB_LD + gl] = hi;
            if (lane == 0) tile[B * PB_LD + gl] = sgn;
        }
        __syncthreads();
        const int nvalid = (int)((ng - g0) < (uint64_t)PB_CHUNK ? (ng - g0) : PB_CHUNK);
        for (int p = warp; p <= B; p += PB_WARPS) {
            uint32_t* dst = q.rows + (uint64_t)p * q.stride + g0;
            const uint32_t* src = tile + p * PB_LD;
            for (int j = lane; j < nvalid; j += 32) dst[j] = src[j];
        }
        __syncthreads();
    }
    flush();
}

// reference stream sizes: BitEncoder words (n + first-one count bits) * 8, one CTA per level
template <class T>
__global__ void k_pb_sizes(const __grid_constant__ PbSet<T> set, int B) {
    pdl_wait();
    pdl_release();
    const PbSeg<T>& q = set.seg[blockIdx.x];
    const int p = threadIdx.x;
    if (p < B) q.sizes[p] = (uint32_t)((q.n + q.counts[p] + 63) / 64 * 8);
}

// ---------------------------------------------------------------------------
// decode planes [s, e): value = 2^(exp-e) * (magnitude bits of planes s..e-1),
// negative where the element's sign is known by plane e (progressive_decode
// :315-344: a sign is read with the first 1 bit) and its sign bit is set.
// `unseen` (row of elements without a 1 bit in planes < e) may be NULL when
// s == 0: then "known" is "nonzero". dnum (device plane count) overrides e.
// ---------------------------------------------------------------------------
// the groups of one staged chunk; FAST: every value is normal (no FP64 path
// in the loop)
template <class T, bool FAST>
__device__ __forceinline__ void pb_decode_groups(const uint32_t* tile, int num, int nvalid, uint64_t g0, uint64_t n,
                                                 int vs, float sc, bool with_unseen, T* __restrict__ out) {
    using FP = typename Traits<T>::FP;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 2
    for (int j = 0; j < PB_GPW; j++) {
        const int gl = warp * PB_GPW + j;
        if (gl >= nvalid) break;
        const uint32_t wl = lane < num ? tile[(num - 1 - lane) * PB_LD + gl] : 0u;
        FP acc = transpose32(wl, lane);
        if (sizeof(T) == 8 && num > 32) {
            const uint32_t wh = lane + 32 < num ? tile[(num - 33 - lane) * PB_LD + gl] : 0u;
            acc |= (FP)((uint64_t)transpose32(wh, lane) << 32);
        }
        const uint32_t sg = tile[num * PB_LD + gl];
        const bool known = with_unseen ? !((tile[(num + 1) * PB_LD + gl] >> lane) & 1u) : acc != 0;
        const T v = pb_value(acc, vs, FAST, sc);
        const uint64_t i = (g0 + gl) * 32 + lane;
        if (i < n) out[i] = (known && ((sg >> lane) & 1u)) ? pb_negate(v) : v;
    }
}

template <class T>
__global__ void __launch_bounds__(256) k_pb_decode(const __grid_constant__ PbSet<T> set, uint32_t total, int s, int e_arg) {
    extern __shared__ uint32_t tile[];   // num + 2 rows x PB_LD
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    pdl_release();
    for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
        const PbSeg<T>& q = set.seg[pb_seg(set, c)];
        const int e = q.dnum ? q.dnum[0] : e_arg, num = e - s;
        const int vs = pb_exp<T>(q.key, q.exp) - e;
        const bool fast = pb_value_fast((T*)nullptr, vs);
        const float sc = (sizeof(T) == 4 && fast) ? pow2f(vs) : 1.f;
        const uint64_t n = q.n, ng = (n + 31) / 32, g0 = (uint64_t)(c - q.chunk0) * PB_CHUNK;
        const int nvalid = (int)((ng - g0) < (uint64_t)PB_CHUNK ? (ng - g0) : PB_CHUNK);
        const int nr = num + (q.unseen ? 2 : 1);
        // a row's 128 words are one 16-byte load per lane (rows are padded to 16 bytes)
        constexpr int U = 4;
        for (int r0 = warp; r0 < nr; r0 += U * PB_WARPS) {
            uint4 w[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int r = r0 + u * PB_WARPS;
                const uint32_t* src = (r < num ? q.rows + (uint64_t)(s + r) * q.stride : (r == num ? q.srow : q.unseen)) + g0;
                w[u] = r < nr && 4 * lane < nvalid ? __ldcs(reinterpret_cast<const uint4*>(src) + lane) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int r = r0 + u * PB_WARPS;
                if (r >= nr) break;
                uint32_t* dst = tile + r * PB_LD + 4 * lane;
                dst[0] = w[u].x;
                dst[1] = w[u].y;
                dst[2] = w[u].z;
                dst[3] = w[u].w;
            }
        }
        __syncthreads();
        if (fast) pb_decode_groups<T, true>(tile, num, nvalid, g0, n, vs, sc, q.unseen != nullptr, q.y);
        else pb_decode_groups<T, false>(tile, num, nvalid, g0, n, vs, sc, q.unseen != nullptr, q.y);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// export: rows -> reference streams (BitEncoder layout), three passes
//   count: bits of every (plane, 256-group chunk), and before each of its warps
//   scan:  chunk bit offsets within each plane
//   write: each group's segment of each plane (<= 64 bits) OR-ed into the
//          zeroed destination
// A thread walks the planes of its group (an element's sign follows its first 1
// bit). The planes' words do not depend on each other, so PK_U are loaded at a
// time and the next ones while these are worked on, and a warp knows its place
// in every plane beforehand, so the warps of a chunk do not wait for one
// another. 2^20 values, 60 planes: count 40 us and write 90 us with a load and
// two barriers a plane, 13 and 40 us so.
// ---------------------------------------------------------------------------
constexpr int PK_T = 256;   // groups (threads) per chunk
constexpr int PK_W = PK_T / 32;
constexpr int PK_U = 10;    // planes loaded ahead

__device__ __forceinline__ int pk_nvalid(uint64_t g, uint64_t ng, uint64_t n) {
    if (g >= ng) return 0;
    const uint64_t r = n - g * 32;
    return r < 32 ? (int)r : 32;
}

// body(p, M) for the planes p in order, M the valid elements' bits
template <class Body>
__device__ __forceinline__ void pk_planes(const uint32_t* __restrict__ rows, uint64_t stride, uint64_t g, uint32_t vm, int B,
                                          Body body) {
    uint32_t nx[PK_U];
    auto load = [&](int p0) {
#pragma unroll
        for (int u = 0; u < PK_U; u++) nx[u] = vm && p0 + u < B ? __ldg(rows + (uint64_t)(p0 + u) * stride + g) & vm : 0u;
    };
    load(0);
    for (int p0 = 0; p0 < B; p0 += PK_U) {
        uint32_t m[PK_U];
#pragma unroll
        for (int u = 0; u < PK_U; u++) m[u] = nx[u];
        load(p0 + PK_U);
#pragma unroll
        for (int u = 0; u < PK_U; u++)
            if (p0 + u < B) body(p0 + u, m[u]);
    }
}

// warp_bits: the bits of a chunk's warps before each of them, [plane][chunk][PK_W]
__global__ void __launch_bounds__(PK_T) k_pb_pack_count(const uint32_t* __restrict__ rows, uint64_t stride, uint64_t n,
                                                        int B, uint32_t* __restrict__ chunk_bits, uint64_t nch,
                                                        uint16_t* __restrict__ warp_bits) {
    __shared__ uint32_t cnt[PK_W][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t ng = (n + 31) / 32;
    const uint64_t g = (uint64_t)blockIdx.x * PK_T + threadIdx.x;
    const int nvalid = pk_nvalid(g, ng, n);
    uint32_t seen = 0;
    pk_planes(rows, stride, g, valid_mask(nvalid), B, [&](int p, uint32_t M) {
        const uint32_t bits = __reduce_add_sync(FULL, (uint32_t)(nvalid + __popc(M & ~seen)));
        seen |= M;
        if (lane == 0) cnt[warp][p] = bits;
    });
    __syncthreads();
    for (int p = threadIdx.x; p < B; p += blockDim.x) {
        const uint64_t at = (uint64_t)p * nch + blockIdx.x;
        uint32_t run = 0;
        for (int w = 0; w < PK_W; w++) {
            warp_bits[at * PK_W + w] = (uint16_t)run;   // at most 7 x 32 x 64
            run += cnt[w][p];
        }
        chunk_bits[at] = run;
    }
}

// exclusive scan of one plane's (blockIdx.x) chunk bits
__global__ void __launch_bounds__(256) k_pb_pack_scan(const uint32_t* __restrict__ chunk_bits, uint64_t nch,
                                                      uint64_t* __restrict__ chunk_off) {
    __shared__ uint64_t wsum[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * nch;
    uint64_t run = 0;
    for (uint64_t c0 = 0; c0 < nch; c0 += 256) {
        const uint64_t c = c0 + threadIdx.x;
        const uint64_t v = c < nch ? chunk_bits[base + c] : 0;
        uint64_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        uint64_t all = 0;
        for (int w = 0; w < 8; w++) {
            if (w == warp) inc += all;
            all += wsum[w];
        }
        if (c < nch) chunk_off[base + c] = run + inc - v;
        run += all;
        __syncthreads();
    }
}

// segment of one group in one plane: magnitude bit of each element, with the
// sign bit inserted after each element whose first 1 bit is in the plane
__device__ __forceinline__ uint64_t pb_segment(uint32_t M, uint32_t F, uint32_t S) {
    uint64_t seg = M;
    uint32_t f = F;
    while (f) {   // highest first: the positions below stay in place
        const int j = 31 - __clz(f);
        f &= ~(1u << j);
        const uint64_t low = seg & ((2ull << j) - 1ull);
        const uint64_t high = seg >> (j + 1);
        seg = low | ((uint64_t)((S >> j) & 1u) << (j + 1)) | (high << (j + 2));
    }
    return seg;
}

__global__ void __launch_bounds__(PK_T) k_pb_pack_write(const uint32_t* __restrict__ rows, uint64_t stride, uint64_t n,
                                                        int B, const uint32_t* __restrict__ srow,
                                                        const uint64_t* __restrict__ chunk_off, uint64_t nch,
                                                        const uint16_t* __restrict__ warp_bits,
                                                        const uint32_t* __restrict__ sizes,
                                                        unsigned long long* __restrict__ dst) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t ng = (n + 31) / 32;
    const uint64_t g = (uint64_t)blockIdx.x * PK_T + threadIdx.x;
    const int nvalid = pk_nvalid(g, ng, n);
    const uint32_t S = nvalid ? srow[g] : 0u;
    // lane p: the warp's first bit in planes p and p + 32
    uint64_t off[2];
    {
        uint64_t run = 0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int p = lane + 32 * h;
            const uint64_t bits = p < B ? (uint64_t)sizes[p] * 8 : 0, at = (uint64_t)p * nch + blockIdx.x;
            uint64_t inc = bits;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            off[h] = p < B ? run + inc - bits + chunk_off[at] + warp_bits[at * PK_W + warp] : 0;
            run += __shfl_sync(FULL, inc, 31);
        }
    }
    uint32_t seen = 0;
    pk_planes(rows, stride, g, valid_mask(nvalid), B, [&](int p, uint32_t M) {
        const uint32_t F = M & ~seen;
        seen |= M;
        const uint32_t len = nvalid + __popc(F);
        uint32_t inc = len;
        if (__all_sync(FULL, len == 32)) {   // no signs in the warp
            inc = 32 * (lane + 1);
        } else {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
        }
        const uint64_t at = __shfl_sync(FULL, p < 32 ? off[0] : off[1], p & 31) + inc - len;
        if (len) {
            const uint64_t seg = pb_segment(M, F, S);
            const uint64_t w = at >> 6;
            const int sh = (int)(at & 63);
            atomicOr(dst + w, (unsigned long long)(seg << sh));
            if (sh && sh + (int)len > 64) atomicOr(dst + w + 1, (unsigned long long)(seg >> (64 - sh)));
        }
    });
}

// ---------------------------------------------------------------------------
// parse: reference streams of planes [a, a+np) of one or more levels -> rows
// a..a+np-1, with the unseen / sign rows carried from the planes before a and
// updated.
//
// One CTA per (level, plane), all co-resident (cooperative launch). The chain
// over a level's planes is a software pipeline over chunks of PZ_G groups: a
// plane's CTA receives each chunk's unseen / sign masks from the plane before
// through a ring in global memory (release / acquire flags) and hands them on
// after its plane. Every wait is bounded: past the limit the CTA records
// PRODM_ETIMEOUT in the level's status and returns.
//
// Within a chunk the start of a group depends on the number of sign bits
// before it, and only groups with unseen elements hold sign bits. Those
// groups are taken in steps of up to 32 pairs: for each pair the threads
// parse every start in a window around the expected one, a pair per start and
// thread, and note which slot of the next pair their end leads to (the
// window's middle is the sign count expected from the rate of the groups just
// parsed; the widths, which grow with the root of the distance from the
// step's first group, are laid out over the threads once per chunk); then one
// warp follows the chain of true starts through the slots, and two others
// parse their words while the next step's windows are tried. A true start
// outside its window ends the step there, and the first pair of a step has its
// exact start, so every step goes on. The groups
// without unseen elements hold one bit per element at offsets known once the
// signs before them are counted. One warp of the CTA moves the masks: it
// fetches the next chunk's and hands on the last one's while the other warps
// parse the current one.
// What bounds it is this chain, not memory: one warp taking a plane's groups
// one after the other, a step per sign bit, ran at 570 SM cycles per group in
// the planes where most elements become significant (129^3 fp64, 60 planes:
// all levels' parse 20.0 ms, 4.8 ms this way; with 320 and 416 starts per step
// 5.0 and 5.3 ms).
// ---------------------------------------------------------------------------
constexpr int PZ_R = 8;                      // ring depth (chunks)
constexpr long long kPzSpin = 1ll << 24;     // polls per wait: an acquire load from L2 and a sleep of 0 to 64 ns each
constexpr int PZ_N = 224;                    // parsing threads: starts tried per step
constexpr int PZ_S = PZ_N + 64;              // and the warps that keep the true starts' words
constexpr int PZ_T = PZ_S + 32;              // and the warp that moves the masks
constexpr int PZ_G = 128;                    // groups per chunk
constexpr int PZ_E = 2 * PZ_G;               // ring entry: a chunk's unseen + sign words
// staged stream words (64-bit): a chunk takes at most 2 PZ_G bits x 32, and its
// start lies at most PZ_G / 2 + 1 words behind the first staged one
constexpr int PZ_W = 3 * PZ_G / 2 + 8;
constexpr uint32_t PZ_END = 0xffffu;

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// one lane polls *p until it is above `above`, at most kPzSpin times
__device__ __forceinline__ bool pz_wait(const int* p, int above, int& seen) {
    for (long long spins = 0; (seen = ld_acquire(p)) <= above; spins++) {
        if (spins > kPzSpin) return false;
        __nanosleep(32);
    }
    return true;
}
__device__ __forceinline__ void pz_sync() { asm volatile("bar.sync 1, %0;" ::"n"(PZ_S) : "memory"); }

struct PzMasks {                 // one chunk's masks, updated by the parse
    uint32_t U[PZ_G], S[PZ_G];   // unseen / sign words of its groups
    uint32_t seq[PZ_G + 1];      // groups with unseen elements, in order
    uint32_t PU[PZ_G + 2];       // unseen elements of the groups seq[0..k)
    int nseq;
};
// the smallest start tried of a window of w starts, d unseen elements into the
// step (one value wherever it is computed: no contraction is left open)
__device__ __forceinline__ uint32_t pz_low(float rate, uint32_t d, uint32_t w) {
    return (uint32_t)fmaxf(__fmaf_rn(rate, (float)d, __fmaf_rn(-0.5f, (float)w, 0.5f)), 0.f);
}

struct PzShared {
    uint8_t used[4096];          // four elements: (unseen bits << 8 | stream bits) -> stream bits used
    uint16_t tab[4096];          // and -> magnitude | sign << 4 | bits used << 8
    uint32_t ws[2 * PZ_W];       // the chunk's stream, 32-bit words from word 2 * pb on
    PzMasks m[3];                // chunks c - 1 (handed on), c (parsed), c + 1 (fetched)
    uint32_t M[PZ_G];            // the plane's words of the groups with unseen elements
    uint32_t cnt[PZ_G];          // their sign bits
    uint16_t before[PZ_N];       // per start tried: the step's sign bits before it,
    uint8_t first[PZ_N], both[PZ_N];   // the first group's and the pair's,
    uint16_t next[PZ_N];         // and the slot of the next pair that its end starts, or PZ_END
    uint32_t base[34];           // per pair of a step: its starts' first slot
    uint32_t start[64];          // the true starts of the last step's groups: the sign bits before each
    int npairs;                  // pairs of a full step
    int k0, run;                 // the step: its first group, the sign bits before it,
    float rate;                  // and sign bits expected per unseen element
    int kept, kept_k0, kept_run; // the last step: groups with a true start, ..
};

// One group from the 64 stream bits W at its start: magnitude bits M and signs
// SG of its unseen elements U, by table steps of four elements
__device__ __forceinline__ void pz_group(const uint16_t* tab, uint64_t W, uint32_t U, uint32_t& M, uint32_t& SG) {
    uint32_t m = 0, sg = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t u = i < 2 ? U << (8 - 4 * i) : U >> (4 * i - 8);
        const uint32_t e = tab[(u & 0xf00u) | ((uint32_t)W & 255u)];
        m |= (e & 15u) << (4 * i);
        sg |= ((e >> 4) & 15u) << (4 * i);
        W >>= e >> 8;
    }
    M = m;
    SG = sg;
}
// its sign bits alone
__device__ __forceinline__ uint32_t pz_count(const uint8_t* used, uint64_t W, uint32_t U) {
    uint32_t lo = (uint32_t)W, hi = (uint32_t)(W >> 32), total = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t u = i < 2 ? U << (8 - 4 * i) : U >> (4 * i - 8);
        const uint32_t e = used[(u & 0xf00u) | (lo & 255u)];
        total += e;
        lo = __funnelshift_r(lo, hi, e);
        hi >>= e;
    }
    return total - 32u;
}
// and by one step per sign bit, for planes with few of them: with d sign bits
// taken, the remaining elements' bits are the frame W >> d (bit i = element
// i); the next element to carry a sign is the lowest unseen one whose bit is
// set there
__device__ __forceinline__ uint32_t pz_count_few(uint64_t W, uint32_t U) {
    const uint32_t lo = (uint32_t)W, hi = (uint32_t)(W >> 32);
    uint32_t d = 0;
    for (uint32_t T = U & lo; T && d < 32; T = U & __funnelshift_rc(lo, hi, d)) {
        U &= T ^ (0u - T);   // the elements behind the lowest set one
        d++;
    }
    return d;
}
__device__ __forceinline__ uint64_t pz_window(const uint32_t* ws, uint32_t at) {
    const uint32_t k = at >> 5, sh = at & 31;
    const uint32_t x0 = ws[k], x1 = ws[k + 1], x2 = ws[k + 2];
    return ((uint64_t)__funnelshift_r(x1, x2, sh) << 32) | __funnelshift_r(x0, x1, sh);
}

__device__ __forceinline__ uint32_t warp_scan(uint32_t v, int lane) {   // inclusive
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// one warp: chunk c's masks into m, with the list of its groups with unseen elements
__device__ __forceinline__ void pz_fetch(const PbParse& q, int k, uint64_t c, uint64_t ng, PzMasks& m, int lane) {
    const uint64_t g0 = c * PZ_G;
    const uint32_t* src = q.ring + ((uint64_t)(k - 1) * PZ_R + c % PZ_R) * PZ_E;
    uint32_t U[PZ_G / 32], S[PZ_G / 32];
#pragma unroll
    for (int t = 0; t < PZ_G / 32; t++) {
        const int i = 32 * t + lane;
        if (k) {
            U[t] = __ldcg(src + i);
            S[t] = __ldcg(src + PZ_G + i);
        } else {
            U[t] = g0 + i < ng ? q.unseen[g0 + i] : 0u;
            S[t] = g0 + i < ng ? q.signs[g0 + i] : 0u;
        }
    }
    uint32_t at = 0, u0 = 0;
#pragma unroll
    for (int t = 0; t < PZ_G / 32; t++) {
        m.U[32 * t + lane] = U[t];
        m.S[32 * t + lane] = S[t];
        const uint32_t has = __ballot_sync(FULL, U[t] != 0), own = __popc(U[t]);
        const uint32_t inc = warp_scan(own, lane);
        if (U[t]) {
            const uint32_t i = at + __popc(has & ((1u << lane) - 1u));
            m.seq[i] = 32 * t + lane;
            m.PU[i] = u0 + inc - own;
        }
        at += __popc(has);
        u0 += __shfl_sync(FULL, inc, 31);
    }
    if (lane == 0) {
        m.nseq = (int)at;
        m.seq[at] = 0;
        m.PU[at] = u0;
        m.PU[at + 1] = u0;
    }
}

__global__ void __launch_bounds__(PZ_T, 3) k_pb_parse(const __grid_constant__ PbParseSet set) {
    extern __shared__ __align__(16) unsigned char pz_smem[];
    PzShared& sh = *reinterpret_cast<PzShared*>(pz_smem);
    int l = 0;   // the CTA's level and plane
    while (l + 1 < set.n && (int)blockIdx.x >= set.seg[l + 1].cta0) l++;
    const PbParse& q = set.seg[l];
    const int k = (int)blockIdx.x - q.cta0;
    const int np = q.np, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t n = q.n;
    int* produced = q.flags;
    int* consumed = q.flags + np;
    const uint64_t ng = (n + 31) / 32, nch = (ng + PZ_G - 1) / PZ_G;
    const uint64_t* words = q.planes[k];
    const uint64_t nw = q.nwords[k];
    uint32_t* row = q.rows + (uint64_t)(q.a + k) * q.stride;
    const bool last = k == np - 1, mover = tid >= PZ_S, keeper = tid >= PZ_N && !mover;
    for (int i = tid; i < 4096; i += PZ_T) {
        const uint32_t u = i >> 8;
        uint32_t w = i & 255, m = 0, sg = 0, used = 0;
        for (int j = 0; j < 4; j++) {
            const uint32_t b = w & 1u;
            w >>= 1;
            used++;
            m |= b << j;
            if (b && ((u >> j) & 1u)) {
                sg |= (w & 1u) << j;
                w >>= 1;
                used++;
            }
        }
        sh.tab[i] = (uint16_t)(m | sg << 4 | used << 8);
        sh.used[i] = (uint8_t)used;
    }
    int seen_produced = 0, seen_consumed = 0;   // mover lane 0: the neighbours' progress as last read
    int gave_up = 0;                            // mover: a wait ran out
    // the mover warp, while the others parse chunk c: chunk c - 1 to the next
    // plane (or the last plane's masks to the level's rows), chunk c + 1 in
    auto move = [&](uint64_t c, bool give, bool take) {
        bool ok = true;
        if (give) {
            const uint64_t o = c - 1, g0 = o * PZ_G;
            const PzMasks& m = sh.m[o % 3];
            if (last) {
                for (int i = lane; i < PZ_G; i += 32)
                    if (g0 + i < ng) {
                        q.unseen[g0 + i] = m.U[i];
                        q.signs[g0 + i] = m.S[i];
                    }
            } else {
                if (lane == 0 && (int)o - seen_consumed >= PZ_R)
                    ok = pz_wait(consumed + k, (int)o - PZ_R, seen_consumed);
                ok = __shfl_sync(FULL, ok, 0);
                if (ok) {
                    uint32_t* dst = q.ring + ((uint64_t)k * PZ_R + o % PZ_R) * PZ_E;
                    for (int i = lane; i < PZ_G; i += 32) {
                        __stcg(dst + i, m.U[i]);
                        __stcg(dst + PZ_G + i, m.S[i]);
                    }
                    __syncwarp();
                    if (lane == 0) {
                        __threadfence();
                        st_release(produced + k, (int)o + 1);
                    }
                }
            }
        }
        if (take && ok) {
            const uint64_t t = c + 1;
            if (k) {
                if (lane == 0 && seen_produced <= (int)t) ok = pz_wait(produced + k - 1, (int)t, seen_produced);
                ok = __shfl_sync(FULL, ok, 0);
            }
            if (ok) {
                pz_fetch(q, k, t, ng, sh.m[t % 3], lane);
                __syncwarp();
                if (k && lane == 0) st_release(consumed + k - 1, (int)t + 1);
            }
        }
        if (!ok) gave_up = 1;
    };
    if (mover) move(~0ull, false, true);   // chunk 0
    uint64_t pos = 0, pb = 0;          // the chunk's first bit; the first staged word
    uint64_t ahead = tid < PZ_W && (uint64_t)tid < nw ? __ldcs(words + tid) : 0ull;   // words pb + tid
    float rs = 0.f, ru = 0.f;          // warp 0: sign bits and unseen elements of the groups just parsed
    for (uint64_t c = 0; c < nch; c++) {
        const uint64_t g0 = c * PZ_G;
        // stage the stream; the next chunk starts PZ_G / 2 words on or later
        if (tid < PZ_W) {
            sh.ws[2 * tid] = (uint32_t)ahead;
            sh.ws[2 * tid + 1] = (uint32_t)(ahead >> 32);
            const uint64_t w = (pos >> 6) + PZ_G / 2 + tid;
            ahead = w < nw ? __ldcs(words + w) : 0ull;
        }
        if (tid < PZ_G) sh.cnt[tid] = 0;
        const uint32_t p0 = (uint32_t)(pos - 64 * pb);
        pb = (pos >> 6) + PZ_G / 2;
        if (__syncthreads_or(gave_up)) {   // (also: the stream and the mover's chunk c are there)
            if (tid == 0) atomicExch(q.status, PRODM_ETIMEOUT);
            return;
        }
        PzMasks& m = sh.m[c % 3];
        uint32_t run_all = 0;
        if (mover) {
            move(c, c > 0, c + 1 < nch);
        } else {
            const int nseq = m.nseq;
            int k0 = 0;
            uint32_t run = 0;
            if (warp == 0) {   // the chunk's windows: 2.5 sigma on either side
                const float p = __fdividef(rs + 0.5f, ru + 1.f);
                const float v = ((p - p * p) + 0.002f) * 2.f * __fdividef((float)m.PU[nseq], (float)max(nseq, 1));
                const float vi = v * (float)lane;
                const uint32_t w = lane ? min(3u + (uint32_t)(5.f * vi * rsqrtf(vi)), 120u) : 1u;
                const uint32_t inc = warp_scan(w, lane);
                const uint32_t fit = __ballot_sync(FULL, inc <= PZ_N);
                sh.base[lane + 1] = inc;
                if (lane == 0) {
                    sh.base[0] = 0;
                    sh.base[33] = ~0u;
                    sh.npairs = __popc(fit);
                    sh.k0 = 0;
                    sh.run = 0;
                    sh.rate = p;
                    sh.kept = 0;
                }
            }
            pz_sync();
            // this thread's pair and place in its window
            const int npairs = sh.npairs;
            int pi = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (pi + step < npairs && sh.base[pi + step] <= (uint32_t)tid) pi += step;
            const uint32_t b0 = sh.base[pi], b1 = sh.base[pi + 1], b2 = sh.base[pi + 2];
            const bool mine = !keeper && (uint32_t)tid < b1, more = pi + 1 < npairs;
            for (;;) {
                const int first = sh.k0;
                if (keeper) {   // the last step's true starts: thread i parses group i's words
                    const int i = tid - PZ_N;
                    if (i < sh.kept) {
                        const uint32_t g = m.seq[sh.kept_k0 + i], U = m.U[g];
                        uint32_t M, SG;
                        pz_group(sh.tab, pz_window(sh.ws, p0 + sh.kept_run + sh.start[i] + 32 * g), U, M, SG);
                        sh.M[g] = M;
                        sh.cnt[g] = __popc(M & U);
                        m.U[g] = U & ~M;
                        m.S[g] |= SG;
                    }
                } else if (mine && first + 2 * pi < nseq) {   // try one start of one pair
                    const int kk = first + 2 * pi;
                    const uint32_t ga = m.seq[kk], gb = m.seq[kk + 1];
                    const uint32_t P0 = m.PU[first], Pa = m.PU[kk], Pb = m.PU[kk + 1], Pc = m.PU[kk + 2];
                    const float rate = sh.rate;
                    // sign bits before it in this step
                    const uint32_t x = pi ? pz_low(rate, Pa - P0, b1 - b0) + (uint32_t)tid - b0 : 0u;
                    const uint32_t at = p0 + sh.run + x;
                    const uint32_t Ua = m.U[ga], Ub = Pc != Pb ? m.U[gb] : 0u;
                    const uint64_t Wa = pz_window(sh.ws, at + 32 * ga);
                    uint32_t cc;
                    if (rate < 0.12f) {
                        cc = pz_count_few(Wa, Ua);
                        sh.first[tid] = (uint8_t)cc;
                        cc += pz_count_few(pz_window(sh.ws, at + 32 * gb + cc), Ub);
                    } else {
                        cc = pz_count(sh.used, Wa, Ua);
                        sh.first[tid] = (uint8_t)cc;
                        cc += pz_count(sh.used, pz_window(sh.ws, at + 32 * gb + cc), Ub);
                    }
                    uint32_t nx = PZ_END;
                    if (more && kk + 2 < nseq) {   // below the window the difference wraps
                        const uint32_t y = x + cc - pz_low(rate, Pc - P0, b2 - b1);
                        if (y < b2 - b1) nx = b1 + y;
                    }
                    sh.before[tid] = (uint16_t)x;
                    sh.next[tid] = (uint16_t)nx;
                    sh.both[tid] = (uint8_t)cc;
                }
                if (first >= nseq) break;   // every group with unseen elements is parsed
                pz_sync();
                if (warp == 0) {   // follow the true starts (lane i: pair i)
                    uint32_t slot = 0, own = 0;
                    int done = 0;
                    for (;;) {
                        const uint32_t nx = sh.next[slot];
                        if (lane == done) own = slot;
                        done++;
                        if (nx == PZ_END) break;   // at the latest behind the step's last pair
                        slot = nx;
                    }
                    const uint32_t r = sh.before[slot] + sh.both[slot];
                    const int k1 = min(k0 + 2 * done, nseq);
                    rs = 0.25f * rs + (float)r;
                    ru = 0.25f * ru + (float)(m.PU[k1] - m.PU[k0]);
                    const uint32_t x = sh.before[own];
                    sh.start[2 * lane] = x;
                    sh.start[2 * lane + 1] = x + sh.first[own];
                    if (lane == 0) {
                        sh.kept = k1 - k0;
                        sh.kept_k0 = k0;
                        sh.kept_run = (int)run;
                        sh.k0 = k1;
                        sh.run = (int)(run + r);
                        sh.rate = __fdividef(rs + 0.5f, ru + 1.f);
                    }
                    k0 = k1;
                    run += r;
                }
                pz_sync();
            }
            pz_sync();   // the last step's words
            // words of all groups: thread t < PZ_G takes group t
            if (tid < PZ_G) {
                const int nv = pk_nvalid(g0 + tid, ng, n);
                const uint32_t own = sh.cnt[tid];
                uint32_t before = warp_scan(own, lane) - own;
                for (int j = 0; j < warp; j++) before += __reduce_add_sync(FULL, sh.cnt[32 * j + lane]);
                uint32_t M;
                if (m.U[tid] != 0 || own != 0) {   // it had unseen elements: parsed above
                    M = sh.M[tid];
                } else {
                    const uint32_t at = p0 + 32u * tid + before;
                    M = __funnelshift_r(sh.ws[at >> 5], sh.ws[(at >> 5) + 1], at & 31);
                }
                if (nv > 0) row[g0 + tid] = M & valid_mask(nv);
            }
            run_all = (uint32_t)sh.run;
        }
        if (mover) run_all = 0;
        __syncthreads();   // the chunk is parsed, and the mover is done with its neighbours
        const uint64_t left = n - 32 * g0;
        pos += (left < 32 * PZ_G ? left : 32 * PZ_G) + run_all;
    }
    // the last chunk's masks
    if (mover && nch) move(nch, true, false);
    gave_up = __syncthreads_or(gave_up);
    if (tid == 0) {
        if (gave_up) atomicExch(q.status, PRODM_ETIMEOUT);
        // a well-formed stream ends in its last word
        else if ((pos + 63) / 64 != nw) atomicCAS(q.status, 0, PRODM_ECORRUPT);
    }
}

// unseen row of a fresh level: every element present
__global__ void k_pb_init_unseen(uint32_t* __restrict__ unseen, uint32_t* __restrict__ signs, uint64_t n) {
    const uint64_t ng = (n + 31) / 32;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += (uint64_t)gridDim.x * blockDim.x) {
        unseen[g] = valid_mask(pk_nvalid(g, ng, n));
        signs[g] = 0;
    }
}

}  // namespace

uint64_t pb_groups(uint64_t n) { return (n + 31) / 32; }
uint64_t pb_row_words(uint64_t n) { return (pb_groups(n) + 3) / 4 * 4; }

template <class T>
static uint32_t pb_number(PbSet<T>& set) {
    uint64_t c = 0;
    for (int l = 0; l < set.n; l++) {
        set.seg[l].chunk0 = (uint32_t)c;
        c += (pb_groups(set.seg[l].n) + PB_CHUNK - 1) / PB_CHUNK;
    }
    return (uint32_t)c;
}

template <class T>
int launch_pb_encode(PbSet<T> set, int B, cudaStream_t st) {
    if (B < 1 || B > (sizeof(T) == 8 ? 63 : 32)) return fail(PRODM_EINVAL, "perbit: num_bitplanes out of range");
    for (int l = 0; l < set.n;) {   // counts of consecutive levels in one clear
        int m = l + 1;
        while (m < set.n && set.seg[m].counts + 64 == set.seg[m - 1].counts) m++;
        PRODM_CUDA(cudaMemsetAsync(set.seg[m - 1].counts, 0, (size_t)(m - l) * 64 * sizeof(uint32_t), st));
        l = m;
    }
    const uint32_t total = pb_number(set);
    if (!total) return PRODM_OK;
    const size_t smem = (size_t)(B + 1) * PB_LD * 4;
    const unsigned grid = persistent_grid_for((const void*)k_pb_encode<T>, 256, smem, total, 1u << 20);
    count_launch();
    cudaError_t e = launch_chain(true, k_pb_encode<T>, dim3(grid), dim3(256), smem, st, set, total, B);
    if (e != cudaSuccess) return cuda_status(e, "k_pb_encode");
    count_launch();
    e = launch_chain(true, k_pb_sizes<T>, dim3(set.n), dim3(64), 0, st, set, B);
    if (e != cudaSuccess) return cuda_status(e, "k_pb_sizes");
    return PRODM_OK;
}

// B: most planes a level may have (shared memory)
template <class T>
int launch_pb_decode(PbSet<T> set, int B, int s, int e, cudaStream_t st) {
    const uint32_t total = pb_number(set);
    if (!total) return PRODM_OK;
    bool counts = false;
    for (int l = 0; l < set.n; l++) counts |= set.seg[l].dnum != nullptr;
    const size_t smem = (size_t)((counts ? B : e - s) + 2) * PB_LD * 4;
    const unsigned grid = persistent_grid_for((const void*)k_pb_decode<T>, 256, smem, total, 1u << 20);
    count_launch();
    const cudaError_t err = launch_chain(true, k_pb_decode<T>, dim3(grid), dim3(256), smem, st, set, total, s, e);
    if (err != cudaSuccess) return cuda_status(err, "k_pb_decode");
    return PRODM_OK;
}

size_t pb_pack_scratch_bytes(uint64_t n, int B) {
    const uint64_t nch = (pb_groups(n) + PK_T - 1) / PK_T;
    return ((size_t)B * nch * (8 + 4 + 2 * PK_W) + 511) / 256 * 256;   // a multiple of 256 bytes
}

int launch_pb_pack(const uint32_t* rows, uint64_t stride, uint64_t n, int B, const uint32_t* sizes, uint64_t total,
                   uint8_t* dst, void* scratch, cudaStream_t st) {
    if ((uintptr_t)dst % 8) return fail(PRODM_EINVAL, "perbit pack: destination must be 8-byte aligned");
    const uint64_t nch = (pb_groups(n) + PK_T - 1) / PK_T;
    uint64_t* chunk_off = (uint64_t*)scratch;
    uint32_t* chunk_bits = (uint32_t*)(chunk_off + (uint64_t)B * nch);
    uint16_t* warp_bits = (uint16_t*)(chunk_bits + (uint64_t)B * nch);
    PRODM_CUDA(cudaMemsetAsync(dst, 0, total, st));
    if (nch == 0) return PRODM_OK;
    k_pb_pack_count<<<(unsigned)nch, PK_T, 0, st>>>(rows, stride, n, B, chunk_bits, nch, warp_bits);
    PRODM_CHECK_LAUNCH("k_pb_pack_count");
    k_pb_pack_scan<<<B, 256, 0, st>>>(chunk_bits, nch, chunk_off);
    PRODM_CHECK_LAUNCH("k_pb_pack_scan");
    k_pb_pack_write<<<(unsigned)nch, PK_T, 0, st>>>(rows, stride, n, B, rows + (uint64_t)B * stride, chunk_off, nch,
                                                    warp_bits, sizes, (unsigned long long*)dst);
    PRODM_CHECK_LAUNCH("k_pb_pack_write");
    return PRODM_OK;
}

int launch_pb_init_unseen(uint32_t* unseen, uint32_t* signs, uint64_t n, cudaStream_t st) {
    k_pb_init_unseen<<<grid_for(pb_groups(n), 256), 256, 0, st>>>(unseen, signs, n);
    PRODM_CHECK_LAUNCH("k_pb_init_unseen");
    return PRODM_OK;
}

// The parse of several levels' planes in as few launches as are co-resident
// (the planes' CTAs wait on one another, so they are launched cooperatively).
// Scratch: the plane pointers and word counts, a ring and two flags per plane.
int launch_pb_parse(const std::vector<PbParseJob>& jobs, cudaStream_t st) {
    size_t planes = 0;
    for (const PbParseJob& j : jobs) {
        const size_t np = j.planes.size();
        if (np < 1 || np > 64 || j.nwords.size() != np) return fail(PRODM_EINVAL, "perbit parse: 1..64 planes per level");
        planes += np;
    }
    if (!planes) return PRODM_OK;
    const size_t head = (planes * 16 + 255) / 256 * 256, fl = (planes * 8 + 255) / 256 * 256;
    std::vector<uint64_t> hv;
    hv.reserve(2 * planes);
    for (const PbParseJob& j : jobs) {
        for (const uint64_t* p : j.planes) hv.push_back((uint64_t)(uintptr_t)p);
        for (uint64_t w : j.nwords) hv.push_back(w);
    }
    Scratch mem(st);
    PRODM_CUDA(mem.alloc(head + fl + planes * PZ_R * PZ_E * 4));
    uint8_t* scratch = mem.get();
    const int rc = launch_put(scratch, hv.data(), hv.size() * 8, st);
    if (rc) return rc;
    cudaError_t e = cudaMemsetAsync(scratch + head, 0, fl, st);
    const unsigned resident = resident_ctas((const void*)k_pb_parse, PZ_T, sizeof(PzShared));
    size_t at = 0, next = 0;
    while (e == cudaSuccess && next < jobs.size()) {
        PbParseSet set;
        set.n = 0;
        unsigned ctas = 0;
        while (next < jobs.size() && set.n < kPbParseLevels &&
               (ctas == 0 || ctas + jobs[next].planes.size() <= resident)) {
            const PbParseJob& j = jobs[next++];
            PbParse& q = set.seg[set.n++];
            q.np = (int)j.planes.size();
            q.planes = (const uint64_t* const*)((uint64_t*)scratch + 2 * at);
            q.nwords = (const uint64_t*)scratch + 2 * at + q.np;
            q.flags = (int*)(scratch + head) + 2 * at;
            q.ring = (uint32_t*)(scratch + head + fl) + at * PZ_R * PZ_E;
            q.rows = j.rows;
            q.stride = j.stride;
            q.unseen = j.unseen;
            q.signs = j.signs;
            q.status = j.status;
            q.n = j.n;
            q.a = j.a;
            q.cta0 = (int)ctas;
            ctas += (unsigned)q.np;
            at += q.np;
        }
        count_launch();
        void* args[] = {(void*)&set};
        e = cudaLaunchCooperativeKernel((const void*)k_pb_parse, dim3(ctas), dim3(PZ_T), args, sizeof(PzShared), st);
    }
    if (e != cudaSuccess) return cuda_status(e, "k_pb_parse");
    return PRODM_OK;
}

template int launch_pb_encode<float>(PbSet<float>, int, cudaStream_t);
template int launch_pb_encode<double>(PbSet<double>, int, cudaStream_t);
template int launch_pb_decode<float>(PbSet<float>, int, int, int, cudaStream_t);
template int launch_pb_decode<double>(PbSet<double>, int, int, int, cudaStream_t);

}  // namespace prodm
