// Negabinary fp32 codec bodies (bit transposes, chunk encode / decode),
// shared by the single-level kernels and the multi-field batched kernels.
#pragma once
#include "common.cuh"

namespace prodm {

// ---------------------------------------------------------------------------
// 32 x 32 bit transpose across a warp: lane e holds row e on entry; on exit
// lane k holds the word whose bit e is bit k of row e. Five exchange stages
// with the lane l ^ j: the two byte-granular stages (j = 16, 8) are one byte
// permute each with a per-lane selector, the three sub-byte stages one
// rotate (a funnel shift by a per-lane amount) and one masked merge each, so a
// stage is a shuffle plus one or two instructions.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), (lane & 16) ? 0x3276u : 0x5410u);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), (lane & 8) ? 0x3715u : 0x6240u);
#pragma unroll
    for (int j = 4; j > 0; j >>= 1) {
        const uint32_t m = j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
        const bool hi = (lane & j) != 0;
        const uint32_t keep = hi ? ~m : m;                       // bits of x that stay
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        const uint32_t ys = __funnelshift_l(y, y, hi ? 32 - j : j);   // partner's bits moved into place
        x = (x & keep) | (ys & ~keep);
    }
    return x;
}

// x * 2^e, equal to ldexpf(x, e): a single multiplication by an exact power of
// two rounds once, as ldexpf does, whenever 2^e is a normal float
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ bool pow2_normal(int e) { return e >= -126 && e <= 127; }
__device__ __forceinline__ float scale2(float v, int e, bool fast, float sc) { return fast ? v * sc : ldexpf(v, e); }

// asynchronous 16-byte global -> shared copy (cp.async), both addresses 16-byte aligned (L2 only)
__device__ __forceinline__ void cp_async16(uint32_t* dst, const uint32_t* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// The byte-granular second stage and the three sub-byte stages of a half
// transpose (below), on the 16 words the first stage selected.
__device__ __forceinline__ void transpose32_half_tail(uint32_t (&a)[16]) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t x = a[k], y = a[k + 8];
        a[k] = __byte_perm(x, y, 0x6240u);
        a[k + 8] = __byte_perm(x, y, 0x7351u);
    }
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const int j = 4 >> s;
        const uint32_t m = s == 0 ? 0x0f0f0f0fu : s == 1 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = (i / j) * 2 * j + (i % j);
            const uint32_t t = ((a[k] >> j) ^ a[k + j]) & m;
            a[k + j] ^= t;
            a[k] ^= t << j;
        }
    }
}

// Half of a 32 x 32 bit transpose: rows R[0..31] (R[r] bit e) -> the 16
// words out[v] (v = 16 * half + 0..15) whose bit r is R[r] bit v. The two
// byte-granular stages are byte permutes, the three sub-byte stages
// mask-and-shift swaps.
__device__ __forceinline__ void transpose32_half(const uint32_t (&R)[32], int half, uint32_t (&a)[16]) {
    const uint32_t sel16 = half ? 0x7632u : 0x5410u;
#pragma unroll
    for (int k = 0; k < 16; k++) a[k] = __byte_perm(R[k], R[k + 16], sel16);
    transpose32_half_tail(a);
}

constexpr int NB_CHUNK = 256;        // blocks per CTA chunk
constexpr int NB_TILE_LD = NB_CHUNK + 1;   // padded tile row: conflict-free column writes

// 32 x 32 bit transpose of one lane's words: bit v of a[k] becomes bit k of
// a[v] (halves and bytes by byte selection, then 4, 2 and 1 bits)
__device__ __forceinline__ void transpose32_lane(uint32_t (&a)[32]) {
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const uint32_t x = a[i], y = a[i + 16];
        a[i] = __byte_perm(x, y, 0x5410u);
        a[i + 16] = __byte_perm(x, y, 0x7632u);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int k = (i & 7) + 2 * (i & 8);
        const uint32_t x = a[k], y = a[k + 8];
        a[k] = __byte_perm(x, y, 0x6240u);
        a[k + 8] = __byte_perm(x, y, 0x7351u);
    }
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const int j = 4 >> s;
        const uint32_t m = s == 0 ? 0x0f0f0f0fu : s == 1 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int k = (i / j) * 2 * j + (i % j);
            const uint32_t x = a[k], y = a[k + j];
            a[k] = (x & m) | ((y << j) & ~m);
            a[k + j] = ((x >> j) & m) | (y & ~m);
        }
    }
}

// Encode the chunks blockIdx.x, blockIdx.x + gridDim.x, .. of total chunks of
// NB_CHUNK 32-value blocks (NegaBinaryBPEncoder.hpp:18-62): src_of(chunk)
// gives the level that holds a chunk and the chunk's number in it. A warp
// takes 32 blocks: their values go to shared memory by cp.async, each lane
// reads the 32 values of its own block back, transposes their digits in
// registers, and the 32 lanes' words of a plane are one 128-byte store. The
// next 32 blocks are on their way while these are transposed. 100 x 500 x 500:
// 55 us with a warp transpose by shuffles per block and a tile of the words in
// shared memory (integer pipe 63 % busy, shared memory and shuffles 48 %), 38 us
// so (DRAM floor 30); 64 fields of 173 M values 414 and 301 us (floor 208).
// The error-table variant is in bitplane.cu.
struct NbSrc {
    const float* x;
    uint32_t* words;
    uint64_t n, nblocks, stride, chunk;
    float scale;
    int se;
    bool fast;
};
constexpr int NB_ROW = 36;   // a block's values in shared memory, 16-byte rows without bank conflicts
constexpr int NB_STAGE = (NB_CHUNK / 32) * 32 * NB_ROW;   // words of a CTA

template <class SrcOf>
__device__ __forceinline__ void nb_encode32_chunks(uint64_t total, int B, uint32_t* stage, SrcOf src_of) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* buf = stage + warp * 32 * NB_ROW;
    uint64_t c = blockIdx.x;
    if (c >= total) return;
    auto fetch = [&](const NbSrc& q) {
        const uint64_t b = q.chunk * NB_CHUNK + (uint64_t)warp * 32;
        if (b < q.nblocks) {
            const uint64_t left = q.n - b * 32;
            const int have = left < 1024 ? (int)left : 1024;
            const float* src = q.x + b * 32;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(buf + lane);
#pragma unroll
            for (int g = 0; g < 32; g++) {
                const int i = 32 * g + lane;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + g * NB_ROW * 4),
                             "l"(src + (i < have ? i : 0)), "r"(i < have ? 4 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    NbSrc q = src_of(c);
    fetch(q);
    for (;;) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        uint32_t a[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint4 v = *reinterpret_cast<const uint4*>(buf + lane * NB_ROW + 4 * i);
            a[4 * i] = v.x;
            a[4 * i + 1] = v.y;
            a[4 * i + 2] = v.z;
            a[4 * i + 3] = v.w;
        }
        __syncwarp();
        const NbSrc h = q;
        c += gridDim.x;
        if (c < total) {
            q = src_of(c);
            fetch(q);
        }
        const uint64_t b = h.chunk * NB_CHUNK + (uint64_t)warp * 32;
        if (b < h.nblocks) {
            // NegaBinaryBPEncoder.hpp:42; the scaling is an exact
            // multiplication whenever 2^se is a normal float
            if (h.fast) {
#pragma unroll
                for (int i = 0; i < 32; i++) a[i] = nb_from_bin((int32_t)(__uint_as_float(a[i]) * h.scale));
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) a[i] = nb_from_bin((int32_t)ldexpf(__uint_as_float(a[i]), h.se));
            }
            transpose32_lane(a);   // a[k]: digit k of the block's values
            if (b + lane < h.nblocks) {
                uint32_t* dst = h.words + (uint64_t)(B - 1) * h.stride + b + lane;
#pragma unroll
                for (int k = 0; k < 32; k++)
                    if (k < B) {
                        *dst = a[k];
                        dst -= h.stride;
                    }
            }
        }
        if (c >= total) break;
    }
}

// Decode chunk c of planes [s, s+num) (plane s+i at base + i * stride):
// coalesced tile load, one warp transpose per block, coalesced stores.
__device__ __forceinline__ void nb_decode32_chunk(const uint32_t* __restrict__ base, uint64_t stride, uint64_t n,
                                                  uint64_t nblocks, int num, int e, int exp, bool dfast, float dscale,
                                                  uint64_t c, uint32_t* tile, float* __restrict__ out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool neg = num != 0 && (e & 1);                   // NegaBinaryBPEncoder.hpp:153, :177
    const uint64_t cb0 = c * NB_CHUNK;
    const int nvalid = (int)((nblocks - cb0) < (uint64_t)NB_CHUNK ? (nblocks - cb0) : NB_CHUNK);
    for (int p = warp; p < num; p += 8) {
        const uint32_t* src = base + (uint64_t)p * stride + cb0;
        uint32_t* row = tile + p * NB_TILE_LD;
        for (int j = lane; j < nvalid; j += 32) row[j] = __ldcs(src + j);
    }
    __syncthreads();
    for (int j = 0; j < 32; j++) {
        const int bl = warp * 32 + j;
        if (bl >= nvalid) break;
        const uint32_t w = lane < num ? tile[lane * NB_TILE_LD + bl] : 0u;
        const uint32_t col = transpose32(w, lane);      // bit i = digit of plane s+i
        const uint32_t a = num ? (__brev(col) >> (32 - num)) : 0u;
        const float val = num ? (dfast ? (float)nb_to_bin(a) * dscale : ldexpf((float)nb_to_bin(a), exp - e)) : 0.f;
        const uint64_t i = (cb0 + bl) * 32 + lane;
        if (i < n) out[i] = neg ? -val : val;
    }
    __syncthreads();
}

}  // namespace prodm
