// Layout conversion between the aligned device stream layout and the
// reference level-file bytes, plus small reductions (sm_103a).
//
// Reference level file (FileWriter.hpp:16-31 with NullLevelCompressor): the
// streams of planes 0..B-1 concatenated; for the grouped encoder stream 0 is
// [u32 nblocks][u8 rb x nblocks][words] (GroupedBPEncoder.hpp:370-377), so
// every later word may sit at any byte offset.
#include <cstring>

#include "common.cuh"
#include "kernels.cuh"

namespace prodm {

namespace {

template <class W>
__device__ __forceinline__ void store_bytes(uint8_t* dst, W w) {
    if (((uintptr_t)dst & (sizeof(W) - 1)) == 0) {
        *(W*)dst = w;
    } else {
#pragma unroll
        for (int i = 0; i < (int)sizeof(W); i++) dst[i] = (uint8_t)(w >> (8 * i));
    }
}
template <class W>
__device__ __forceinline__ W load_bytes(const uint8_t* src) {
    if (((uintptr_t)src & (sizeof(W) - 1)) == 0) return *(const W*)src;
    W w = 0;
#pragma unroll
    for (int i = 0; i < (int)sizeof(W); i++) w |= (W)src[i] << (8 * i);
    return w;
}

// one CTA row of threads per plane (blockIdx.y = plane); plane p at planes + p * cap
template <class W>
__global__ void k_gr_pack(const W* __restrict__ planes, uint64_t cap, const uint32_t* __restrict__ sizes,
                          uint64_t nblocks, const uint8_t* __restrict__ rbs, uint8_t* __restrict__ dst) {
    const int p = blockIdx.y;
    uint64_t off = 0;
    for (int q = 0; q < p; q++) off += sizes[q];
    uint64_t bytes = sizes[p];
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, ts = (uint64_t)gridDim.x * blockDim.x;
    if (p == 0) {
        uint64_t hdr = 4 + nblocks;
        for (uint64_t i = t0; i < hdr; i += ts) {
            uint8_t v;
            if (i < 4) v = (uint8_t)((uint32_t)nblocks >> (8 * i));
            else v = rbs[i - 4];
            dst[i] = v;
        }
        off += hdr;
        bytes -= hdr;
    }
    const uint64_t nw = bytes / sizeof(W);
    const W* src = planes + (uint64_t)p * cap;
    for (uint64_t w = t0; w < nw; w += ts) store_bytes<W>(dst + off + w * sizeof(W), src[w]);
}

// the planes travel in the launch; table (nullable) receives their addresses
template <class W>
__global__ void k_unpack_planes(const uint8_t* __restrict__ src, const __grid_constant__ UnpackSet set,
                                void** __restrict__ table) {
    const int p = blockIdx.y;
    const uint64_t nw = set.words[p];
    const uint8_t* s = src + set.off[p];
    W* d = (W*)set.dst[p];
    if (table && blockIdx.x == 0 && threadIdx.x == 0) table[p] = d;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x)
        d[w] = load_bytes<W>(s + w * sizeof(W));
}

template <class T>
__global__ void k_maxabs(const T* __restrict__ x, uint64_t n, typename KeyOf<T>::type* key) {
    using K = typename KeyOf<T>::type;
    K m = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        K k = abs_key(x[i]);
        m = max_key(k, m);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        K w = __shfl_xor_sync(0xffffffffu, m, o);
        m = max_key(w, m);
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(key, m);
}

// level error bound = max (x4 for negabinary, ComposedRefactor.hpp:111-112)
template <class T>
__global__ void k_bounds(const typename KeyOf<T>::type* __restrict__ keys, int nl, int negabinary, T* __restrict__ bounds) {
    pdl_wait();
    pdl_release();
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < nl) {
        T m = key_to_val(keys[l], T());
        bounds[l] = negabinary ? m * (T)4 : m;
    }
}

__global__ void k_fill_u32(uint32_t* dst, uint64_t n, uint32_t v) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = v;
}

// Tables made on the host for one call (factors, sizes, stream descriptors)
// travel in launches of their own where nothing waits for the call's end. An
// asynchronous copy from pageable memory may read its source after the call has
// returned: the runtime promises no staging, a GPU with access to pageable
// memory may read it in place, and in a captured graph the copy reads it at
// every replay. What it costs is the launch, about 4 us more than a small copy
// (257^3 fp32 files through the lossless stage, eleven uploads a pass: 0.84-0.86
// ms by copies, 0.88-0.92 by launches), so calls that wait anyway copy and keep
// the table until then. The host pays for the whole parameter, so there are three
// sizes of it; larger tables take several launches of the largest.
template <int WORDS>
struct PutWords {
    uint32_t w[WORDS];
};
constexpr int kPutSmall = 256, kPutMiddle = 2048, kPutLarge = 8000;   // (a kernel's parameters hold 32,764 bytes)
template <int WORDS>
__global__ void __launch_bounds__(256) k_put(uint32_t* __restrict__ dst, uint32_t n,
                                             const __grid_constant__ PutWords<WORDS> src) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) dst[i] = src.w[i];
}
template <int WORDS>
int put_words(uint32_t* dst, const uint8_t* src, uint32_t n, cudaStream_t st) {
    PutWords<WORDS> v;
    memcpy(v.w, src, (size_t)n * 4);
    k_put<WORDS><<<(n + 255) / 256, 256, 0, st>>>(dst, n, v);
    PRODM_CHECK_LAUNCH("k_put");
    return PRODM_OK;
}

}  // namespace

// Tables above eight launches (factors of dims of tens of thousands of nodes)
// are copied, and the call waits for the copy.
int launch_put(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes > 8 * (size_t)kPutLarge * 4) {
        PRODM_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        PRODM_CUDA(cudaStreamSynchronize(st));
        return PRODM_OK;
    }
    uint32_t* to = (uint32_t*)dst;
    const uint8_t* from = (const uint8_t*)src;
    int rc = PRODM_OK;
    for (size_t n = bytes / 4; n && !rc;) {
        const uint32_t m = (uint32_t)(n < kPutLarge ? n : kPutLarge);
        rc = m <= kPutSmall    ? put_words<kPutSmall>(to, from, m, st)
             : m <= kPutMiddle ? put_words<kPutMiddle>(to, from, m, st)
                               : put_words<kPutLarge>(to, from, m, st);
        to += m;
        from += (size_t)m * 4;
        n -= m;
    }
    return rc;
}

int launch_gr_pack(const void* planes, uint64_t cap, const uint32_t* sizes, int B, uint64_t nblocks, const uint8_t* rbs,
                   int word_bytes, uint8_t* dst, cudaStream_t st) {
    dim3 grid(grid_for(2 * nblocks, 256, 1), B);
    if (word_bytes == 4) k_gr_pack<uint32_t><<<grid, 256, 0, st>>>((const uint32_t*)planes, cap, sizes, nblocks, rbs, dst);
    else k_gr_pack<uint64_t><<<grid, 256, 0, st>>>((const uint64_t*)planes, cap, sizes, nblocks, rbs, dst);
    PRODM_CHECK_LAUNCH("k_gr_pack");
    return PRODM_OK;
}

int launch_unpack_planes(const uint8_t* src, const UnpackSet& set, int word_bytes, void** table, cudaStream_t st) {
    if (set.n <= 0) return PRODM_OK;
    uint64_t most = 0;
    for (int p = 0; p < set.n; p++) most = set.words[p] > most ? set.words[p] : most;
    dim3 grid(grid_for(most, 256, 4), set.n);
    if (word_bytes == 4) k_unpack_planes<uint32_t><<<grid, 256, 0, st>>>(src, set, table);
    else k_unpack_planes<uint64_t><<<grid, 256, 0, st>>>(src, set, table);
    PRODM_CHECK_LAUNCH("k_unpack_planes");
    return PRODM_OK;
}

template <class T>
int launch_maxabs(const T* x, uint64_t n, void* maxkey, cudaStream_t st) {
    k_maxabs<T><<<grid_for(n, 256, 8), 256, 0, st>>>(x, n, (typename KeyOf<T>::type*)maxkey);
    PRODM_CHECK_LAUNCH("k_maxabs");
    return PRODM_OK;
}

template <class T>
int launch_bounds_from_keys(const void* keys, int nl, int negabinary, T* bounds, cudaStream_t st) {
    count_launch();
    const cudaError_t e = launch_chain(true, k_bounds<T>, dim3(1), dim3(32), 0, st,
                                       (const typename KeyOf<T>::type*)keys, nl, negabinary, bounds);
    if (e != cudaSuccess) return cuda_status(e, "k_bounds");
    return PRODM_OK;
}

int launch_fill_u32(uint32_t* dst, uint64_t n, uint32_t v, cudaStream_t st) {
    k_fill_u32<<<grid_for(n, 256, 4), 256, 0, st>>>(dst, n, v);
    PRODM_CHECK_LAUNCH("k_fill_u32");
    return PRODM_OK;
}

template int launch_maxabs<float>(const float*, uint64_t, void*, cudaStream_t);
template int launch_maxabs<double>(const double*, uint64_t, void*, cudaStream_t);
template int launch_bounds_from_keys<float>(const void*, int, int, float*, cudaStream_t);
template int launch_bounds_from_keys<double>(const void*, int, int, double*, cudaStream_t);

}  // namespace prodm
