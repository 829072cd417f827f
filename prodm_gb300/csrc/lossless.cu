// Lossless stage on the device (sm_103a): the ZCB codec (zero-compacted
// bytes; this project's format, not zstd) and AdaptiveLevelCompressor's
// stopping rule (AdaptiveLevelCompressor.hpp:13-40).
//
// A stream compresses as 4096-byte chunks of 32-bit words (the last word
// zero-padded), each independent of the others:
//   u64 raw length | u32 chunk count C | u32 end offset of each chunk's data
//   (relative to the end of this table) | chunk data
// chunk data: 32 u32 word masks (bit k of mask m: word 32m+k nonzero), a
// 4-bit byte mask per nonzero word (8 per u32, in word order, padded to a
// u32), the nonzero bytes in order (padded to 4 bytes). The raw length comes
// first as in the reference's zstd wrapper (ZSTD.hpp:9-20). One warp per
// chunk in all three passes: count (sizes, for the stopping rule and the
// retrieval cost model), write, read.
#include <cstring>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace prodm {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int ZW = 8;   // warps per CTA

__device__ __forceinline__ int zseg(const ZStream* s, int ns, uint64_t g) { return find_seg(s, ns, g, &ZStream::chunk0); }

// word w of chunk c (4 bytes, zero beyond the stream's end)
__device__ __forceinline__ uint32_t zword(const uint8_t* __restrict__ src, uint64_t len, uint64_t b) {
    if (b + 4 <= len && ((uintptr_t)(src + b) & 3) == 0) return __ldcs((const uint32_t*)(src + b));
    uint32_t w = 0;
    for (int k = 0; k < 4; k++)
        if (b + k < len) w |= (uint32_t)src[b + k] << (8 * k);
    return w;
}

__device__ __forceinline__ uint32_t nib_of(uint32_t w) {
    return (w & 0xffu ? 1u : 0u) | (w & 0xff00u ? 2u : 0u) | (w & 0xff0000u ? 4u : 0u) | (w & 0xff000000u ? 8u : 0u);
}

// nonzero bytes of the lanes before this one, and of all lanes
__device__ __forceinline__ uint32_t nib_before(uint32_t nb, uint32_t lt, uint32_t& all) {
    const uint32_t c = __popc(nb);   // 0 .. 4
    const uint32_t b0 = __ballot_sync(FULL, c & 1u), b1 = __ballot_sync(FULL, c & 2u), b2 = __ballot_sync(FULL, c & 4u);
    all = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
    return __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
}

__device__ __forceinline__ uint32_t chunk_bytes(uint32_t nzw, uint32_t nzb) {
    return 128 + 4 * ((nzw + 7) / 8) + 4 * ((nzb + 3) / 4);
}

// One warp per chunk. Every kernel has a chunk's loads in flight before it
// uses them (eight words a lane here and in the writer, the chunk's data
// staged in shared memory in the reader): waiting for each word before the
// next, the finest level of a 257^3 fp32 field took 43 us to count, 68 us to
// write and 41 us to read, against 23, 56 and 26 us.
__global__ void __launch_bounds__(32 * ZW) k_zcb_count(const ZStream* __restrict__ ss, int ns, uint64_t total,
                                                       uint32_t* __restrict__ csize) {
    const int lane = threadIdx.x & 31;
    for (uint64_t g = (uint64_t)blockIdx.x * ZW + (threadIdx.x >> 5); g < total; g += (uint64_t)gridDim.x * ZW) {
        const ZStream s = ss[zseg(ss, ns, g)];
        const uint64_t base = (g - s.chunk0) * 4096;
        uint32_t nzw = 0, nzb = 0;   // the lane's own, in any order
        auto add = [&](uint32_t w) {
            nzw += w != 0;
            nzb += __popc(nib_of(w));
        };
        if (base + 4096 <= s.len && ((uintptr_t)s.src & 15) == 0) {
            const uint4* p = reinterpret_cast<const uint4*>(s.src + base);
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = __ldcs(p + 32 * i + lane);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                add(v[i].x);
                add(v[i].y);
                add(v[i].z);
                add(v[i].w);
            }
        } else {
#pragma unroll 8
            for (int i = 0; i < 32; i++) add(zword(s.src, s.len, base + 4 * (32 * i + lane)));
        }
        nzw = __reduce_add_sync(FULL, nzw);
        nzb = __reduce_add_sync(FULL, nzb);
        if (lane == 0) csize[g] = chunk_bytes(nzw, nzb);
    }
}

// per stream: chunk data offsets (exclusive scan) and the compressed size
__global__ void k_zcb_scan(const ZStream* __restrict__ ss, const uint32_t* __restrict__ csize,
                           uint32_t* __restrict__ coff, uint32_t* __restrict__ out_size) {
    const ZStream s = ss[blockIdx.x];
    const int lane = threadIdx.x;
    const uint64_t nch = (s.len + 4095) / 4096;
    uint32_t run = 0;
    for (uint64_t c0 = 0; c0 < nch; c0 += 32) {
        const uint64_t c = c0 + lane;
        const uint32_t v = c < nch ? csize[s.chunk0 + c] : 0u;
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += t;
        }
        if (c < nch) coff[s.chunk0 + c] = run + inc - v;
        run += __shfl_sync(FULL, inc, 31);
    }
    if (lane == 0) {
        out_size[blockIdx.x] = (uint32_t)(12 + 4 * nch + run);
        if (nch == 0 && s.dst) {   // an empty stream is its header (the writer works by chunks)
            uint32_t* out = (uint32_t*)s.dst;
            out[0] = out[1] = out[2] = 0;
        }
    }
}

// dst of each stream: 4-byte aligned, its compressed size long
__global__ void __launch_bounds__(32 * ZW) k_zcb_write(const ZStream* __restrict__ ss, int ns, uint64_t total,
                                                       const uint32_t* __restrict__ csize,
                                                       const uint32_t* __restrict__ coff) {
    __shared__ uint32_t nibs[ZW][128];
    __shared__ uint32_t bytes[ZW][1024];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    uint8_t* bb = (uint8_t*)bytes[wp];
    for (uint64_t g = (uint64_t)blockIdx.x * ZW + wp; g < total; g += (uint64_t)gridDim.x * ZW) {
        const ZStream s = ss[zseg(ss, ns, g)];
        const uint64_t c = g - s.chunk0, nch = (s.len + 4095) / 4096;
        const uint64_t base = c * 4096;
        uint32_t* out = (uint32_t*)s.dst;
        if (c == 0 && lane == 0) {
            out[0] = (uint32_t)s.len;
            out[1] = (uint32_t)(s.len >> 32);
            out[2] = (uint32_t)nch;
        }
        for (int k = lane; k < 128; k += 32) nibs[wp][k] = 0;
        __syncwarp();
        uint32_t nzw = 0, nzb = 0, mymask = 0;
        const bool whole = base + 4096 <= s.len && ((uintptr_t)s.src & 3) == 0;
        for (int i0 = 0; i0 < 32; i0 += 8) {
            uint32_t v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint64_t at = base + 4 * (32 * (i0 + u) + lane);
                v[u] = whole ? __ldcs((const uint32_t*)(s.src + at)) : zword(s.src, s.len, at);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t w = v[u], m = __ballot_sync(FULL, w != 0);
                if (lane == i0 + u) mymask = m;
                const uint32_t nb = nib_of(w);
                uint32_t all;
                const uint32_t before = nib_before(nb, lt, all);
                if (w) {
                    const uint32_t ord = nzw + __popc(m & lt);
                    atomicOr(&nibs[wp][ord >> 3], nb << (4 * (ord & 7)));
                    uint32_t at = nzb + before;
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((nb >> k) & 1u) bb[at++] = (uint8_t)(w >> (8 * k));
                }
                nzw += __popc(m);
                nzb += all;
            }
        }
        if (lane == 0)
            for (uint32_t k = nzb; k & 3; k++) bb[k] = 0;
        __syncwarp();
        uint32_t* d = out + 3 + nch + coff[g] / 4;
        d[lane] = mymask;
        const uint32_t nn = (nzw + 7) / 8, nbw = (nzb + 3) / 4;
        for (uint32_t k = lane; k < nn; k += 32) d[32 + k] = nibs[wp][k];
        for (uint32_t k = lane; k < nbw; k += 32) d[32 + nn + k] = bytes[wp][k];
        if (lane == 0) out[3 + c] = coff[g] + csize[g];
        __syncwarp();
    }
}

// src of each stream: its compressed bytes, 4-byte aligned, `clen` long
// (headers checked on the host); dst: the raw bytes. A chunk whose offsets
// or counts do not fit its data records PRODM_ECORRUPT and is skipped.
__global__ void __launch_bounds__(32 * ZW) k_zcb_read(const ZStream* __restrict__ ss, int ns, uint64_t total,
                                                      int* __restrict__ status) {
    __shared__ uint32_t data[ZW][1152];
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    for (uint64_t g = (uint64_t)blockIdx.x * ZW + (threadIdx.x >> 5); g < total; g += (uint64_t)gridDim.x * ZW) {
        const ZStream s = ss[zseg(ss, ns, g)];
        const uint64_t c = g - s.chunk0, nch = (s.len + 4095) / 4096;
        const uint32_t* in = (const uint32_t*)s.src;
        const uint64_t dlen = s.clen - 12 - 4 * nch;          // data area bytes
        const uint32_t start = c ? in[3 + c - 1] : 0u, end = in[3 + c];
        if (end < start + 128 || end > dlen || (start & 3) || (end & 3)) {
            if (lane == 0) atomicCAS(status, 0, PRODM_ECORRUPT);
            continue;
        }
        const uint32_t* d = in + 3 + nch + start / 4;
        const uint32_t clen = end - start;
        const uint32_t mymask = d[lane];
        const uint32_t nzw_all = __reduce_add_sync(FULL, __popc(mymask));
        const uint32_t nn = (nzw_all + 7) / 8;
        if (128 + 4 * nn > clen) {
            if (lane == 0) atomicCAS(status, 0, PRODM_ECORRUPT);
            continue;
        }
        // the chunk's nibbles and bytes (at most 512 + 4096) into shared memory
        const uint32_t words = min(clen / 4 - 32, 1152u);
        uint32_t* st = data[threadIdx.x >> 5];
        __syncwarp();
#pragma unroll 4
        for (uint32_t k = lane; k < words; k += 32) st[k] = __ldcs(d + 32 + k);
        __syncwarp();
        const uint8_t* by = (const uint8_t*)(st + nn);
        const uint32_t blen = min(clen - 128 - 4 * nn, 4 * (words - min(words, nn)));
        uint32_t nzw = 0, nzb = 0;
        bool bad = false;
        const uint64_t base = c * 4096;
        const bool whole = base + 4096 <= s.len && ((uintptr_t)s.dst & 3) == 0;
#pragma unroll 4
        for (int i = 0; i < 32; i++) {
            const uint32_t m = __shfl_sync(FULL, mymask, i);
            uint32_t nb = 0;
            if ((m >> lane) & 1u) {
                const uint32_t ord = nzw + __popc(m & lt);
                nb = (st[ord >> 3] >> (4 * (ord & 7))) & 15u;
            }
            uint32_t all;
            uint32_t at = nzb + nib_before(nb, lt, all), w = 0;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((nb >> k) & 1u) {
                    if (at < blen) w |= (uint32_t)by[at] << (8 * k);
                    else bad = true;
                    at++;
                }
            const uint64_t b = base + 4 * (32 * i + lane);
            if (whole || (b + 4 <= s.len && ((uintptr_t)(s.dst + b) & 3) == 0)) {
                *(uint32_t*)(s.dst + b) = w;
            } else {
                for (int k = 0; k < 4; k++)
                    if (b + k < s.len) s.dst[b + k] = (uint8_t)(w >> (8 * k));
            }
            nzw += __popc(m);
            nzb += all;
        }
        if (__any_sync(FULL, bad) && lane == 0) atomicCAS(status, 0, PRODM_ECORRUPT);
    }
}

// plain copies: stream i's len bytes from src to dst, any alignment
// (blockIdx.y = stream)
__global__ void __launch_bounds__(256) k_ll_copy(const ZStream* __restrict__ ss) {
    const ZStream s = ss[blockIdx.y];
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, ts = (uint64_t)gridDim.x * blockDim.x;
    const uintptr_t both = (uintptr_t)s.src | (uintptr_t)s.dst;
    uint64_t done = 0;
    if ((both & 15) == 0) {
        const uint64_t n = s.len / 16;
        for (uint64_t i = t0; i < n; i += ts) ((uint4*)s.dst)[i] = __ldcs((const uint4*)s.src + i);
        done = n * 16;
    } else if ((both & 3) == 0) {
        const uint64_t n = s.len / 4;
        for (uint64_t i = t0; i < n; i += ts) ((uint32_t*)s.dst)[i] = __ldcs((const uint32_t*)s.src + i);
        done = n * 4;
    }
    for (uint64_t i = done + t0; i < s.len; i += ts) s.dst[i] = s.src[i];
}
// the first 12 bytes of compressed streams (raw length, chunk count)
__global__ void k_zcb_headers(const ZStream* __restrict__ ss, int ns, uint8_t* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 12 * ns; i += gridDim.x * blockDim.x)
        out[i] = ss[i / 12].src[i % 12];
}

unsigned zgrid(uint64_t chunks) {
    uint64_t g = (chunks + ZW - 1) / ZW;
    const uint64_t cap = (uint64_t)device_sms() * 8;
    return (unsigned)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

uint64_t zcb_bound(uint64_t len) {
    const uint64_t nch = (len + 4095) / 4096;
    return 12 + 4 * nch + nch * (128 + 512) + 4 * ((len + 3) / 4);
}

int launch_zcb_count(const ZStream* d_ss, int ns, uint64_t total_chunks, uint32_t* csize, uint32_t* coff,
                     uint32_t* out_sizes, cudaStream_t st) {
    if (total_chunks) {
        k_zcb_count<<<zgrid(total_chunks), 32 * ZW, 0, st>>>(d_ss, ns, total_chunks, csize);
        PRODM_CHECK_LAUNCH("k_zcb_count");
    }
    k_zcb_scan<<<ns, 32, 0, st>>>(d_ss, csize, coff, out_sizes);
    PRODM_CHECK_LAUNCH("k_zcb_scan");
    return PRODM_OK;
}

int launch_zcb_write(const ZStream* d_ss, int ns, uint64_t total_chunks, const uint32_t* csize, const uint32_t* coff,
                     cudaStream_t st) {
    if (!total_chunks) return PRODM_OK;
    k_zcb_write<<<zgrid(total_chunks), 32 * ZW, 0, st>>>(d_ss, ns, total_chunks, csize, coff);
    PRODM_CHECK_LAUNCH("k_zcb_write");
    return PRODM_OK;
}

int launch_zcb_read(const ZStream* d_ss, int ns, uint64_t total_chunks, int* status, cudaStream_t st) {
    if (!total_chunks) return PRODM_OK;
    k_zcb_read<<<zgrid(total_chunks), 32 * ZW, 0, st>>>(d_ss, ns, total_chunks, status);
    PRODM_CHECK_LAUNCH("k_zcb_read");
    return PRODM_OK;
}

// AdaptiveLevelCompressor::compress_level's rule on the given sizes
int adaptive_stopping(const uint32_t* raw, const uint32_t* comp, int B, int latter, uint8_t* compressed) {
    int stopping = B;
    for (int p = 0; p < B; p++) compressed[p] = 0;
    for (int i = 0; i < B; i++) {
        const float ratio = (float)(raw[i] * 1.0 / comp[i]);
        compressed[i] = 1;
        if (i && ratio < 1.05) {
            stopping = i;
            break;
        }
    }
    const int start = stopping < latter ? latter : stopping + 1;
    for (int i = start; i < B; i++) compressed[i] = 1;
    return stopping;
}

}  // namespace prodm

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------
namespace prodm {

namespace {
uint64_t align256(uint64_t x) { return (x + 255) / 256 * 256; }

// descriptors on the device with per-chunk scratch and `extra` bytes
struct ZJob {
    Scratch mem;
    const ZStream* ss = nullptr;
    uint32_t* csize = nullptr;
    uint32_t* coff = nullptr;
    uint32_t* outsz = nullptr;
    int* status = nullptr;
    uint8_t* extra = nullptr;
    uint64_t chunks = 0;
    cudaStream_t st;
    bool copying = false;
    explicit ZJob(cudaStream_t s) : mem(s), st(s) {}
    ~ZJob() {
        if (copying) cudaStreamSynchronize(st);
    }
    // room for n streams of `chunks` chunks in all
    int reserve(size_t n, uint64_t nchunks, uint64_t extra_bytes) {
        chunks = nchunks;
        const uint64_t a = align256(n * sizeof(ZStream)), b = align256(chunks * 4 + 4), c = align256(n * 4 + 4);
        PRODM_CUDA(mem.alloc(a + 2 * b + c + 256 + extra_bytes));
        uint8_t* base = mem.get();
        ss = (const ZStream*)base;
        csize = (uint32_t*)(base + a);
        coff = (uint32_t*)(base + a + b);
        outsz = (uint32_t*)(base + a + 2 * b);
        status = (int*)(base + a + 2 * b + c);
        extra = base + a + 2 * b + c + 256;
        return PRODM_OK;
    }
    // the descriptors by value (the call may end before they are used), or for a
    // call that ends in wait() by a copy, which `h` has to outlive this job for
    int put(const std::vector<ZStream>& h) { return launch_put(mem.get(), h.data(), h.size() * sizeof(ZStream), st); }
    int upload(const std::vector<ZStream>& h) {
        copying = true;
        PRODM_CUDA(cudaMemcpyAsync(mem.get(), h.data(), h.size() * sizeof(ZStream), cudaMemcpyHostToDevice, st));
        return PRODM_OK;
    }
    int wait() {
        PRODM_CUDA(cudaStreamSynchronize(st));
        copying = false;
        return PRODM_OK;
    }
};
// the streams' first chunks in the flattened index; returns all chunks
uint64_t number_chunks(std::vector<ZStream>& ss, size_t n) {
    uint64_t c = 0;
    for (size_t i = 0; i < n; i++) {
        ss[i].chunk0 = c;
        c += (ss[i].len + 4095) / 4096;
    }
    return c;
}
int launch_copies(const ZStream* d, const ZStream* h, size_t n, cudaStream_t st) {
    uint64_t most = 0;
    for (size_t i = 0; i < n; i++) most = h[i].len > most ? h[i].len : most;
    for (size_t at = 0; at < n; at += 32768) {   // (a grid's y extent)
        const unsigned ny = (unsigned)(n - at < 32768 ? n - at : 32768);
        k_ll_copy<<<dim3(grid_for(most / 16 + 1, 256, n > 16 ? 1 : 4), ny), 256, 0, st>>>(d + at);
        PRODM_CHECK_LAUNCH("k_ll_copy");
    }
    return PRODM_OK;
}
}  // namespace

// One call takes all the streams there are (every level of a handle): one
// upload of descriptors and one launch per pass, where a level at a time
// synchronised three times and a plane at a time copied once or twice
// (257^3 fp32 files through the stage: 7.8 ms a pass of which the kernels
// took 0.9; 1.05 ms now).
int ll_sizes(const std::vector<LlPart>& parts, uint32_t* h_comp, cudaStream_t st) {
    std::vector<ZStream> ss;
    for (const LlPart& p : parts) ss.push_back(ZStream{p.src, nullptr, p.raw, 0, 0});
    if (ss.empty()) return PRODM_OK;
    ZJob j(st);
    int rc = j.reserve(ss.size(), number_chunks(ss, ss.size()), 0);
    if (rc || (rc = j.upload(ss))) return rc;
    if ((rc = launch_zcb_count(j.ss, (int)ss.size(), j.chunks, j.csize, j.coff, j.outsz, st))) return rc;
    PRODM_CUDA(cudaMemcpyAsync(h_comp, j.outsz, ss.size() * 4, cudaMemcpyDeviceToHost, st));
    return j.wait();
}

int ll_store(const std::vector<LlPart>& parts, cudaStream_t st) {
    // compressed streams first; those whose place is not 4-byte aligned go
    // through scratch; then the copies
    std::vector<ZStream> ss, copies;
    std::vector<uint64_t> at;   // scratch offset of a stream, or ~0
    uint64_t scr = 0;
    for (const LlPart& p : parts) {
        if (!p.packed) {
            if (p.raw) copies.push_back(ZStream{p.src, p.dst, p.raw, 0, 0});
            continue;
        }
        ss.push_back(ZStream{p.src, p.dst, p.raw, p.stored, 0});
        const bool direct = (uintptr_t)p.dst % 4 == 0;
        at.push_back(direct ? ~0ull : scr);
        if (!direct) scr += align256(p.stored);
    }
    const size_t nz = ss.size();
    const uint64_t chunks = number_chunks(ss, nz);
    size_t ncopy = copies.size();
    for (uint64_t a : at) ncopy += a != ~0ull;
    if (nz + ncopy == 0) return PRODM_OK;
    ZJob j(st);
    int rc = j.reserve(nz + ncopy, chunks, scr);
    if (rc) return rc;
    for (size_t i = 0; i < nz; i++)
        if (at[i] != ~0ull) {
            copies.push_back(ZStream{j.extra + at[i], ss[i].dst, ss[i].clen, 0, 0});
            ss[i].dst = j.extra + at[i];
        }
    ss.insert(ss.end(), copies.begin(), copies.end());
    if ((rc = j.put(ss))) return rc;
    if (nz) {
        if ((rc = launch_zcb_count(j.ss, (int)nz, chunks, j.csize, j.coff, j.outsz, st))) return rc;
        if ((rc = launch_zcb_write(j.ss, (int)nz, chunks, j.csize, j.coff, st))) return rc;
    }
    return ncopy ? launch_copies(j.ss + nz, ss.data() + nz, ncopy, st) : PRODM_OK;
}

int ll_raw_sizes(std::vector<LlPart>& parts, cudaStream_t st) {
    std::vector<ZStream> ss;
    for (const LlPart& p : parts)
        if (p.packed) {
            if (p.stored < 12) return fail(PRODM_ECORRUPT, "lossless: compressed stream shorter than its header");
            ss.push_back(ZStream{p.src, nullptr, 0, p.stored, 0});
        }
    std::vector<uint8_t> hdr(12 * ss.size());
    if (!ss.empty()) {
        ZJob j(st);
        int rc = j.reserve(ss.size(), 0, hdr.size());
        if (rc || (rc = j.upload(ss))) return rc;
        k_zcb_headers<<<grid_for(hdr.size(), 256), 256, 0, st>>>(j.ss, (int)ss.size(), j.extra);
        PRODM_CHECK_LAUNCH("k_zcb_headers");
        PRODM_CUDA(cudaMemcpyAsync(hdr.data(), j.extra, hdr.size(), cudaMemcpyDeviceToHost, st));
        if ((rc = j.wait())) return rc;
    }
    size_t k = 0;
    for (LlPart& p : parts) {
        if (!p.packed) {
            p.raw = p.stored;
            continue;
        }
        uint64_t len;
        uint32_t nch;
        std::memcpy(&len, hdr.data() + 12 * k, 8);
        std::memcpy(&nch, hdr.data() + 12 * k + 8, 4);
        k++;
        if (len > 0xffffffffull || nch != (len + 4095) / 4096 || p.stored < 12 + 4 * (uint64_t)nch)
            return fail(PRODM_ECORRUPT, "lossless: malformed compressed stream header");
        p.raw = len;
    }
    return PRODM_OK;
}

int ll_expand(const std::vector<LlPart>& parts, cudaStream_t st) {
    // copies first: the uncompressed streams, and compressed ones that are not
    // 4-byte aligned into scratch
    std::vector<ZStream> ss, copies;
    std::vector<uint64_t> at;
    uint64_t scr = 0;
    for (const LlPart& p : parts) {
        if (!p.packed) {
            if (p.raw) copies.push_back(ZStream{p.src, p.dst, p.raw, 0, 0});
            continue;
        }
        ss.push_back(ZStream{p.src, p.dst, p.raw, p.stored, 0});
        const bool direct = (uintptr_t)p.src % 4 == 0;
        at.push_back(direct ? ~0ull : scr);
        if (!direct) scr += align256(p.stored);
    }
    const size_t nz = ss.size();
    const uint64_t chunks = number_chunks(ss, nz);
    size_t ncopy = copies.size();
    for (uint64_t a : at) ncopy += a != ~0ull;
    if (nz + ncopy == 0) return PRODM_OK;
    ZJob j(st);
    int rc = j.reserve(nz + ncopy, 0, scr);
    if (rc) return rc;
    for (size_t i = 0; i < nz; i++)
        if (at[i] != ~0ull) {
            copies.push_back(ZStream{ss[i].src, j.extra + at[i], ss[i].clen, 0, 0});
            ss[i].src = j.extra + at[i];
        }
    ss.insert(ss.end(), copies.begin(), copies.end());
    if ((rc = j.upload(ss))) return rc;
    if (ncopy && (rc = launch_copies(j.ss + nz, ss.data() + nz, ncopy, st))) return rc;
    if (!nz) return j.wait();
    PRODM_CUDA(cudaMemsetAsync(j.status, 0, 4, st));
    if ((rc = launch_zcb_read(j.ss, (int)nz, chunks, j.status, st))) return rc;
    int hstat = 0;
    PRODM_CUDA(cudaMemcpyAsync(&hstat, j.status, 4, cudaMemcpyDeviceToHost, st));
    if ((rc = j.wait())) return rc;
    if (hstat) return fail(PRODM_ECORRUPT, "lossless: malformed compressed chunk");
    return PRODM_OK;
}

// one level's streams (device, concatenated, raw sizes h_sizes) -> stored
// streams (compressed where the rule says, else raw) concatenated into d_out
static int ll_compress_level(const uint8_t* d_raw, const uint32_t* h_sizes, int B, int latter, uint8_t* d_out,
                             uint64_t cap, uint32_t* h_out_sizes, int* h_stop, cudaStream_t st) {
    std::vector<LlPart> parts(B);
    uint64_t o = 0, total = 0;
    for (int p = 0; p < B; p++) {
        parts[p] = LlPart{d_raw + o, nullptr, h_sizes[p], 0, true};
        o += h_sizes[p];
    }
    std::vector<uint32_t> comp(B);
    int rc = ll_sizes(parts, comp.data(), st);
    if (rc) return rc;
    std::vector<uint8_t> flags(B);
    *h_stop = adaptive_stopping(h_sizes, comp.data(), B, latter, flags.data());
    for (int p = 0; p < B; p++) {
        parts[p].packed = flags[p] != 0;
        parts[p].stored = flags[p] ? comp[p] : h_sizes[p];
        parts[p].dst = d_out + total;
        h_out_sizes[p] = (uint32_t)parts[p].stored;
        total += parts[p].stored;
    }
    if (total > cap) return fail(PRODM_EINVAL, "lossless: output capacity below the level's stored size");
    if ((rc = ll_store(parts, st))) return rc;
    PRODM_CUDA(cudaStreamSynchronize(st));
    return PRODM_OK;
}

// stored streams of `num` planes (sizes h_sizes, flags) -> raw streams
// concatenated into d_out (capacity cap); h_raw_sizes: their raw sizes
static int ll_decompress_planes(const uint8_t* d_in, const uint32_t* h_sizes, const uint8_t* h_flags, int num,
                                uint8_t* d_out, uint64_t cap, uint32_t* h_raw_sizes, cudaStream_t st) {
    std::vector<LlPart> parts(num);
    uint64_t o = 0, r = 0;
    for (int i = 0; i < num; i++) {
        parts[i] = LlPart{d_in + o, nullptr, 0, h_sizes[i], h_flags[i] != 0};
        o += h_sizes[i];
    }
    int rc = ll_raw_sizes(parts, st);
    if (rc) return rc;
    for (int i = 0; i < num; i++) {
        if (r + parts[i].raw > cap) return fail(PRODM_EINVAL, "lossless: output capacity below the raw size");
        parts[i].dst = d_out + r;
        h_raw_sizes[i] = (uint32_t)parts[i].raw;
        r += parts[i].raw;
    }
    return ll_expand(parts, st);
}

}  // namespace prodm

using namespace prodm;

extern "C" {

int prodm_lossless_compress_bound(const uint32_t* h_sizes, int num_bitplanes, uint64_t* out) {
    if (!h_sizes || !out || num_bitplanes < 1 || num_bitplanes > 64) return fail(PRODM_EINVAL, "bad arguments");
    uint64_t t = 0;
    for (int p = 0; p < num_bitplanes; p++) t += zcb_bound(h_sizes[p]) > h_sizes[p] ? zcb_bound(h_sizes[p]) : h_sizes[p];
    *out = t;
    return PRODM_OK;
}

int prodm_lossless_compress_level(const void* d_blob, const uint32_t* h_sizes, int num_bitplanes, int latter_index,
                                  void* d_out, uint64_t capacity, uint32_t* h_out_sizes, int* h_stopping_index,
                                  void* stream) {
    if (!d_blob || !h_sizes || !d_out || !h_out_sizes || !h_stopping_index || num_bitplanes < 1 || num_bitplanes > 64 ||
        latter_index < 0)
        return fail(PRODM_EINVAL, "prodm_lossless_compress_level: bad arguments");
    return ll_compress_level((const uint8_t*)d_blob, h_sizes, num_bitplanes, latter_index, (uint8_t*)d_out, capacity,
                             h_out_sizes, h_stopping_index, (cudaStream_t)stream);
}

int prodm_lossless_decompress_level(const void* d_blob, const uint32_t* h_sizes, int starting_bitplane,
                                    int num_bitplanes, int stopping_index, int latter_index, void* d_out,
                                    uint64_t capacity, uint32_t* h_raw_sizes, void* stream) {
    if ((num_bitplanes > 0 && (!d_blob || !h_sizes || !d_out || !h_raw_sizes)) || starting_bitplane < 0 ||
        num_bitplanes < 0 || starting_bitplane + num_bitplanes > 64)
        return fail(PRODM_EINVAL, "prodm_lossless_decompress_level: bad arguments");
    std::vector<uint8_t> flags(num_bitplanes);
    for (int i = 0; i < num_bitplanes; i++) {   // AdaptiveLevelCompressor.hpp:43-52
        const int p = starting_bitplane + i;
        flags[i] = (p <= stopping_index || p >= latter_index) ? 1 : 0;
    }
    return ll_decompress_planes((const uint8_t*)d_blob, h_sizes, flags.data(), num_bitplanes, (uint8_t*)d_out,
                                capacity, h_raw_sizes, (cudaStream_t)stream);
}

}  // extern "C"
