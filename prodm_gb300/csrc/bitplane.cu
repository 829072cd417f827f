// Bitplane encoders / decoders and error collectors (sm_103a).
//
// Stream layout on the device ("aligned layout"): the words of plane p of a
// level start at plane[p] (word aligned). NegaBinary planes all hold
// ceil(n / block) words; grouped planes hold between 0 and 2 * nblocks words.
// The grouped encoder's per-block recording bitplanes (the u8 header of
// stream 0, GroupedBPEncoder.hpp:66-71) are kept in a separate rb array.
// pack.cu turns this into the reference level-file byte layout.
//
// Warp mapping: one warp per block of 32 (fp32, u32 words) or 64 (fp64, u64
// words: each lane holds elements lane and lane + 32) values; __ballot_sync
// transposes one bitplane of the block into one stream word; lane p then
// owns the word of plane p (and p + 32 for fp64).
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "errtab.cuh"
#include "kernels.cuh"
#include "nbcodec.cuh"

namespace prodm {

namespace {

constexpr unsigned FULL = 0xffffffffu;

template <class T>
__device__ __forceinline__ int level_exp(const typename KeyOf<T>::type* maxkey, int exp_arg) {
    return maxkey ? frexp_exp(key_to_val(*maxkey, T())) : exp_arg;
}

// quantisation shared by the encoders
__device__ __forceinline__ int64_t trunc_fps(double v) { return (int64_t)v; }

// ---------------------------------------------------------------------------
// per-thread error accumulators -> per-CTA partial tables (B+1 doubles each):
// a fixed butterfly per warp, then the warps' totals in warp order, so a
// table does not depend on scheduling
// ---------------------------------------------------------------------------
template <int NACC, class A>
__device__ void flush_errors(A (&acc)[NACC], int B, double* partial) {
    __shared__ double red[8][NACC];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NACC; k++) {
        double v = (double)acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    for (int k = threadIdx.x; k <= B && k < NACC; k += blockDim.x) {
        double v = 0;
        for (int w = 0; w < nw; w++) v += red[w][k];
        partial[(size_t)blockIdx.x * (B + 1) + k] = v;
    }
}

// NegaBinaryBPEncoder::collect_level_errors (NegaBinaryBPEncoder.hpp:231-239)
// in shifted units: acc[B] += m^2, acc[B-k] += (nb2bin(nb & (2^k-1)) + m)^2,
// acc[0] += shifted^2.
template <int NACC>
__device__ __forceinline__ void nb_errors(double (&acc)[NACC], uint64_t nb, double shifted, double m, int B) {
    acc[B < NACC ? B : NACC - 1] += m * m;
#pragma unroll
    for (int k = 1; k < NACC - 1; k++) {
        if (k < B) {
            double d = (double)nb_to_bin((uint64_t)(nb & ((1ull << k) - 1ull))) + m;
            acc[B - k] += d * d;
        }
    }
    acc[0] += shifted * shifted;
}
// GroupedBPEncoder::collect_level_errors (GroupedBPEncoder.hpp:324-335), a = |shifted|
template <int NACC>
__device__ __forceinline__ void gr_errors(double (&acc)[NACC], double a, int B) {
    uint64_t fp = (uint64_t)a;
    double m = a - (double)fp;
    acc[B < NACC ? B : NACC - 1] += m * m;
#pragma unroll
    for (int k = 1; k < NACC - 1; k++) {
        if (k < B) {
            double d = (double)(fp & ((1ull << k) - 1ull)) + m;
            acc[B - k] += d * d;
        }
    }
    acc[0] += a * a;
}

// per-lane accumulators of the fp64 tables and of the squared-error collector:
// double whatever the data type (the reference sums in double)
template <class T> struct Acc { using type = double; static constexpr int N = 33; };
template <> struct Acc<double> { using type = double; static constexpr int N = 65; };

// fp32 negabinary encoder without tables
__global__ void __launch_bounds__(256, 3) k_nb_encode32(const float* __restrict__ x, uint64_t n,
                                                       const uint32_t* __restrict__ maxkey, int exp_arg, int B,
                                                       uint32_t* __restrict__ out, uint64_t stride) {
    __shared__ __align__(16) uint32_t stage[NB_STAGE];
    NbSrc q;
    q.x = x;
    q.words = out;
    q.n = n;
    q.nblocks = (n + 31) / 32;
    q.stride = stride;
    q.se = B - ((maxkey ? frexp_exp(__uint_as_float(*maxkey)) : exp_arg) + 2);   // NegaBinaryBPEncoder.hpp:21
    q.fast = pow2_normal(q.se);
    q.scale = q.fast ? pow2f(q.se) : 1.f;
    nb_encode32_chunks((q.nblocks + NB_CHUNK - 1) / NB_CHUNK, B, stage, [&](uint64_t c) {
        q.chunk = c;
        return q;
    });
}

// Every level of one fp32 field (or of many) in one launch, without tables:
// segments are the levels in chunk order.
__global__ void __launch_bounds__(256, 3) k_nb_encode32_levels(const ChunkSeg* __restrict__ segs, int nseg,
                                                               uint64_t total, int B) {
    __shared__ __align__(16) uint32_t stage[NB_STAGE];
    pdl_wait();
    pdl_release();
    int cur = -1;
    NbSrc q;
    nb_encode32_chunks(total, B, stage, [&](uint64_t c) {
        const int s = find_seg(segs, nseg, c, &ChunkSeg::chunk_begin);
        const ChunkSeg& g = segs[s];
        if (s != cur) {
            cur = s;
            q.x = g.x;
            q.words = g.words;
            q.n = g.n;
            q.nblocks = g.nblocks;
            q.stride = g.stride;
            q.se = B - (frexp_exp(__uint_as_float(*g.key)) + 2);     // NegaBinaryBPEncoder.hpp:21
            q.fast = pow2_normal(q.se);
            q.scale = q.fast ? pow2f(q.se) : 1.f;
        }
        q.chunk = c - g.chunk_begin;
        return q;
    });
}

// ---------------------------------------------------------------------------
// fp32 negabinary encoder with exact squared-error tables (errtab.cuh):
// NegaBinaryBPEncoder.hpp:65-125. Each lane takes four values per step (one
// from each of four consecutive blocks): their scaled values, negabinary
// digits and t = nb ^ 0xAAAAAAAA; the byte products of t go to the lane's
// exact sums, values below 2^23 to the warp's queue, and the four digit words
// are transposed into the plane tile (whose popcounts give the bit counts).
// ---------------------------------------------------------------------------
// plane tile of the table encoder: rows of ERR_LD words (16-byte aligned), so
// each lane stores its four transposed words of a step as one 16-byte store
// (conflict-free: rows differ by 65 16-byte units) and the chunk's plane runs
// leave with 16-byte copies
static_assert(errtab::kSlotsPad == kErrRecWords && errtab::WORDS + 16 <= errtab::kSlotsPad,
              "record width of the table encoders");
constexpr int ERR_LD = 260;
constexpr int kErrTileBytes = 32 * ERR_LD * 4;
constexpr size_t kErrSmemNB = (size_t)kErrTileBytes + 8 * sizeof(errtab::WarpQ) +
                              errtab::kSlotsPad * sizeof(unsigned long long);
// chunks a CTA encodes between two flushes of its 32-bit lane sums (each
// chunk adds at most 8 * 260100 to a lane sum)
constexpr int kErrFlushChunks = 2048;

// the 8 four-value steps of one warp over its 32 blocks; FULLW: every value
// of the blocks is inside the level (no bounds checks)
template <bool FULLB, bool FULLW>
__device__ __forceinline__ void nb_err_steps(const float* __restrict__ xw, int64_t rem, int B, int se, bool fast,
                                             float scale, uint32_t* trow, errtab::Lane& acc, errtab::WarpQ& wq,
                                             uint32_t& head, int& qn) {
    const int lane = threadIdx.x & 31;
    float vn[4];
    auto load4 = [&](int j0) {
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const int o = (j0 + g) * 32;
            vn[g] = (FULLW || o < rem) ? __ldcs(xw + o) : 0.f;
        }
    };
    load4(0);
#pragma unroll 1
    for (int j0 = 0; j0 < 32; j0 += 4) {
        float sh[4];
        if (fast) {                                                 // NegaBinaryBPEncoder.hpp:42
#pragma unroll
            for (int g = 0; g < 4; g++) sh[g] = vn[g] * scale;
        } else {
#pragma unroll
            for (int g = 0; g < 4; g++) sh[g] = ldexpf(vn[g], se);
        }
        if (j0 + 4 < 32) load4(j0 + 4);                            // next step's values in flight
        uint32_t t[4], nb[4];
        bool small[4];
#pragma unroll
        for (int g = 0; g < 4; g++) {
            const bool ok = FULLW || (j0 + g) * 32 < rem;
            const uint32_t tq = (uint32_t)(int32_t)sh[g] + 0xaaaaaaaau;   // :43-44; nb = t ^ 0xAAAAAAAA
            nb[g] = tq ^ 0xaaaaaaaau;
            t[g] = ok ? tq : 0u;                                          // padding adds nothing
            const bool big = fabsf(sh[g]) >= 8388608.f;
            acc.add_big_square(sh[g], big);                               // padding is 0: never big
            small[g] = ok && !big;
        }
        errtab::enqueue4(wq, head, qn, small, sh, lane);
        errtab::drain_full<true>(wq, head, qn, lane);
        acc.add4(t[0], t[1], t[2], t[3]);
        uint32_t w[4];
#pragma unroll
        for (int g = 0; g < 4; g++) {
            w[g] = transpose32(nb[g], lane);
            acc.pc += __popc(w[g]);
        }
        if (FULLB || lane < B) *reinterpret_cast<uint4*>(trow + j0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

template <bool FULLB>
__device__ __forceinline__ void nb_encode32_chunk_err(const float* __restrict__ x, uint64_t n, uint64_t nblocks, int B,
                                                      int se, bool fast, float scale, uint32_t* __restrict__ out,
                                                      uint64_t stride, uint64_t c, uint32_t* tile, errtab::Lane& acc,
                                                      errtab::WarpQ& wq, uint32_t& head, int& qn) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int plane = B - 1 - lane;      // lane k owns bit k = plane B-1-k
    const uint64_t cb0 = c * NB_CHUNK;
    const uint64_t v0 = (cb0 + (uint64_t)warp * 32) * 32;     // first value of the warp's 32 blocks
    const float* xw = x + v0 + lane;
    const int64_t rem = (int64_t)n - (int64_t)v0 - lane;      // this lane's values left in the level
    uint32_t* trow = tile + plane * ERR_LD + warp * 32;
    if ((int64_t)n - (int64_t)v0 >= 1024)                     // warp-uniform: all 32 blocks inside
        nb_err_steps<FULLB, true>(xw, rem, B, se, fast, scale, trow, acc, wq, head, qn);
    else
        nb_err_steps<FULLB, false>(xw, rem, B, se, fast, scale, trow, acc, wq, head, qn);
    __syncwarp();
    // the warp writes out its own 32 columns of the tile (blocks warp*32 ..
    // warp*32 + 31 of the chunk), so warps never wait for one another
    const int nvalid = (int)((nblocks - cb0) < (uint64_t)NB_CHUNK ? (nblocks - cb0) : NB_CHUNK);
    const int wb = warp * 32;
    if ((stride & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        // 16-byte runs, four planes per instruction (8 lanes per plane); words
        // past nvalid are zero (blocks past the level) and land in the plane
        // row's padding to a multiple of four words
        const int nq = (nvalid + 3) >> 2;
        const int q = lane & 7;
        const bool ok = wb / 4 + q < nq;
#pragma unroll
        for (int p0 = 0; p0 < 32; p0 += 4) {
            const int p = p0 + (lane >> 3);
            if (p0 < B) {
                const uint4 v = reinterpret_cast<const uint4*>(tile + p * ERR_LD + wb)[q];
                if (ok && p < B) reinterpret_cast<uint4*>(out + (uint64_t)p * stride + cb0 + wb)[q] = v;
            }
        }
    } else {
        const bool ok = wb + lane < nvalid;
        for (int p = 0; p < B; p++) {
            const uint32_t v = tile[p * ERR_LD + wb + lane];
            if (ok) out[(uint64_t)p * stride + cb0 + wb + lane] = v;
        }
    }
    // the warp's own barrier (id 1 + warp, 32 threads) before its columns
    // are written again; as a barrier it also keeps the compiler from
    // interleaving the next chunk's loads with this copy (which spills)
    asm volatile("bar.sync %0, 32;" ::"r"(warp + 1) : "memory");
}

// Every level (segment) of one fp32 field with tables in one launch. Records
// (errtab::kSlotsPad u64 each) sit at recs + (level * gridDim.x + CTA); a CTA
// zeroes the record of every level it enters or skips and adds its sums at
// each level change, so every record the final reduction reads is written.
__global__ void __launch_bounds__(256, 2) k_nb_encode32_err(const ChunkSeg* __restrict__ segs, ChunkSeg one,
                                                            int nseg, uint64_t total, int B, int exp_arg,
                                                            unsigned long long* __restrict__ recs) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* tile = (uint32_t*)smem;
    errtab::WarpQ* wq = (errtab::WarpQ*)(smem + kErrTileBytes);
    unsigned long long* red = (unsigned long long*)(wq + 8);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    errtab::Lane acc;
    acc.zero();
    errtab::zero_q(wq[warp], lane);
    uint32_t head = 0;
    int qn = 0;
    auto rec_of = [&](int s) { return recs + ((size_t)s * gridDim.x + blockIdx.x) * errtab::kSlotsPad; };
    auto zero_recs = [&](int s0, int s1) {   // levels [s0, s1)
        for (int s = s0; s < s1; s++)
            for (int k = threadIdx.x; k < errtab::kSlotsPad; k += blockDim.x) rec_of(s)[k] = 0;
        __syncthreads();
    };
    auto flush = [&](int s) {
        if (qn) {   // the queue's last partial batch
            __syncwarp();
            errtab::run_batch<true>(wq[warp], head, qn, lane);
            head += qn;
            qn = 0;
        }
        errtab::flush(acc, wq, red, rec_of(s));
    };
    int cur = -1, se = 0, since = 0;
    bool fast = true;
    float scale = 1.f;
    const float* qx = one.x;
    uint32_t* qw = one.words;
    uint64_t qnv = one.n, qnb = one.nblocks, qst = one.stride, qc0 = 0;
    // one flush site: at a level change, every kErrFlushChunks chunks, and at the end
    for (uint64_t c = blockIdx.x;; c += gridDim.x) {
        const bool done = c >= total;
        const int s = done ? nseg : (segs ? find_seg(segs, nseg, c, &ChunkSeg::chunk_begin) : 0);
        if (cur >= 0 && (s != cur || since == kErrFlushChunks)) {
            flush(cur);
            since = 0;
        }
        if (s != cur) {
            zero_recs(cur + 1, s < nseg ? s + 1 : nseg);
            if (done) break;
            cur = s;
            const uint32_t* key = one.key;
            if (segs) {
                qx = segs[s].x;
                qw = segs[s].words;
                qnv = segs[s].n;
                qnb = segs[s].nblocks;
                qst = segs[s].stride;
                qc0 = segs[s].chunk_begin;
                key = segs[s].key;
            }
            se = B - ((key ? frexp_exp(__uint_as_float(*key)) : exp_arg) + 2);   // NegaBinaryBPEncoder.hpp:21
            fast = pow2_normal(se);
            scale = fast ? pow2f(se) : 1.f;
        }
        since++;
        if (B == 32)
            nb_encode32_chunk_err<true>(qx, qnv, qnb, B, se, fast, scale, qw, qst, c - qc0, tile, acc, wq[warp], head,
                                        qn);
        else
            nb_encode32_chunk_err<false>(qx, qnv, qnb, B, se, fast, scale, qw, qst, c - qc0, tile, acc, wq[warp], head,
                                         qn);
    }
}

// Tables of every level from the CTA records: one CTA of 1024 threads per
// level. Thread (k, i), k < 5, sums record word i over records k, k + 5, ..
// (loads of all words in flight at once; low words of 128-bit sums also
// count their carries), then thread i combines the five partial sums in k
// order (so the doubles are summed in a fixed order) and thread i <= B
// computes entry i. keys (or exp_arg when keys is null) give the level
// exponent, exp_add the encoder's offset (2 for negabinary).
constexpr int kFinalParts = 5;
static_assert(kFinalParts * errtab::kSlotsPad <= 1024, "one thread per (part, record word)");

template <bool NB>
__global__ void __launch_bounds__(1024) k_errtab_final(const unsigned long long* __restrict__ recs, int nrec, int B,
                                                       const ChunkSeg* __restrict__ segs, ChunkSeg one, int exp_arg,
                                                       int exp_add, double* __restrict__ out) {
    __shared__ unsigned long long P[kFinalParts][errtab::kSlotsPad];    // partial sums (u64 words or double bits)
    __shared__ unsigned long long Cy[kFinalParts][errtab::kSlotsPad];   // carries out of the low words
    __shared__ unsigned long long R[errtab::kSlotsPad];
    const int l = blockIdx.x;
    const unsigned long long* rl = recs + (size_t)l * nrec * errtab::kSlotsPad;
    const int t = threadIdx.x;
    if (t < kFinalParts * errtab::kSlotsPad) {
        const int k = t / errtab::kSlotsPad, i = t - k * errtab::kSlotsPad;
        if (i < errtab::WORDS) {
            const unsigned long long* p = rl + i;
            if (errtab::slot_kind(i) == 3) {
                double v = 0;
#pragma unroll 8
                for (int r = k; r < nrec; r += kFinalParts) v += __longlong_as_double(p[(size_t)r * errtab::kSlotsPad]);
                P[k][i] = __double_as_longlong(v);
            } else {
                unsigned long long v = 0, c = 0;
#pragma unroll 8
                for (int r = k; r < nrec; r += kFinalParts) {
                    const unsigned long long o = v;
                    v += p[(size_t)r * errtab::kSlotsPad];
                    c += v < o ? 1 : 0;
                }
                P[k][i] = v;
                Cy[k][i] = c;
            }
        }
    }
    __syncthreads();
    if (t < errtab::WORDS) {
        const int kind = errtab::slot_kind(t);
        if (kind == 3) {
            double v = 0;
            for (int k = 0; k < kFinalParts; k++) v += __longlong_as_double(P[k][t]);
            R[t] = __double_as_longlong(v);
        } else if (kind != 2) {
            unsigned long long v = 0, c = 0;
            for (int k = 0; k < kFinalParts; k++) {
                const unsigned long long o = v;
                v += P[k][t];
                c += Cy[k][t] + (v < o ? 1 : 0);
            }
            R[t] = v;
            Cy[0][t] = c;   // carries into the high word (read by thread t + 1 after the barrier)
        }
    }
    __syncthreads();
    if (t < errtab::WORDS && errtab::slot_kind(t) == 2) {
        unsigned long long v = Cy[0][t - 1];
        for (int k = 0; k < kFinalParts; k++) v += P[k][t];
        R[t] = v;
    }
    __syncthreads();
    const uint32_t* key = segs ? segs[l].key : one.key;
    const uint64_t n = segs ? segs[l].n : one.n;
    const int e = (key ? frexp_exp(__uint_as_float(*key)) : exp_arg) + exp_add;
    for (int i = t; i <= B; i += blockDim.x) out[(size_t)l * (B + 1) + i] = errtab::table_entry<NB>(R, n, B, e, i);
}

// Every level of one fp32 field decoded in one launch (segments = levels in
// chunk order, kDecodeChunkBlocks 32-value blocks per chunk). Plane rows start
// on 16-byte boundaries, so a chunk's run of one plane (512 bytes) is one
// warp-wide 16-byte cp.async; the next chunk's planes are fetched into the
// second [plane][block] tile while the current chunk is decoded. Each
// 32-value block is decoded by two threads (one half transpose each), and a
// thread writes its 16 values as four 16-byte stores when the level's output
// is 16-byte aligned. NegaBinaryBPEncoder.hpp:132-192 with start plane 0 and
// num = dnum planes.
constexpr int DEC_LD = kDecodeChunkBlocks + 4;   // tile row (words): 16-byte aligned, conflict-free columns

__global__ void __launch_bounds__(256) k_nb_decode_levels(const ChunkSeg* __restrict__ segs, int nseg,
                                                         uint64_t total) {
    constexpr int CB = kDecodeChunkBlocks;
    __shared__ __align__(16) uint32_t tiles[2][32 * DEC_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();   // plane counts from the interpreter
    pdl_release();
    auto fetch = [&](uint64_t c, uint32_t* tile) {
        const ChunkSeg& q = segs[find_seg(segs, nseg, c, &ChunkSeg::chunk_begin)];
        const int num = q.dnum[0];
        const uint64_t b0 = (c - q.chunk_begin) * CB;
        const uint32_t nb = (uint32_t)min((uint64_t)CB, q.nblocks - b0);
        const uint32_t nq = (nb + 3) / 4;     // 16-byte pieces (inside the padded row)
        for (int p = warp; p < num; p += 8) {
            const uint32_t* src = q.words + (uint64_t)p * q.stride + b0;
            for (uint32_t j = lane; j < nq; j += 32) cp_async16(tile + p * DEC_LD + 4 * j, src + 4 * j);
        }
        cp_async_commit();
    };
    uint64_t c = blockIdx.x;
    if (c >= total) return;
    fetch(c, tiles[0]);
    for (int it = 0; c < total; it++, c += gridDim.x) {
        cp_async_wait_all();
        __syncthreads();
        if (c + gridDim.x < total) fetch(c + gridDim.x, tiles[(it + 1) & 1]);
        const uint32_t* tile = tiles[it & 1];
        const ChunkSeg& q = segs[find_seg(segs, nseg, c, &ChunkSeg::chunk_begin)];
        const int num = q.dnum[0];
        const uint64_t b0 = (c - q.chunk_begin) * CB;
        const uint32_t nb = (uint32_t)min((uint64_t)CB, q.nblocks - b0);
        const uint32_t t = threadIdx.x >> 1;
        const int half = threadIdx.x & 1;
        if (t < nb) {
            float vals[16];
            if (num == 0) {
#pragma unroll
                for (int v = 0; v < 16; v++) vals[v] = 0.f;
            } else {
                const int exp = frexp_exp(__uint_as_float(*q.key)) + 2;      // NegaBinaryBPEncoder.hpp:21
                const bool neg = num & 1;                                     // :153, :177
                const bool dfast = pow2_normal(exp - num);
                const float dscale = dfast ? (neg ? -pow2f(exp - num) : pow2f(exp - num)) : 1.f;
                // rows in reverse plane order: value v's digits come out most significant first
                uint32_t R[32];
#pragma unroll
                for (int p = 0; p < 32; p++) R[31 - p] = p < num ? tile[p * DEC_LD + t] : 0u;
                uint32_t a[16];
                transpose32_half(R, half, a);
#pragma unroll
                for (int v = 0; v < 16; v++) {
                    const int32_t iv = nb_to_bin(a[v] >> (32 - num));
                    vals[v] = dfast ? (float)iv * dscale
                                    : (neg ? -ldexpf((float)iv, exp - num) : ldexpf((float)iv, exp - num));
                }
            }
            const uint64_t e0 = (b0 + t) * 32 + 16 * (uint64_t)half;
            float* dst = q.y + e0;
            if (e0 + 16 <= q.n && ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0)) {
                float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
                for (int k = 0; k < 4; k++) d4[k] = make_float4(vals[4 * k], vals[4 * k + 1], vals[4 * k + 2], vals[4 * k + 3]);
            } else {
#pragma unroll
                for (int v = 0; v < 16; v++)
                    if (e0 + v < q.n) dst[v] = vals[v];
            }
        }
    }
    cp_async_wait_all();
}

// fp32 negabinary decoder, planes [s, s+num) at base[i * stride]
__global__ void __launch_bounds__(256) k_nb_decode32(const uint32_t* __restrict__ base, uint64_t stride, uint64_t n,
                                                    const uint32_t* __restrict__ maxkey, int exp_arg, int s, int num,
                                                    const uint8_t* __restrict__ dnum, float* __restrict__ out) {
    __shared__ uint32_t tile[32 * NB_TILE_LD];
    if (dnum) num = dnum[0] - s;
    const int exp = (maxkey ? frexp_exp(__uint_as_float(*maxkey)) : exp_arg) + 2;
    const int e = s + num;
    const uint64_t nblocks = (n + 31) / 32;
    const uint64_t nchunks = (nblocks + NB_CHUNK - 1) / NB_CHUNK;
    const bool dfast = pow2_normal(exp - e);
    const float dscale = dfast ? pow2f(exp - e) : 1.f;
    for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x)
        nb_decode32_chunk(base, stride, n, nblocks, num, e, exp, dfast, dscale, c, tile, out);
}

// ---------------------------------------------------------------------------
// Grouped encoder -- GroupedBPEncoder.hpp:18-73 (+ :76-145 errors)
// Chunk = 8 warps x 32 blocks per CTA.
// ---------------------------------------------------------------------------
constexpr int GR_WARPS = 8;
constexpr int GR_BPW = 32;                       // blocks per warp
constexpr int GR_CHUNK = GR_WARPS * GR_BPW;      // blocks per CTA
// The decoders and the first pass have 32 warps with 8 blocks each: a warp's
// blocks come one after the other, and 8 warps with 32 were fp32 13.2 us for 8.1
// (decode 65^3), 18.9 for 16.0 (129^3), 42.9 for 40.5 (257 x 257 x 129, 1040
// chunks); first pass 9.2 for 6.7, 9.5 for 8.2 and (257^3) 35.6 for 35.6. With
// many chunks the decoder's 8 warps, which load a group of blocks ahead, are
// faster when all planes are there (150 x 257 x 301: 51 us for 56). An fp64 warp needs twice the registers, so
// past a chunk an SM it is 8 warps there (decode 257 x 257 x 129 52.3 us for
// 56.5, first pass 257^3 39.5 for 43.8; before, 65^3 24.9 for 17.9 and 129^3 16.6
// for 9.5).
constexpr int GR_WIDE = 32;
inline bool gr_wide64(unsigned chunks) { return chunks <= (unsigned)kSMs; }
inline bool gr_wide_decode32(unsigned chunks) { return chunks <= 8u * kSMs; }

// |trunc(ldexp(v, B - exp))| and the sign (GroupedBPEncoder.hpp:41-42). For
// doubles whose scaled value is not needed (SH false: no error tables) the
// magnitude comes from the bits with integer operations (fixed_mag).
template <class T, bool SH = true>
__device__ __forceinline__ typename Traits<T>::FP gr_mag(T v, int B, int exp, bool& neg, T& shifted) {
    if constexpr (std::is_same<T, double>::value && !SH) {
        neg = below_zero(v);
        return fixed_mag(v, B - exp);
    } else {
        shifted = ldexp_t(v, B - exp);                  // :41
        int64_t fix = (int64_t)shifted;                 // :42
        neg = v < 0;
        return (typename Traits<T>::FP)(neg ? -fix : fix);
    }
}

// ldexp((T)acc, s), negated when neg (GroupedBPEncoder.hpp:359-368); for
// doubles with a normal result by integer operations (fixed_value)
template <class T>
__device__ __forceinline__ T gr_value(typename Traits<T>::FP acc, int s, bool neg) {
    if constexpr (std::is_same<T, double>::value) {
        if (fixed_value_normal(s)) {
            const long long b = __double_as_longlong(fixed_value(acc, s));
            return __longlong_as_double(neg ? b ^ (long long)0x8000000000000000ull : b);
        }
    }
    const T v = ldexp_t((T)acc, s);
    return neg ? -v : v;
}

// ---------------------------------------------------------------------------
// fp64 negabinary encoder -- NegaBinaryBPEncoder.hpp:18-62 (+ :65-125 errors)
// and decoder
// ---------------------------------------------------------------------------
// fp64 encoder with the error tables (NegaBinaryBPEncoder.hpp:65-125), a warp a
// block
__global__ void __launch_bounds__(256) k_nb_encode64_err(const double* __restrict__ x, uint64_t n,
                                                         const unsigned long long* __restrict__ maxkey, int exp_arg, int B,
                                                         uint64_t* __restrict__ out, uint64_t stride,
                                                         double* __restrict__ partial) {
    const int exp = level_exp<double>(maxkey, exp_arg) + 2;   // :21
    const int lane = threadIdx.x & 31;
    const uint64_t nblocks = (n + 63) / 64;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    double acc[Acc<double>::N];
#pragma unroll
    for (int k = 0; k < Acc<double>::N; k++) acc[k] = 0;
    for (uint64_t b = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += warps) {
        uint64_t nb[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint64_t i = b * 64 + h * 32 + lane;
            nb[h] = 0;
            if (i < n) {
                const double shifted = ldexp(x[i], B - exp);          // :42
                const int64_t q = trunc_fps(shifted);
                nb[h] = nb_from_bin(q);
                nb_errors(acc, nb[h], shifted, shifted - (double)q, B);
            }
        }
        uint64_t mine0 = 0, mine1 = 0;
        for (int p = 0; p < B; p++) {                        // encode_block :240-250
            const int k = B - 1 - p;
            const uint64_t w = (uint64_t)__ballot_sync(FULL, (nb[0] >> k) & 1u) |
                               (uint64_t)__ballot_sync(FULL, (nb[1] >> k) & 1u) << 32;
            if ((p & 31) == lane) {
                if (p < 32) mine0 = w; else mine1 = w;
            }
        }
        if (lane < B) out[(uint64_t)lane * stride + b] = mine0;
        if (lane + 32 < B) out[(uint64_t)(lane + 32) * stride + b] = mine1;
    }
    flush_errors(acc, B, partial);
}

// (int64_t)ldexp(v, k) by integer operations while |v| 2^k < 2^63
__device__ __forceinline__ int64_t nb_fix64(double v, int k) {
    const int ev = (int)(((uint64_t)__double_as_longlong(v) >> 52) & 0x7ff);
    if (ev == 0x7ff || ev - 1075 + k > 10) return trunc_fps(ldexp(v, k));
    const int64_t m = (int64_t)fixed_mag(v, k);
    return __double_as_longlong(v) < 0 ? -m : m;
}

// fp64 without tables. A warp takes eight blocks, four 32 x 32 bit transposes
// each, the second four's values on their way while the first are transposed,
// and their words leave through shared memory, eight lanes a plane: a store per
// word is one to a sector of its own, and a ballot per plane 120 of them a block.
// 513 x 513 x 257, 60 planes: 1499 us that way, 261 so (DRAM floor 164; with 32
// blocks a warp 279, and 33^3 twice as slow).
constexpr int NB64_BLOCKS = 8, NB64_LD = NB64_BLOCKS + 1;
__global__ void __launch_bounds__(256, 3) k_nb_encode64(const double* __restrict__ x, uint64_t n,
                                                        const unsigned long long* __restrict__ maxkey, int exp_arg, int B,
                                                        uint64_t* __restrict__ out, uint64_t stride) {
    constexpr int U = 4;   // blocks loaded ahead
    __shared__ uint64_t stages[8][64 * NB64_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* stage = stages[warp];
    const uint64_t nblocks = (n + 63) / 64, step = (uint64_t)gridDim.x * 8 * NB64_BLOCKS;
    pdl_wait();
    pdl_release();
    const int k = B - (level_exp<double>(maxkey, exp_arg) + 2);   // :21
    for (uint64_t b0 = ((uint64_t)blockIdx.x * 8 + warp) * NB64_BLOCKS; b0 < nblocks; b0 += step) {
        double nx[2 * U];
        auto load = [&](int j0) {
#pragma unroll
            for (int t = 0; t < 2 * U; t++) {
                const uint64_t i = (b0 + j0) * 64 + t * 32 + lane;
                nx[t] = i < n ? __ldcs(x + i) : 0.0;
            }
        };
        load(0);
#pragma unroll
        for (int j0 = 0; j0 < NB64_BLOCKS; j0 += U) {
            double v[2 * U];
#pragma unroll
            for (int t = 0; t < 2 * U; t++) v[t] = nx[t];
            if (j0 + U < NB64_BLOCKS) load(j0 + U);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint64_t m0 = nb_from_bin(nb_fix64(v[2 * u], k)), m1 = nb_from_bin(nb_fix64(v[2 * u + 1], k));
                // lane i: digit i (low halves) and 32 + i of values 0..31 and 32..63
                const uint32_t lo0 = transpose32((uint32_t)m0, lane), hi0 = transpose32((uint32_t)(m0 >> 32), lane);
                const uint32_t lo1 = transpose32((uint32_t)m1, lane), hi1 = transpose32((uint32_t)(m1 >> 32), lane);
                stage[lane * NB64_LD + j0 + u] = (uint64_t)lo1 << 32 | lo0;   // row: digit
                stage[(lane + 32) * NB64_LD + j0 + u] = (uint64_t)hi1 << 32 | hi0;
            }
        }
        __syncwarp();
        const uint64_t b = b0 + (lane & 7);
        for (int d = lane >> 3; d < B; d += 4)   // digit d is plane B - 1 - d
            if (b < nblocks) out[(uint64_t)(B - 1 - d) * stride + b] = stage[d * NB64_LD + (lane & 7)];
        __syncwarp();
    }
}

// fp64 NegaBinaryBPEncoder::progressive_decode -- :132-192. planes [s, s+num)
// with plane (s+i) at base[i * stride]; a device count (dnum[0]) overrides num.
// A warp takes eight blocks: their words of four planes come in one load and
// are turned to a plane per lane in shared memory. 513 x 513 x 257, two
// retrievals: 780 us a decode with a load per block and plane and a shuffle per
// plane, 252 so (DRAM floor, with 14 and 36 planes, about 130).
__global__ void __launch_bounds__(256, 2) k_nb_decode64(const uint64_t* __restrict__ base, uint64_t stride, uint64_t n,
                                                        const unsigned long long* __restrict__ maxkey, int exp_arg, int s,
                                                        int num, const uint8_t* __restrict__ dnum,
                                                        double* __restrict__ out) {
    __shared__ uint64_t stages[8][64 * NB64_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* stage = stages[warp];
    pdl_wait();
    pdl_release();
    if (dnum) num = dnum[0] - s;
    const int exp = level_exp<double>(maxkey, exp_arg) + 2, e = s + num;
    const uint64_t nblocks = (n + 63) / 64, step = (uint64_t)gridDim.x * 8 * NB64_BLOCKS;
    if (num == 0) {
        for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
            out[i] = 0.0;
        return;
    }
    for (uint64_t b0 = ((uint64_t)blockIdx.x * 8 + warp) * NB64_BLOCKS; b0 < nblocks; b0 += step) {
        uint64_t w[16];   // planes lane / 8 + 4 t of block lane % 8
#pragma unroll
        for (int t = 0; t < 16; t++) {
            const int p = (lane >> 3) + 4 * t;
            w[t] = p < num && b0 + (lane & 7) < nblocks ? __ldcs(base + (uint64_t)p * stride + b0 + (lane & 7)) : 0;
        }
#pragma unroll
        for (int t = 0; t < 16; t++) stage[((lane >> 3) + 4 * t) * NB64_LD + (lane & 7)] = w[t];
        __syncwarp();
#pragma unroll 2
        for (int j = 0; j < NB64_BLOCKS && b0 + j < nblocks; j++) {
            const uint64_t w0 = stage[lane * NB64_LD + j];
            const uint32_t pl0 = transpose32((uint32_t)w0, lane), ph0 = transpose32((uint32_t)(w0 >> 32), lane);
            uint32_t pl1 = 0, ph1 = 0;
            if (num > 32) {
                const uint64_t w1 = stage[(lane + 32) * NB64_LD + j];
                pl1 = transpose32((uint32_t)w1, lane);
                ph1 = transpose32((uint32_t)(w1 >> 32), lane);
            }
            const uint64_t i = (b0 + j) * 64 + lane;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                // plane p at bit 63 - p, then digit num - 1 - p
                const uint64_t a = h ? (uint64_t)__brev(ph0) << 32 | __brev(ph1) : (uint64_t)__brev(pl0) << 32 | __brev(pl1);
                const int64_t q = (int64_t)nb_to_bin(a >> (64 - num));
                const uint64_t mag = (uint64_t)(q < 0 ? -q : q);
                if (i + 32 * h < n) out[i + 32 * h] = gr_value<double>(mag, exp - e, (q < 0) != (bool)(e & 1));   // :153, :177
            }
        }
        __syncwarp();
    }
}

// word counts contributed by a block with recording plane r to plane p
__device__ __forceinline__ uint32_t gr_words(int r, int p) { return (r < p ? 1u : 0u) + (r == p ? 2u : 0u); }

// Every kernel below takes the chunks of all levels of a field in one launch
// (GrSet, one segment per level): a chain of one launch per level left a small
// level's few CTAs alone on the chip for their latency (65^3 fp32, five
// retrievals: decode 385 us in 25 launches, 91 us in 5; encode 157 and 24 us). The recording planes of a
// warp's 32 blocks are fetched by one load and the next blocks' words loaded
// a few blocks ahead, so a warp waits for memory once per group of blocks
// instead of twice per block.
template <class T>
__device__ __forceinline__ const GrSeg<T>& gr_seg(const GrSet<T>& set, uint32_t& chunk) {
    int l = 0;
    while (l + 1 < set.n && blockIdx.x >= set.seg[l + 1].chunk0) l++;
    chunk = blockIdx.x - set.seg[l].chunk0;
    return set.seg[l];
}

// first pass: each block's recording bitplane and the chunk's word counts
template <class T, bool ERR, int NW>
__global__ void __launch_bounds__(NW * 32) k_gr_rb(const __grid_constant__ GrSet<T> set, int B,
                                               double* __restrict__ partial) {
    using FP = typename Traits<T>::FP;
    using A = typename Acc<T>::type;
    constexpr int BS = Traits<T>::kBlock, H = BS / 32, BPW = GR_CHUNK / NW;
    constexpr int U = ERR ? 1 : 8 / H;   // blocks loaded ahead
    uint32_t chunk;
    const GrSeg<T>& q = gr_seg(set, chunk);
    const T* __restrict__ x = q.x;
    const uint64_t n = q.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (n + BS - 1) / BS;
    __shared__ uint32_t cnt[NW][64];
    uint32_t c0 = 0, c1 = 0;
    A acc[Acc<T>::N];
    if (ERR) {
#pragma unroll
        for (int k = 0; k < Acc<T>::N; k++) acc[k] = 0;
    }
    pdl_wait();
    pdl_release();
    const int exp = level_exp<T>(q.key, q.exp);
    const bool fast = pow2_normal(B - exp);
    const float sc = fast ? pow2f(B - exp) : 1.f;
    const uint64_t b0 = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * BPW;
    int rv = B;   // lane j: block j's recording plane
    for (int j0 = 0; j0 < BPW && b0 + j0 < nblocks; j0 += U) {
        T v[U * H];
#pragma unroll
        for (int t = 0; t < U * H; t++) {
            const uint64_t i = (b0 + j0) * BS + t * 32 + lane;
            v[t] = i < n ? __ldg(x + i) : (T)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            FP orv = 0;
#pragma unroll
            for (int h = 0; h < H; h++) {
                if constexpr (std::is_same<T, float>::value) {
                    const int64_t fix = (int64_t)scale2(v[u * H + h], B - exp, fast, sc);
                    orv |= (FP)(fix < 0 ? -fix : fix);
                } else {
                    bool neg;
                    T sh;
                    orv |= gr_mag<T, ERR>(v[u * H + h], B, exp, neg, sh);
                    if (ERR && (b0 + j0 + u) * BS + h * 32 + lane < n) gr_errors(acc, (A)fabs(sh), B);
                }
            }
            int r;
            if (BS == 32) {
                const uint32_t o = __reduce_or_sync(FULL, (uint32_t)orv);
                r = o ? B - 1 - (31 - __clz(o)) : B;
            } else {
                const uint32_t lo = __reduce_or_sync(FULL, (uint32_t)orv);
                const uint32_t hi = __reduce_or_sync(FULL, (uint32_t)((uint64_t)orv >> 32));
                r = hi ? B - 1 - (63 - __clz(hi)) : lo ? B - 1 - (31 - __clz(lo)) : B;
            }
            if (lane == j0 + u) rv = r;
            if (b0 + j0 + u < nblocks) {
                c0 += gr_words(r, lane);
                c1 += gr_words(r, lane + 32);
            }
        }
    }
    if (lane < BPW && b0 + lane < nblocks) q.rbs[b0 + lane] = (uint8_t)rv;
    cnt[warp][lane] = c0;
    cnt[warp][lane + 32] = c1;
    __syncthreads();
    if (threadIdx.x < 64 && (int)threadIdx.x < B) {
        uint32_t t = 0;
        for (int w = 0; w < NW; w++) t += cnt[w][threadIdx.x];
        q.cw[(uint64_t)chunk * B + threadIdx.x] = t;
    }
    if (ERR) flush_errors(acc, B, partial);
}

// exclusive scan of the chunks' word counts, per plane (blockIdx.x) and level
// (blockIdx.y); stream byte sizes
template <class T>
__global__ void k_gr_scan(const __grid_constant__ GrSet<T> set, int B) {
    constexpr int BS = Traits<T>::kBlock;
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t carry;
    const GrSeg<T>& q = set.seg[blockIdx.y];
    const uint64_t nblocks = (q.n + BS - 1) / BS, nchunks = (nblocks + GR_CHUNK - 1) / GR_CHUNK;
    const int p = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    pdl_release();
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t base = 0; base < nchunks; base += blockDim.x) {
        const uint64_t c = base + threadIdx.x;
        const uint32_t v = c < nchunks ? q.cw[c * B + p] : 0;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t ws = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
            uint32_t wi = ws;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, wi, o);
                if (lane >= o) wi += t;
            }
            wsum[lane] = wi - ws;   // exclusive warp offsets
        }
        __syncthreads();
        const uint32_t excl = carry + wsum[warp] + incl - v;
        if (c < nchunks) q.co[c * B + p] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        q.sizes[p] = carry * (uint32_t)sizeof(typename Traits<T>::S) + (p == 0 ? (uint32_t)(4 + nblocks) : 0u);
}

// A warp's blocks: its first one's word index in planes lane and lane + 32,
// and the recording planes (lane j: block j; 255, which no plane reaches,
// where there is no block)
template <int NW = GR_WARPS>
__device__ __forceinline__ int gr_warp_offsets(const uint8_t* __restrict__ rbs, uint64_t nblocks, uint64_t chunk,
                                               const uint32_t* __restrict__ chunk_off, int B, uint32_t& off0,
                                               uint32_t& off1) {
    constexpr int BPW = GR_CHUNK / NW;
    __shared__ uint32_t cnt[NW][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t b = chunk * GR_CHUNK + (uint64_t)warp * BPW + lane;
    const int rv = lane < BPW && b < nblocks ? rbs[b] : 255;
    off0 = lane < B ? chunk_off[chunk * B + lane] : 0;
    off1 = lane + 32 < B ? chunk_off[chunk * B + lane + 32] : 0;
    uint32_t c0 = 0, c1 = 0;
#pragma unroll 8
    for (int j = 0; j < BPW; j++) {
        const int r = __shfl_sync(FULL, rv, j);
        c0 += gr_words(r, lane);
        c1 += gr_words(r, lane + 32);
    }
    cnt[warp][lane] = c0;
    cnt[warp][lane + 32] = c1;
    __syncthreads();
    for (int w = 0; w < warp; w++) {
        off0 += cnt[w][lane];
        off1 += cnt[w][lane + 32];
    }
    return rv;
}

// Plane words leave through shared memory, SB blocks of a warp at a time: row
// i holds the words of one plane (one per block that reaches it and the sign
// words of the blocks that start there, so at most 2 SB), and SB lanes write
// them as one run. A lane per plane and one word per block instead, every word
// is a store to a sector of its own.
template <class S, int SB>
struct GrStage {
    static constexpr int LD = 2 * SB + 1;
    // the runs of 32 rows: row i (below rows) has c_i words (lane i's c) and goes to out + i * step + off_i
    static __device__ __forceinline__ void flush(S* out, int64_t step, int rows, const S* stage, uint32_t off, uint32_t c,
                                                 int lane) {
        const int k = lane & (SB - 1);
#pragma unroll 4
        for (int i0 = 0; i0 < rows; i0 += 32 / SB) {
            const int i = i0 + lane / SB;
            const uint32_t o = __shfl_sync(FULL, off, i & 31);
            const int ci = (int)__shfl_sync(FULL, c, i & 31), m = i < rows ? ci : 0;
            S* dst = out + i * step + o;
            if (k < m) dst[k] = stage[i * LD + k];
            if (k + SB < m) dst[k + SB] = stage[i * LD + k + SB];
        }
    }
};

// fp64 writer. 513 x 513 x 257, 60 planes: 326 us; 1050 us with a store per
// word and two blocks loaded at a time (DRAM floor 164 us).
constexpr int GR_SB64 = 8;
constexpr size_t kGrStage64 = (size_t)GR_WARPS * 64 * GrStage<uint64_t, GR_SB64>::LD * sizeof(uint64_t);
__global__ void __launch_bounds__(256, 3) k_gr_write64(const __grid_constant__ GrSet<double> set, int B) {
    using S = uint64_t;
    using Stage = GrStage<S, GR_SB64>;
    constexpr int U = 4;   // blocks loaded ahead
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t chunk;
    const GrSeg<double>& q = gr_seg(set, chunk);
    const double* __restrict__ x = q.x;
    const uint64_t n = q.n, cap = q.cap;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (n + 63) / 64;
    S* stage = (S*)smem + warp * 64 * Stage::LD;
    pdl_wait();
    pdl_release();
    const uint64_t b0 = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * GR_BPW;
    double nx[2 * U];
    auto load = [&](int j0) {
#pragma unroll
        for (int t = 0; t < 2 * U; t++) {
            const uint64_t i = (b0 + j0) * 64 + t * 32 + lane;
            nx[t] = j0 < GR_BPW && i < n ? __ldcs(x + i) : 0.0;
        }
    };
    load(0);
    const int exp = level_exp<double>(q.key, q.exp);
    uint32_t off0, off1, c0 = 0, c1 = 0;
    const int rv = gr_warp_offsets(q.rbs, nblocks, chunk, q.co, B, off0, off1);
    for (int j0 = 0; j0 < GR_BPW && b0 + j0 < nblocks; j0 += U) {
        double v[2 * U];
#pragma unroll
        for (int t = 0; t < 2 * U; t++) v[t] = nx[t];
        load(j0 + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = __shfl_sync(FULL, rv, j0 + u);
            uint64_t m[2];
            S sign = 0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                bool neg;
                double sh;
                m[h] = gr_mag<double, false>(v[2 * u + h], B, exp, neg, sh);
                sign |= (S)__ballot_sync(FULL, neg) << (h * 32);
            }
            // encode_block :337-357 by four warp bit transposes: lane k gets the
            // words of magnitude bit k (low halves) and bit 32 + k (high halves)
            // of values 0..31 and 32..63; lane p then fetches plane p (bit
            // B-1-p) and plane p + 32 (bit B-33-p). Planes below r are not written.
            const uint32_t lo0 = transpose32((uint32_t)m[0], lane), hi0 = transpose32((uint32_t)(m[0] >> 32), lane);
            const uint32_t lo1 = transpose32((uint32_t)m[1], lane), hi1 = transpose32((uint32_t)(m[1] >> 32), lane);
            S w[2];
#pragma unroll
            for (int t = 0; t < 2; t++) {   // plane lane + 32 t (a valid plane for the shuffles' sake)
                const int p = lane + 32 * t < B ? lane + 32 * t : 0;
                const int k = B - 1 - p, src = k & 31;
                const uint32_t a0 = __shfl_sync(FULL, lo0, src), d0 = __shfl_sync(FULL, hi0, src);
                const uint32_t a1 = __shfl_sync(FULL, lo1, src), d1 = __shfl_sync(FULL, hi1, src);
                w[t] = k >= 32 ? ((S)d1 << 32 | d0) : ((S)a1 << 32 | a0);
            }
            if (lane >= r) {
                S* dst = stage + lane * Stage::LD + c0;
                if (lane == r) *dst++ = sign;
                *dst = w[0];
            }
            if (lane + 32 >= r) {
                S* dst = stage + (lane + 32) * Stage::LD + c1;
                if (lane + 32 == r) *dst++ = sign;
                *dst = w[1];
            }
            c0 += gr_words(r, lane);
            c1 += gr_words(r, lane + 32);
        }
        if ((j0 + U) % GR_SB64 == 0 || b0 + j0 + U >= nblocks) {
            __syncwarp();
            Stage::flush(q.out, (int64_t)cap, min(B, 32), stage, off0, c0, lane);
            Stage::flush(q.out + 32 * cap, (int64_t)cap, B - 32, stage + 32 * Stage::LD, off1, c1, lane);
            __syncwarp();
            off0 += c0;
            off1 += c1;
            c0 = c1 = 0;
        }
    }
}

// fp32 grouped writer: one transpose per block instead of B ballots (150 x 257
// x 301, 32 planes: 41 us, 88 us with a store per word). With
// ERR, the exact squared-error tables (errtab.cuh, GroupedBPEncoder.hpp:76-145
// with collect_level_errors :324-335) of the CTA's chunk go to its record
// recs + blockIdx.x (one level per launch): four blocks per step, t =
// trunc(|x|), bit counts from the transposed magnitude words.
constexpr size_t kErrSmemGR = 8 * sizeof(errtab::WarpQ) + errtab::kSlotsPad * sizeof(unsigned long long);

template <bool ERR>
__global__ void __launch_bounds__(256) k_gr_write32(const __grid_constant__ GrSet<float> set, int B,
                                                   unsigned long long* __restrict__ recs) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t chunk;
    const GrSeg<float>& q = gr_seg(set, chunk);
    const float* __restrict__ x = q.x;
    const uint64_t n = q.n, cap = q.cap;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (n + 31) / 32;
    constexpr int SB = ERR ? 8 : 16, U = 4;   // blocks staged; blocks loaded ahead
    using Stage = GrStage<uint32_t, SB>;
    __shared__ uint32_t stages[GR_WARPS][32 * Stage::LD];
    uint32_t* stage = stages[warp];
    pdl_wait();
    pdl_release();
    const uint64_t b0 = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * GR_BPW;
    float nx[U];
    auto load = [&](int j0) {
#pragma unroll
        for (int g = 0; g < U; g++) {
            const uint64_t i = (b0 + j0 + g) * 32 + lane;
            nx[g] = j0 < GR_BPW && i < n ? __ldcs(x + i) : 0.f;
        }
    };
    load(0);
    const int exp = level_exp<float>(q.key, q.exp);
    uint32_t off0, off1;
    const int rv = gr_warp_offsets(q.rbs, nblocks, chunk, q.co, B, off0, off1);
    const int plane = B - 1 - lane;                    // lane k owns bit k, row k of the stage
    uint32_t off = __shfl_sync(FULL, off0, plane & 31), c = 0;
    const bool fast = pow2_normal(B - exp);
    const float sc = fast ? pow2f(B - exp) : 1.f;
    errtab::WarpQ* wq = (errtab::WarpQ*)smem;
    unsigned long long* red = (unsigned long long*)(wq + 8);
    errtab::Lane acc;
    uint32_t head = 0;
    int qn = 0;
    if (ERR) {
        acc.zero();
        errtab::zero_q(wq[warp], lane);
    }
    for (int j0 = 0; j0 < GR_BPW && (ERR || b0 + j0 < nblocks); j0 += U) {
        float v[U], sh[U], mag[U];
        uint32_t m[U], sign[U];
        bool small[U];
#pragma unroll
        for (int g = 0; g < U; g++) v[g] = nx[g];
        load(j0 + U);
#pragma unroll
        for (int g = 0; g < U; g++) {
            const bool ok = (b0 + j0 + g) * 32 + lane < n;
            sh[g] = scale2(v[g], B - exp, fast, sc);
            const int64_t fix = (int64_t)sh[g];
            const bool neg = v[g] < 0.f;
            m[g] = (uint32_t)(neg ? -fix : fix);
            sign[g] = __ballot_sync(FULL, neg);
            if (ERR) {
                mag[g] = fabsf(sh[g]);
                const bool big = mag[g] >= 8388608.f;
                acc.add_big_square(mag[g], big);                              // padding is 0: never big
                small[g] = ok && !big;
            }
        }
        if (ERR) {
            errtab::enqueue4(wq[warp], head, qn, small, mag, lane);
            errtab::drain_full<false>(wq[warp], head, qn, lane);
            acc.add4(m[0], m[1], m[2], m[3]);
        }
#pragma unroll
        for (int g = 0; g < U; g++) {
            const uint32_t w = transpose32(m[g], lane);
            if (ERR) acc.pc += __popc(w);
            const int r = __shfl_sync(FULL, rv, j0 + g);
            if (plane >= r) {
                uint32_t* dst = stage + lane * Stage::LD + c;
                if (plane == r) *dst++ = sign[g];
                *dst = w;
            }
            c += gr_words(r, plane);
        }
        if ((j0 + U) % SB == 0 || (!ERR && b0 + j0 + U >= nblocks)) {
            __syncwarp();
            Stage::flush(q.out + (B - 1) * (int64_t)cap, -(int64_t)cap, B, stage, off, c, lane);
            __syncwarp();
            off += c;
            c = 0;
        }
    }
    if (ERR) {
        if (qn) {
            __syncwarp();
            errtab::run_batch<false>(wq[warp], head, qn, lane);
        }
        unsigned long long* rec = recs + (size_t)blockIdx.x * errtab::kSlotsPad;
        for (int k = threadIdx.x; k < errtab::kSlotsPad; k += blockDim.x) rec[k] = 0;
        __syncthreads();
        errtab::flush(acc, wq, red, rec);
    }
}

// GroupedBPEncoder::progressive_decode -- :210-297 (planes [s, e)); plane p's
// words at planes[p] (absolute plane index). signs: per-block sign words kept
// between calls (nullable when s == 0). A device count (dnum[0]) overrides e.
// Lane p loads plane p's word of a block (planes p and p + 32 in 64 bits),
// GR_DU blocks ahead of the ones in work. The sign words of a warp's 32 blocks
// are fetched together before them, lane j block j's: gr_signs.
// 513 x 513 x 257 fp64, most of 60 planes: 284 us; 419 us with four blocks
// loaded, decoded and stored in turn and the sign words among them.
template <int BPW, class S>
__device__ __forceinline__ S gr_signs(const S* const* __restrict__ planes, S* signs, uint64_t b, int rv, uint32_t off0,
                                      uint32_t off1, int s, int e, int lane) {
    uint32_t at = 0;   // where block lane's sign word stands in its plane
#pragma unroll 8
    for (int j = 0; j < BPW; j++) {
        const int r = __shfl_sync(FULL, rv, j);
        uint32_t o = __shfl_sync(FULL, off0, r & 31);
        if (sizeof(S) == 8) {
            const uint32_t o1 = __shfl_sync(FULL, off1, r & 31);
            o = r < 32 ? o : o1;
            off1 += gr_words(r, lane + 32);
        }
        off0 += gr_words(r, lane);
        if (lane == j) at = o;
    }
    if (rv >= e) return 0;                 // nothing of the block is there yet (or there is no block)
    if (rv < s) return signs[b + lane];    // kept by an earlier call
    const S sign = __ldcs(planes[rv] + at);
    if (signs) signs[b + lane] = sign;
    return sign;
}
constexpr int GR_DU = 4;

template <int NW>
__global__ void __launch_bounds__(NW * 32) k_gr_decode32(const __grid_constant__ GrSet<float> set, int B, int s, int e) {
    constexpr int BPW = GR_CHUNK / NW, U = 2 * GR_DU;
    uint32_t chunk;
    const GrSeg<float>& q = gr_seg(set, chunk);
    const uint64_t n = q.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (n + 31) / 32;
    pdl_wait();
    pdl_release();
    if (q.dnum) e = q.dnum[0];
    const int exp = level_exp<float>(q.key, q.exp);
    uint32_t off, unused;
    const int rv = gr_warp_offsets<NW>(q.rbs, nblocks, chunk, q.co, B, off, unused);
    const uint32_t* src = (lane < B && lane >= s && lane < e) ? q.planes[lane] : nullptr;
    const bool fast = pow2_normal(exp - e);
    const float sc = fast ? pow2f(exp - e) : 1.f;
    const uint64_t b0 = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * BPW;
    const uint32_t signs = gr_signs<BPW>(q.planes, q.signs, b0, rv, off, 0u, s, e, lane);
    uint32_t nx[U];
    auto load = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = j0 < BPW ? __shfl_sync(FULL, rv, j0 + u) : 255;
            nx[u] = src && lane >= r ? __ldcs(src + off + (lane == r ? 1 : 0)) : 0;
            off += gr_words(r, lane);
        }
    };
    load(0);
    for (int j0 = 0; j0 < BPW && b0 + j0 < nblocks; j0 += U) {
        uint32_t w[U];
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = nx[u];
        load(j0 + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = __shfl_sync(FULL, rv, j0 + u);
            const uint32_t sign = __shfl_sync(FULL, signs, j0 + u);
            const uint64_t i = (b0 + j0 + u) * 32 + lane;
            if (r < e) {
                const uint32_t col = transpose32(w[u], lane);
                const uint32_t acc = __brev(col) >> (32 - e);
                const float v = scale2((float)acc, exp - e, fast, sc);
                if (i < n) q.y[i] = ((sign >> lane) & 1u) ? -v : v;
            } else if (i < n) {
                q.y[i] = 0.f;
            }
        }
    }
}

// fp64
template <int NW>
__global__ void __launch_bounds__(NW * 32) k_gr_decode64(const __grid_constant__ GrSet<double> set, int B, int s, int e) {
    using S = uint64_t;
    constexpr int BPW = GR_CHUNK / NW, U = GR_DU;
    uint32_t chunk;
    const GrSeg<double>& q = gr_seg(set, chunk);
    const uint64_t n = q.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (n + 63) / 64;
    pdl_wait();
    pdl_release();
    if (q.dnum) e = q.dnum[0];
    const int exp = level_exp<double>(q.key, q.exp);
    uint32_t off0, off1;
    const int rv = gr_warp_offsets<NW>(q.rbs, nblocks, chunk, q.co, B, off0, off1);
    const S* src0 = (lane >= s && lane < e) ? q.planes[lane] : nullptr;
    const S* src1 = (lane + 32 >= s && lane + 32 < e) ? q.planes[lane + 32] : nullptr;
    const uint64_t b0 = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * BPW;
    const S signs = gr_signs<BPW>(q.planes, q.signs, b0, rv, off0, off1, s, e, lane);
    S n0[U], n1[U];
    auto load = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = j0 < BPW ? __shfl_sync(FULL, rv, j0 + u) : 255;
            n0[u] = src0 && lane >= r ? __ldcs(src0 + off0 + (lane == r ? 1 : 0)) : 0;
            n1[u] = src1 && lane + 32 >= r ? __ldcs(src1 + off1 + (lane + 32 == r ? 1 : 0)) : 0;
            off0 += gr_words(r, lane);
            off1 += gr_words(r, lane + 32);
        }
    };
    load(0);
    for (int j0 = 0; j0 < BPW && b0 + j0 < nblocks; j0 += U) {
        S w0[U], w1[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            w0[u] = n0[u];
            w1[u] = n1[u];
        }
        load(j0 + U);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int r = __shfl_sync(FULL, rv, j0 + u);
            const S sign = __shfl_sync(FULL, signs, j0 + u);
            const uint64_t i = (b0 + j0 + u) * 64 + lane;
            if (r < e) {
                // decode_block :359-368 by four warp bit transposes: lane p holds
                // planes p and p + 32 (zero where not read); after the
                // transposes lane v holds, per half h of the block, a word whose
                // bit p is plane p's bit of value 32 h + v (planes 0..31) and one
                // for planes 32..63. Plane p weighs 2^(e-1-p): the bit-reversed
                // words, shifted into place.
                const uint32_t pl0 = transpose32((uint32_t)w0[u], lane), ph0 = transpose32((uint32_t)(w0[u] >> 32), lane);
                uint32_t pl1 = 0, ph1 = 0;
                if (e > 32) {
                    pl1 = transpose32((uint32_t)w1[u], lane);
                    ph1 = transpose32((uint32_t)(w1[u] >> 32), lane);
                }
                // planes 0..31 -> bits e-1 .. e-32, planes 32..63 -> bits e-33 ..
                const uint64_t a0 = (uint64_t)__brev(pl0) << 32 | __brev(pl1);   // plane p at bit 63 - p
                const uint64_t a1 = (uint64_t)__brev(ph0) << 32 | __brev(ph1);
                if (i < n) q.y[i] = gr_value<double>(a0 >> (64 - e), exp - e, (sign >> lane) & 1u);
                if (i + 32 < n) q.y[i + 32] = gr_value<double>(a1 >> (64 - e), exp - e, (sign >> (lane + 32)) & 1u);
            } else {
                if (i < n) q.y[i] = 0.0;
                if (i + 32 < n) q.y[i + 32] = 0.0;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Squared error collector -- SquaredErrorCollector.hpp:54-96. The bit-clearing
// loop is evaluated in closed form: entry k receives (v - v with bits <= b
// cleared)^2 for b = exp_diff + (idx0 - k) while b < prec, else v^2.
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) k_sq_collect(const T* __restrict__ x, uint64_t n, int B, T maxv,
                                                    double* __restrict__ partial) {
    using A = typename Acc<T>::type;
    using U = typename Traits<T>::Bits;
    constexpr int prec = Traits<T>::kPrec;
    A acc[Acc<T>::N];
#pragma unroll
    for (int k = 0; k < Acc<T>::N; k++) acc[k] = 0;
    const int lexp = frexp_exp(maxv);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        T v = x[i];
        if (v == (T)0) continue;
        int de = frexp_exp(v);
        U bits;
        memcpy(&bits, &v, sizeof(T));
        int exp_diff = lexp - de + prec - B;
        int idx0 = B;
        if (exp_diff <= 0) { idx0 += exp_diff; exp_diff = 0; }
        if (idx0 <= 0) continue;
        const T vv = v * v;
#pragma unroll
        for (int k = 0; k < Acc<T>::N; k++) {
            if (k <= idx0 && k <= B) {
                int bb = exp_diff + (idx0 - k);
                if (bb < prec) {
                    U cleared = bits & ~((((U)2) << bb) - (U)1);
                    T f;
                    memcpy(&f, &cleared, sizeof(T));
                    T d = v - f;
                    acc[k] += (A)(d * d);
                } else {
                    acc[k] += (A)vv;
                }
            }
        }
    }
    flush_errors(acc, B, partial);
}

// sum partial tables in fixed order, then scale by 2^(2*(exp - B)) when exp
// scaling applies (encoder tables, NegaBinaryBPEncoder.hpp:121-123).
template <class T>
__global__ void k_reduce_partials(const double* __restrict__ partial, int nparts, int B,
                                  const typename KeyOf<T>::type* __restrict__ maxkey, int exp_arg, int exp_add,
                                  int scale, double* __restrict__ out) {
    // one warp per table entry; lane-strided partial sums then a fixed-order
    // shuffle tree, so the result does not depend on scheduling
    const int lane = threadIdx.x & 31;
    for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k <= B; k += gridDim.x * (blockDim.x >> 5)) {
        double s = 0;
        for (int p = lane; p < nparts; p += 32) s += partial[(size_t)p * (B + 1) + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) {
            if (scale) {
                int exp = level_exp<T>(maxkey, exp_arg) + exp_add;
                s = ldexp(s, 2 * (-B + exp));
            }
            out[k] = s;
        }
    }
}

// per-chunk word counts from the rb arrays (used when only the headers are known)
template <class T>
__global__ void k_chunk_words_from_rb(const __grid_constant__ GrSet<T> set, int B) {
    constexpr int BS = Traits<T>::kBlock;
    uint32_t chunk;
    const GrSeg<T>& q = gr_seg(set, chunk);
    __shared__ uint32_t cnt[GR_WARPS][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t nblocks = (q.n + BS - 1) / BS;
    const uint64_t b = (uint64_t)chunk * GR_CHUNK + (uint64_t)warp * GR_BPW + lane;
    const int rv = b < nblocks ? q.rbs[b] : 255;
    uint32_t c0 = 0, c1 = 0;
#pragma unroll 8
    for (int j = 0; j < GR_BPW; j++) {
        const int r = __shfl_sync(FULL, rv, j);
        c0 += gr_words(r, lane);
        c1 += gr_words(r, lane + 32);
    }
    cnt[warp][lane] = c0;
    cnt[warp][lane + 32] = c1;
    __syncthreads();
    if (threadIdx.x < 64 && (int)threadIdx.x < B) {
        uint32_t s = 0;
        for (int w = 0; w < GR_WARPS; w++) s += cnt[w][threadIdx.x];
        q.cw[(uint64_t)chunk * B + threadIdx.x] = s;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
// opt-in to more than 48 KB of dynamic shared memory, once per device and kernel
static int allow_smem(const void* k, size_t bytes) {
    static std::mutex mu;
    static std::vector<std::pair<int, const void*>> done;
    int dev = 0;
    PRODM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    for (const auto& d : done)
        if (d.first == dev && d.second == k) return PRODM_OK;
    PRODM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done.push_back({dev, k});
    return PRODM_OK;
}

// the opt-in comes first: the occupancy query counts it
static unsigned nb_err_grid(uint64_t need) {
    (void)allow_smem((const void*)k_nb_encode32_err, kErrSmemNB);
    return persistent_grid_for((const void*)k_nb_encode32_err, 256, kErrSmemNB, need, kPartialSlots);
}

// fp32 negabinary with tables: the encode launch (records in partial), then
// the final reduction of nseg levels into errs_out
static int nb_err_launch(const ChunkSeg* segs, const ChunkSeg& one, int nseg, uint64_t total, int B, int exp,
                         double* partial, double* errs_out, cudaStream_t st) {
    int rc;
    if ((rc = allow_smem((const void*)k_nb_encode32_err, kErrSmemNB))) return rc;
    const unsigned grid = nb_err_grid(segs ? (uint64_t)kPartialSlots : total);
    unsigned long long* recs = (unsigned long long*)partial;
    k_nb_encode32_err<<<grid, 256, kErrSmemNB, st>>>(segs, one, nseg, total, B, exp, recs);
    PRODM_CHECK_LAUNCH("k_nb_encode32_err");
    k_errtab_final<true><<<nseg, 1024, 0, st>>>(recs, (int)grid, B, segs, one, exp, 2, errs_out);
    PRODM_CHECK_LAUNCH("k_errtab_final");
    return PRODM_OK;
}

template <class T>
int launch_nb_encode(const T* x, uint64_t n, const void* maxkey, int exp, int B, void* out, uint64_t stride,
                     double* partial, double* errs_out, cudaStream_t st) {
    using K = typename KeyOf<T>::type;
    constexpr int BS = Traits<T>::kBlock;
    const uint64_t nblocks = (n + BS - 1) / BS;
    const int th = 256;
    if (std::is_same<T, float>::value) {
        const uint64_t nch = (nblocks + NB_CHUNK - 1) / NB_CHUNK;
        if (errs_out) {
            ChunkSeg one = {};
            one.x = (const float*)x;
            one.words = (uint32_t*)out;
            one.n = n;
            one.nblocks = nblocks;
            one.stride = stride;
            one.key = (const uint32_t*)maxkey;
            return nb_err_launch(nullptr, one, 1, nch, B, exp, partial, errs_out, st);
        }
        const unsigned grid = persistent_grid_for((const void*)k_nb_encode32, th, 0, nch, nch);
        k_nb_encode32<<<grid, th, 0, st>>>((const float*)x, n, (const uint32_t*)maxkey, exp, B, (uint32_t*)out, stride);
        PRODM_CHECK_LAUNCH("k_nb_encode32");
        return PRODM_OK;
    }
    if constexpr (std::is_same<T, double>::value) {
        if (errs_out) {
            const unsigned grid = persistent_grid_for((const void*)k_nb_encode64_err, th, 0, nblocks, kPartialSlots);
            k_nb_encode64_err<<<grid, th, 0, st>>>(x, n, (const K*)maxkey, exp, B, (uint64_t*)out, stride, partial);
            PRODM_CHECK_LAUNCH("k_nb_encode64_err");
            k_reduce_partials<T><<<(B + 8) / 8, 256, 0, st>>>(partial, (int)grid, B, (const K*)maxkey, exp, 2, 1, errs_out);
            PRODM_CHECK_LAUNCH("k_reduce_partials");
        } else {
            const uint64_t nch = (nblocks + 8 * NB64_BLOCKS - 1) / (8 * NB64_BLOCKS);
            const unsigned grid = persistent_grid_for((const void*)k_nb_encode64, th, 0, nch, nch);
            count_launch();
            const cudaError_t e = launch_chain(true, k_nb_encode64, dim3(grid), dim3(th), 0, st, x, n, (const K*)maxkey, exp, B,
                                               (uint64_t*)out, stride);
            if (e != cudaSuccess) return cuda_status(e, "k_nb_encode64");
        }
    }
    return PRODM_OK;
}

int launch_nb_decode_levels(const ChunkSeg* segs, int nseg, uint64_t total_chunks, cudaStream_t st, bool pdl) {
    const unsigned grid = persistent_grid_for((const void*)k_nb_decode_levels, 256, 0, total_chunks, total_chunks);
    count_launch();
    const cudaError_t e = launch_chain(pdl, k_nb_decode_levels, dim3(grid), dim3(256), 0, st, segs, nseg, total_chunks);
    if (e != cudaSuccess) return cuda_status(e, "k_nb_decode_levels");
    return PRODM_OK;
}

int nb_encode_levels_grid(int with_errors) {
    if (with_errors) return (int)nb_err_grid((uint64_t)kPartialSlots);
    return (int)persistent_grid_for((const void*)k_nb_encode32_levels, 256, 0, (uint64_t)kPartialSlots, kPartialSlots);
}

int launch_nb_encode_levels(const ChunkSeg* segs, int nseg, uint64_t total_chunks, int B, double* partial,
                            double* errs_out, cudaStream_t st) {
    if (errs_out) return nb_err_launch(segs, ChunkSeg{}, nseg, total_chunks, B, 0, partial, errs_out, st);
    return launch_nb_encode_segments(segs, nseg, total_chunks, B, (unsigned)nb_encode_levels_grid(0), st, true);
}

int launch_nb_encode_segments(const ChunkSeg* segs, int nseg, uint64_t total_chunks, int B, unsigned grid, cudaStream_t st,
                              bool pdl) {
    count_launch();
    const cudaError_t e = launch_chain(pdl, k_nb_encode32_levels, dim3(grid), dim3(256), 0, st, segs, nseg, total_chunks, B);
    if (e != cudaSuccess) return cuda_status(e, "k_nb_encode32_levels");
    return PRODM_OK;
}

template <class T>
int launch_nb_decode(const void* base, uint64_t stride, uint64_t n, const void* maxkey, int exp, int s, int num,
                     const uint8_t* dnum, T* out, cudaStream_t st) {
    using K = typename KeyOf<T>::type;
    constexpr int BS = Traits<T>::kBlock;
    const uint64_t nblocks = (n + BS - 1) / BS;
    const int th = 256;
    if (std::is_same<T, float>::value) {
        const uint64_t nch = (nblocks + NB_CHUNK - 1) / NB_CHUNK;
        const unsigned grid = persistent_grid_for((const void*)k_nb_decode32, th, 0, nch, nch);
        k_nb_decode32<<<grid, th, 0, st>>>((const uint32_t*)base, stride, n, (const uint32_t*)maxkey, exp, s, num, dnum,
                                           (float*)out);
        PRODM_CHECK_LAUNCH("k_nb_decode32");
        return PRODM_OK;
    }
    if constexpr (std::is_same<T, double>::value) {
        const uint64_t nch = (nblocks + 8 * NB64_BLOCKS - 1) / (8 * NB64_BLOCKS);
        const unsigned grid = persistent_grid_for((const void*)k_nb_decode64, th, 0, nch, nch);
        count_launch();
        const cudaError_t e = launch_chain(true, k_nb_decode64, dim3(grid), dim3(th), 0, st, (const uint64_t*)base, stride, n,
                                           (const K*)maxkey, exp, s, num, dnum, out);
        if (e != cudaSuccess) return cuda_status(e, "k_nb_decode64");
    }
    return PRODM_OK;
}

uint64_t gr_nchunks(uint64_t nblocks) { return (nblocks + GR_CHUNK - 1) / GR_CHUNK; }

// the segments' first chunks; the launch's chunks
template <class T>
static unsigned gr_number(GrSet<T>& set) {
    uint64_t c = 0;
    for (int l = 0; l < set.n; l++) {
        set.seg[l].chunk0 = (uint32_t)c;
        c += gr_nchunks((set.seg[l].n + Traits<T>::kBlock - 1) / Traits<T>::kBlock);
    }
    return (unsigned)c;
}

#define PRODM_CHAIN(name, ...)                                   \
    do {                                                         \
        count_launch();                                          \
        const cudaError_t e_ = launch_chain(true, __VA_ARGS__);  \
        if (e_ != cudaSuccess) return cuda_status(e_, name);     \
    } while (0)

template <class T>
int launch_gr_encode(GrSet<T> set, int B, double* partial, double* errs_out, cudaStream_t st) {
    constexpr bool f32 = std::is_same<T, float>::value;
    const dim3 grid(gr_number(set)), block(GR_WARPS * 32);
    if (errs_out && set.n != 1) return fail(PRODM_EINVAL, "grouped encode: error tables take one level per call");
    if (!grid.x) return PRODM_OK;
    if (!f32 && errs_out) {
        if constexpr (!f32) {
            PRODM_CHAIN("k_gr_rb", (k_gr_rb<T, true, GR_WARPS>), grid, block, 0, st, set, B, partial);
            k_reduce_partials<T><<<(B + 8) / 8, 256, 0, st>>>(partial, (int)grid.x, B, set.seg[0].key, set.seg[0].exp, 0,
                                                             1, errs_out);
            PRODM_CHECK_LAUNCH("k_reduce_partials");
        }
    } else {
        const int warps = f32 || gr_wide64(grid.x) ? GR_WIDE : GR_WARPS;
        PRODM_CHAIN("k_gr_rb", (warps == GR_WIDE ? k_gr_rb<T, false, GR_WIDE> : k_gr_rb<T, false, GR_WARPS>), grid,
                    dim3(warps * 32), 0, st, set, B, (double*)nullptr);
    }
    PRODM_CHAIN("k_gr_scan", k_gr_scan<T>, dim3(B, set.n), dim3(1024), 0, st, set, B);
    if constexpr (f32) {
        unsigned long long* recs = (unsigned long long*)partial;
        if (errs_out) {
            // (with the static stages above the 48 KB that need no leave)
            const cudaError_t e = cudaFuncSetAttribute((const void*)k_gr_write32<true>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kErrSmemGR);
            if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute");
            PRODM_CHAIN("k_gr_write32", k_gr_write32<true>, grid, block, kErrSmemGR, st, set, B, recs);
            ChunkSeg one = {};
            one.n = set.seg[0].n;
            one.key = set.seg[0].key;
            k_errtab_final<false><<<1, 1024, 0, st>>>(recs, (int)grid.x, B, nullptr, one, set.seg[0].exp, 0, errs_out);
            PRODM_CHECK_LAUNCH("k_errtab_final");
        } else {
            PRODM_CHAIN("k_gr_write32", k_gr_write32<false>, grid, block, 0, st, set, B, (unsigned long long*)nullptr);
        }
    } else {
        const cudaError_t e = cudaFuncSetAttribute((const void*)k_gr_write64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)kGrStage64);
        if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute");
        PRODM_CHAIN("k_gr_write64", k_gr_write64, grid, block, kGrStage64, st, set, B);
    }
    return PRODM_OK;
}

// chunk offsets and plane sizes of levels whose rb arrays are known
template <class T>
int launch_gr_offsets(GrSet<T> set, int B, cudaStream_t st) {
    const unsigned grid = gr_number(set);
    if (!grid) return PRODM_OK;
    k_chunk_words_from_rb<T><<<grid, GR_WARPS * 32, 0, st>>>(set, B);
    PRODM_CHECK_LAUNCH("k_chunk_words_from_rb");
    k_gr_scan<T><<<dim3(B, set.n), 1024, 0, st>>>(set, B);
    PRODM_CHECK_LAUNCH("k_gr_scan");
    return PRODM_OK;
}

template <class T>
int launch_gr_decode(GrSet<T> set, int B, int s, int e, cudaStream_t st) {
    const dim3 grid(gr_number(set));
    if (!grid.x) return PRODM_OK;
    if constexpr (std::is_same<T, float>::value) {
        const int warps = gr_wide_decode32(grid.x) ? GR_WIDE : GR_WARPS;
        PRODM_CHAIN("k_gr_decode32", (warps == GR_WIDE ? k_gr_decode32<GR_WIDE> : k_gr_decode32<GR_WARPS>), grid,
                    dim3(warps * 32), 0, st, set, B, s, e);
    } else {
        const int warps = gr_wide64(grid.x) ? GR_WIDE : GR_WARPS;
        PRODM_CHAIN("k_gr_decode64", (warps == GR_WIDE ? k_gr_decode64<GR_WIDE> : k_gr_decode64<GR_WARPS>), grid,
                    dim3(warps * 32), 0, st, set, B, s, e);
    }
    return PRODM_OK;
}

#undef PRODM_CHAIN

template <class T>
int launch_sq_collect(const T* x, uint64_t n, int B, T maxv, double* partial, double* out, cudaStream_t st) {
    const int th = 256;
    const unsigned grid = persistent_grid_for((const void*)k_sq_collect<T>, th, 0, (n + th - 1) / th, kPartialSlots);
    k_sq_collect<T><<<grid, th, 0, st>>>(x, n, B, maxv, partial);
    PRODM_CHECK_LAUNCH("k_sq_collect");
    k_reduce_partials<T><<<(B + 8) / 8, 256, 0, st>>>(partial, (int)grid, B, nullptr, 0, 0, 0, out);
    PRODM_CHECK_LAUNCH("k_reduce_partials");
    return PRODM_OK;
}

#define INST(T)                                                                                                       \
    template int launch_nb_encode<T>(const T*, uint64_t, const void*, int, int, void*, uint64_t, double*, double*,    \
                                     cudaStream_t);                                                                   \
    template int launch_nb_decode<T>(const void*, uint64_t, uint64_t, const void*, int, int, int, const uint8_t*, T*, \
                                     cudaStream_t);                                                                   \
    template int launch_gr_encode<T>(GrSet<T>, int, double*, double*, cudaStream_t);                                  \
    template int launch_gr_offsets<T>(GrSet<T>, int, cudaStream_t);                                                   \
    template int launch_gr_decode<T>(GrSet<T>, int, int, int, cudaStream_t);                                          \
    template int launch_sq_collect<T>(const T*, uint64_t, int, T, double*, double*, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace prodm
