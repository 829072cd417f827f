// Host-side launchers of the CUDA kernels (declarations).
#pragma once
#include <functional>
#include <vector>

#include "common.cuh"

namespace prodm {

// mgard.cu
template <class T>
int launch_decompose_level_packed(const T* in, uint64_t s0, uint64_t s1, const Box& F, const Box& C, T* coef, T* coarse,
                                  T* fnat, void* maxkey_level, void* maxkey_coarse, cudaStream_t st);
template <class T>
int launch_decompose_level_inplace(const T* in, const Box& F, const Box& C, T* out, uint64_t o0, uint64_t o1, T* fnat,
                                   cudaStream_t st);
template <class T>
int launch_recompose_level_packed(const T* coarse, const T* coef, const Box& F, const Box& C, T* out, uint64_t s0,
                                  uint64_t s1, cudaStream_t st, bool pdl = false);
template <class T>
int launch_recompose_level_inplace(const T* rin, const Box& F, const Box& C, T* out, uint64_t s0, uint64_t s1,
                                   cudaStream_t st);
template <class T>
int launch_copy_box(const T* src, uint64_t a0, uint64_t a1, const Box& B, T* dst, uint64_t b0, uint64_t b1,
                    cudaStream_t st);
template <class T>
int launch_coef_to_natural(const T* coef, const Box& F, const Box& C, T* fnat, cudaStream_t st);
template <class T>
int launch_reordered_to_natural(const T* rin, const Box& F, const Box& C, T* fnat, cudaStream_t st);
template <class W>
void mass_factors(uint32_t n, W* tab);
// coef != nullptr: read the level's packed coefficients (coarse box *C) instead of fnat
template <class T>
int launch_l2_correction(const T* fnat, const Box& F, T* t1, T* t2, T* z, const T* const tabs[3], cudaStream_t st,
                         const T* coef = nullptr, const Box* C = nullptr);
template <class T>
int launch_add_box(T* dst, uint64_t b0, uint64_t b1, const T* z, const Box& B, T sign, cudaStream_t st);
template <class T>
int launch_interleave(T* data, uint64_t s0, uint64_t s1, const Box& F, const Box& C, T* buf, bool gather,
                      cudaStream_t st);

// adjoint.cu: transpose of one hierarchical recomposition level (field
// gradient of box F -> gradient of the level's packed coefficients and of the
// coarse box C, natural order)
template <class T>
int launch_recompose_adjoint_level(const T* g, const Box& F, const Box& C, T* gcoef, T* gcoarse, cudaStream_t st);
// the same for the orthogonal basis (tabs: Thomas factors per dim; scratch
// boxes (n0, c1, c2), (n0, n1, c2), F, and one C box)
template <class T>
int launch_recompose_adjoint_level_orth(const T* g, const Box& F, const Box& C, T* gcoef, T* gcoarse,
                                        const T* const tabs[3], T* s_a, T* s_b, T* s_w, T* s_u, cudaStream_t st);

// bitplane.cu
template <class T>
int launch_nb_encode(const T* x, uint64_t n, const void* maxkey, int exp, int B, void* out, uint64_t stride,
                     double* partial, double* errs_out, cudaStream_t st);
template <class T>
int launch_nb_decode(const void* base, uint64_t stride, uint64_t n, const void* maxkey, int exp, int s, int num,
                     const uint8_t* dnum, T* out, cudaStream_t st);
uint64_t gr_nchunks(uint64_t nblocks);
// grouped encoder: one segment per level of a launch; planes p of a level's
// streams at out + p * cap (encode) or planes[p] (decode)
template <class T>
struct GrSeg {
    const T* x;                                       // encode input
    T* y;                                             // decode output
    const typename KeyOf<T>::type* key;               // level |max| key, or NULL and the exponent exp
    uint8_t* rbs;                                     // recording planes, one per block
    uint32_t* cw;                                     // encode: word counts, [chunk][B]
    uint32_t* co;                                     // word offsets, [chunk][B]
    uint32_t* sizes;                                  // encode: stream bytes, B
    typename Traits<T>::S* out;
    const typename Traits<T>::S* const* planes;
    typename Traits<T>::S* signs;                     // decode: sign words kept between calls, or NULL
    const uint8_t* dnum;                              // decode: planes (overrides e), or NULL
    uint64_t n, cap;
    uint32_t chunk0;                                  // set by the launchers
    int exp;
};
constexpr int kGrLevels = 17;
template <class T>
struct GrSet {
    int n;
    GrSeg<T> seg[kGrLevels];
};
template <class T>
int launch_gr_encode(GrSet<T> set, int B, double* partial, double* errs_out, cudaStream_t st);
template <class T>
int launch_gr_offsets(GrSet<T> set, int B, cudaStream_t st);
template <class T>
int launch_gr_decode(GrSet<T> set, int B, int s, int e, cudaStream_t st);
template <class T>
int launch_sq_collect(const T* x, uint64_t n, int B, T maxv, double* partial, double* out, cudaStream_t st);
constexpr int kPartialSlots = kSMs * 4;   // per-CTA partial error tables of the fused collectors
// bytes of `parts` per-CTA partials: B + 1 doubles (fp64 tables, squared-error
// collector) or one record of the exact fp32 tables (errtab.cuh)
constexpr int kErrRecWords = 200;   // errtab::kSlotsPad
inline uint64_t partial_bytes(uint64_t parts, int B) {
    return parts * (uint64_t)(kErrRecWords > B + 1 ? kErrRecWords : B + 1) * 8;
}

// interpret.cu: with d_bounds (level bounds, nlevels values) the max-error
// tables are formed in the kernel and d_errs is not read
template <class T>
int launch_interpret(int nfields, int kind, int est_kind, const int* d_ndims, const int* d_levels, double s, int B,
                     const uint32_t* d_sizes, uint64_t sz_stride, const double* d_errs, uint64_t err_stride,
                     const double* d_tols, double tol0, uint8_t* d_index, uint64_t idx_stride, uint32_t* d_rsz,
                     cudaStream_t st, bool pdl = false, bool early = false, const T* d_bounds = nullptr);

// one segment per (field, level) of the multi-level fp32 negabinary encode /
// decode launches; chunk_begin is the segment's first global chunk
struct ChunkSeg {
    const float* x;         // encode input
    float* y;               // decode output
    uint32_t* words;        // plane 0 of the level's streams
    uint64_t n, nblocks, stride;
    const uint32_t* key;
    const uint8_t* dnum;    // decode: retrieved plane count
    uint64_t chunk_begin;
};
// bitplane.cu: every level of one fp32 field decoded in one launch; segments
// chunked by kDecodeChunkBlocks blocks
constexpr int kDecodeChunkBlocks = 128;
int launch_nb_decode_levels(const ChunkSeg* segs, int nseg, uint64_t total_chunks, cudaStream_t st, bool pdl = false);
// bitplane.cu: every level of one fp32 field in one encode launch; with
// errs_out, per-level squared-error tables (partial: nseg * nb_encode_levels_grid(1)
// records of kErrRecWords words)
int nb_encode_levels_grid(int with_errors);
// the launch itself without error tables, over the segments of any number of fields
int launch_nb_encode_segments(const ChunkSeg* segs, int nseg, uint64_t total_chunks, int B, unsigned grid, cudaStream_t st,
                              bool pdl);
int launch_nb_encode_levels(const ChunkSeg* segs, int nseg, uint64_t total_chunks, int B, double* partial,
                            double* errs_out, cudaStream_t st);

// fused.cu
bool decode_recompose_nb32_ok(const Box& F);
int launch_decode_recompose_nb32(const void* base, uint64_t stride, int planes, uint64_t nblocks, const void* maxkey,
                                 const uint8_t* dnum, const float* coarse, const Box& F, const Box& C, float* out,
                                 uint64_t s0, uint64_t s1, int* status, cudaStream_t st, bool pdl = false);
void fused_tma_test_hook(int tx_extra, long long wait_cycles);
// one segment per field of the batched fused launch: the finest level of an
// fp32 negabinary field decoded and recomposed from its
// coarse box; unit_begin is the field's first global unit
struct FusedSeg {
    const uint32_t* base;   // plane 0 of the level's streams
    uint64_t stride;        // words per plane row
    const uint32_t* key;    // level |max| key
    const uint8_t* dnum;    // retrieved plane count
    const float* coarse;
    float* out;
    Box F, C;
    uint64_t s0, s1;
    uint64_t unit_begin;
    const void* map;        // the planes' tensor map (a CUtensorMap in device memory)
    uint32_t bw;            // the unit's block range plus alignment, in words
    uint32_t rpu;           // rows per unit: a multiple of 8, at most kMaxUnitRows; 4, 2 or 1 of long rows; or the
                            // warp-specialised form's
    uint32_t tall;          // 1 = the map's box is the tile's row stride x 32 plane rows
                            // (one copy per unit), 0 = bw words x 1 plane (one copy per plane)
};
constexpr uint32_t kMaxUnitRows = 64;
// box width of a level's tensor map for units of nr rows (0: rows too long),
// the map of one level's planes (CUtensorMap, 128 bytes, into `map`), the
// launch over segments whose maps live in device memory (64-byte aligned)
// rows per unit: a multiple of 8, about `values` values
uint32_t fused_unit_rows(const Box& F, uint32_t values);
uint32_t fused_unit_blocks_rows(const Box& F, uint32_t nr);      // tile blocks of nr rows
uint32_t fused_tma_box(const Box& F, uint32_t& nr);            // lowers nr until its box fits
int encode_plane_map(void* map, const void* base, uint64_t nblocks, int planes, uint64_t stride, uint32_t bw,
                     uint32_t box_planes = 1);
bool fused_tma_tall();                                            // PRODM_TMA_TALL (default 1)
// the warp-specialised batched kernel: units of fused_ws_unit_rows() rows,
// tall maps with boxes of kWsMultiStride words x 32 plane rows
constexpr uint32_t kWsMultiStride = 96;
uint32_t fused_ws_unit_rows();
int launch_decode_recompose_nb32_ws_multi(const FusedSeg* segs, int nseg, uint64_t total_units, uint32_t tld,
                                          int* status, cudaStream_t st);
uint32_t fused_tma_stride(uint32_t bw);                           // tile row stride of the TMA kernels for box bw
int launch_decode_recompose_nb32_tma_multi(const FusedSeg* segs, int nseg, uint64_t total_units, uint32_t tld,
                                           uint32_t max_bw, unsigned ctas_per_sm, int* status, cudaStream_t st);

// perbit.cu: per-bit format; rows of 32-element group words (magnitude
// planes 0..B-1, sign row B, unseen row B+1), each row `stride` words
uint64_t pb_groups(uint64_t n);
uint64_t pb_row_words(uint64_t n);
// one segment per level of a launch
template <class T>
struct PbSeg {
    const T* x;                           // encode input
    T* y;                                 // decode output
    const typename KeyOf<T>::type* key;   // level |max| key, or NULL and the exponent exp
    uint32_t* rows;
    uint64_t stride;
    uint32_t* counts;                     // encode: first-one counts, 64 words
    uint32_t* sizes;                      // encode: stream bytes, B
    const uint8_t* dnum;                  // decode: planes (overrides e), or NULL
    const uint32_t* srow;                 // decode: sign row
    const uint32_t* unseen;               // decode: elements without a 1 bit so far, or NULL (s == 0)
    uint64_t n;
    uint32_t chunk0;                      // set by the launchers
    int exp;
};
template <class T>
struct PbSet {
    int n;
    PbSeg<T> seg[17];
};
template <class T>
int launch_pb_encode(PbSet<T> set, int B, cudaStream_t st);
template <class T>
int launch_pb_decode(PbSet<T> set, int B, int s, int e, cudaStream_t st);
size_t pb_pack_scratch_bytes(uint64_t n, int B);
int launch_pb_pack(const uint32_t* rows, uint64_t stride, uint64_t n, int B, const uint32_t* sizes, uint64_t total,
                   uint8_t* dst, void* scratch, cudaStream_t st);
int launch_pb_init_unseen(uint32_t* unseen, uint32_t* signs, uint64_t n, cudaStream_t st);
// planes [a, a + planes.size()) of one level, read from the reference's streams
// (nwords 64-bit words each) into the level's rows; status: a device word, 0 or
// the PRODM_E* code of a failed parse
struct PbParseJob {
    std::vector<const uint64_t*> planes;
    std::vector<uint64_t> nwords;
    int a;
    uint64_t n;
    uint32_t* rows;
    uint64_t stride;
    uint32_t* unseen;
    uint32_t* signs;
    int* status;
};
// the same for the kernel: ring and flags of its planes, its first CTA
struct PbParse {
    const uint64_t* const* planes;
    const uint64_t* nwords;
    uint32_t* rows;
    uint64_t stride;
    uint32_t* unseen;
    uint32_t* signs;
    uint32_t* ring;
    int* flags;
    int* status;
    uint64_t n;
    int a, np, cta0;
};
constexpr int kPbParseLevels = 17;
struct PbParseSet {
    int n;
    PbParse seg[kPbParseLevels];
};
int launch_pb_parse(const std::vector<PbParseJob>& jobs, cudaStream_t st);

// lossless.cu: ZCB codec, one descriptor per stream; chunk0 = the stream's
// first chunk in the flattened chunk index (sorted), clen = compressed length
struct ZStream {
    const uint8_t* src;
    uint8_t* dst;
    uint64_t len;
    uint64_t clen;
    uint64_t chunk0;
};
uint64_t zcb_bound(uint64_t len);
int launch_zcb_count(const ZStream* d_ss, int ns, uint64_t total_chunks, uint32_t* csize, uint32_t* coff,
                     uint32_t* out_sizes, cudaStream_t st);
int launch_zcb_write(const ZStream* d_ss, int ns, uint64_t total_chunks, const uint32_t* csize, const uint32_t* coff,
                     cudaStream_t st);
int launch_zcb_read(const ZStream* d_ss, int ns, uint64_t total_chunks, int* status, cudaStream_t st);
int adaptive_stopping(const uint32_t* raw, const uint32_t* comp, int B, int latter, uint8_t* compressed);
// One stream of the stage: raw bytes src and stored bytes dst (store), or
// stored src and raw dst (expand); packed: the stored bytes are compressed
struct LlPart {
    const uint8_t* src;
    uint8_t* dst;
    uint64_t raw, stored;
    bool packed;
};
int ll_sizes(const std::vector<LlPart>& parts, uint32_t* h_comp, cudaStream_t st);   // every stream's compressed size
int ll_store(const std::vector<LlPart>& parts, cudaStream_t st);                     // stream ordered
int ll_raw_sizes(std::vector<LlPart>& parts, cudaStream_t st);                       // raw sizes of stored streams
int ll_expand(const std::vector<LlPart>& parts, cudaStream_t st);                    // waits: a malformed chunk is an error

// fileio.cu: byte ranges of a file into the handle's loader (sink(src,
// offset within the range, bytes, src_is_host)); *mode: 1 cuFile, 0 pinned
struct FileStaging;
void file_staging_free(FileStaging* s);
int file_staging_mode(const FileStaging* s);
int read_file_range(FileStaging*& fs, const char* path, uint64_t file_off, uint64_t bytes,
                    const std::function<int(const void*, uint64_t, uint64_t, int)>& sink, cudaStream_t st,
                    int* mode);

// pack.cu
int launch_gr_pack(const void* planes, uint64_t cap, const uint32_t* sizes, int B, uint64_t nblocks, const uint8_t* rbs,
                   int word_bytes, uint8_t* dst, cudaStream_t st);
// a table of the caller's frame to device memory (both 4-byte aligned, a multiple of 4 bytes)
int launch_put(void* dst, const void* src, size_t bytes, cudaStream_t st);
// planes of one level's streams (byte offset and words of each behind src) to aligned rows
struct UnpackSet {
    int n;
    uint64_t off[64], words[64];
    void* dst[64];
};
int launch_unpack_planes(const uint8_t* src, const UnpackSet& set, int word_bytes, void** table, cudaStream_t st);
template <class T>
int launch_maxabs(const T* x, uint64_t n, void* maxkey, cudaStream_t st);
template <class T>
int launch_bounds_from_keys(const void* keys, int nl, int negabinary, T* bounds, cudaStream_t st);
int launch_fill_u32(uint32_t* dst, uint64_t n, uint32_t v, cudaStream_t st);

}  // namespace prodm
