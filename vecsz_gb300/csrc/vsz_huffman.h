// Internal interface of the Huffman kernels (huffman.cu).
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "vsz_kernels.h"
#include "vsz_types.h"

namespace vsz {

constexpr int kDecBits     = 12;   // primary decode table: 4096 entries
constexpr int kDec2Max     = 8;    // widest secondary table: codewords of up to 20 bits in two lookups

// Decode table entries (k_huff_table).  Primary table, indexed by the next kDecBits bits:
//   (sym << 8) | len           len in 1..kDecBits: a whole codeword
//   (off << 12) | (w2 << 8) | 0x80   a longer codeword: index table2[off + next w2 bits]
//   (node << 8)                walk the tree bit by bit from `node` after kDecBits bits
// Secondary table2 entries: (sym << 8) | total length, or (node << 8) to walk from `node` after
// kDecBits + w2 bits (codewords longer than kDecBits + kDec2Max).  A zero entry is not a codeword.
// Capacity: every secondary table hangs off a distinct internal node at depth kDecBits, and one
// with L leaves below it is at most 2^min(kDec2Max, L - 1) entries wide (a subtree of depth D has
// at least D + 1 leaves), so a tree of `leaves` leaves needs at most 256 / 9 entries per leaf.
// k_huff_table leaves the walk entries in place of secondary tables that would not fit.
__host__ __device__ inline size_t table2_capacity(uint32_t max_nodes) {
    const size_t leaves = ((size_t)max_nodes + 1) / 2;
    return ((size_t)(1u << kDec2Max) * leaves + 8) / 9 + 256;
}
// The split decoder's tables in shared memory: a primary table one bit wider and the first
// entries of the secondary one (a 1024-symbol tree of a smooth field has 2.5-4.3 K of them).
constexpr int kWinBits     = 13;
constexpr int kDec2Smem    = 3072;
constexpr size_t kWinImageWords = ((size_t)1 << kWinBits) + kDec2Smem;
// Whether a stream takes the split decoder (k_huff_decode_split) or a lane per chunk (k_huff_decode_win).
// The window decoder's time is one lane's chain whatever the number of chunks: 60 us where every codeword
// has at most kDecBits bits, 80-160 at 6-9 bits a code, 150-400 with trees of 8K nodes and more.  The split
// decoder runs in rounds of CTAs (9728 chunks of 16 lanes fill 152 SMs), each 25-45 us where its
// tables hold the codewords and a warp's words fit its buffer (kSpanBits bits a code), 100-400 where not.
// Decode of a field, window -> split, us:
//   one round: 8000 chunks, 7 bits 98 -> 34; 13.7 bits, 118K nodes 325 -> 228; but 16 bits 190 -> 354 (512: 205 -> 160)
//   two: 15.6 K chunks, 6.3 bits 132 -> 87, 8 bits, 7.8K nodes 229 -> 160; uniform residuals, 8 bits 76 -> 82; 12 bits
//     100 -> 194; 12.7 K chunks, 2.6 bits 87 -> 93
//   three: 29.3 K chunks, 6.3 bits 159 -> 138, 9 bits 108 -> 95; 5.4 bits 67 -> 72; 8 bits, 7.8K nodes (27 K) 203 -> 243
//   32.8 K chunks: 6.5 bits 126 -> 147, 9 bits 92 -> 99
// So: one round always, unless nearly no codeword is in the tables; two where codewords are of many lengths
// (0.4 bits below the fixed length for as many leaves) and fit both tables and buffer; three at 6 bits or
// more with trees whose long codewords are in the image.
constexpr size_t kSplitChunks = size_t(1) << 13, kSplitTwoRounds = 19456, kSplitMaxChunks = 30000;
inline bool huff_split_applies(size_t nchunks, unsigned long long payload_bits, uint32_t nodes) {
    const double bits = (double)payload_bits / ((double)nchunks * 512.0);
    if (nchunks <= kSplitChunks) return bits <= 14.0 || nchunks <= 1024;
    if (bits < 4.0 || bits > 9.5 || nodes > 8192u || bits > std::log2((nodes + 1u) / 2.0) - 0.4) return false;
    return nchunks <= kSplitTwoRounds || (nchunks <= kSplitMaxChunks && bits >= 6.0 && nodes <= 5000u);
}
// The same for a batch (k_huff_decode_split_batch), by its chunks and its largest tree.  A task is 64 chunks
// of one field there, two rounds of one CTA, so one field past the image costs the batch what it costs a
// large field: largest tree 2.2K nodes 90 -> 53 us, 3.8K 158 -> 164, 5.0K 187 -> 319, 8.1K 182 -> 330.
constexpr uint32_t kSplitBatchNodes = 3072;
inline bool huff_split_batch(size_t total_chunks, uint32_t most_nodes) {
    return total_chunks <= kSplitChunks && most_nodes <= kSplitBatchNodes;
}
constexpr int kChunkSyms   = 512;  // codewords per entry of this library's decode index
constexpr int kSyncBits    = 8192; // chunk size (bits) of the self-synchronising decoder

// Width of the serialized child indices (src/huffman.hh:425-502).
__host__ __device__ inline int tree_index_width(uint32_t nc) { return nc <= 256 ? 1 : (nc <= 65536 ? 2 : 4); }
// [u8 endian][L][R][C u32][t u8]
__host__ __device__ inline size_t tree_bytes_size(uint32_t nc) {
    int w = tree_index_width(nc);
    return 1 + 2 * (size_t)w * nc + 4 * (size_t)nc + nc;
}

struct HuffBuildArgs {
    const unsigned long long* hist;
    int dict;                     // symbols [0, dict) (a 1D padded field adds one: 2 * radius)
    int hdr_dict;                 // dictionary size written into the head; 0: dict
    unsigned long long* cb_word;  // right-aligned codeword per symbol
    uint8_t* cb_len;              // codeword length per symbol (0 = unused)
    uint8_t* out;                 // [BE nc][BE dict][tree bytes], any alignment
    uint32_t* info;               // [0] node count [1] tree bytes [2] max code length [3] nodes created
    void* scratch;                // huff_build_scratch_bytes(dict), used when shared memory is too small
    int ws_in_smem;
    int* status;
};

struct HuffEncodeArgs {
    const uint16_t* codes;
    size_t n;
    const unsigned long long* cb_word;
    const uint8_t* cb_len;
    int dict;
    uint8_t* out;                     // payload start = out + out_off.eval(), any alignment;
    DevOffset out_off;                // bytes before the payload start are kept
    unsigned long long* total_bits;
    uint16_t* chunk_bits;             // nchunks: bits per 512 codes (scan input; the decode index)
    unsigned long long* chunk_off;    // nchunks: first bit of each chunk
    unsigned long long* scan_status;  // scan scratch: scan_tmp_tiles(nchunks) + 1
    uint32_t* scan_counter;
    int scan_cleared;                 // scan_status and scan_counter are zero already
    unsigned long long* edge_idx;     // 2 nchunks: word index of a chunk's partial first / last word
    uint32_t* edge_bits;              // 2 nchunks: its bits (stored byte order)
    int* status;
    size_t nchunks;
    int codes_aligned;
    int cb_in_smem;
    const uint32_t* build_info;       // optional: the tree's info; max length > 64 is refused
};

struct HuffTableArgs {
    const uint8_t* huff;  // [BE nc][BE dict][tree bytes]...
    size_t huff_bytes;
    int dict;
    uint32_t max_nodes;
    uint32_t* table;      // 1 << kDecBits entries
    uint32_t* child;      // 2 * max_nodes
    uint32_t* node_sym;   // max_nodes: 0x80000000 | symbol for leaves
    uint32_t* parent;     // max_nodes (scratch)
    uint32_t* walk;       // max_nodes: both children of an internal node, 16 bits each:
                          // 0x8000 | symbol for a leaf, else the node index (dict <= 16384)
    uint32_t* table2;     // table2_capacity(max_nodes) secondary entries
    uint32_t* win;        // kWinImageWords, 16-byte aligned: the split decoder's tables, or null (always for
                          // one-node trees)
    uint32_t* info;       // [0] single-symbol tree flag [1] its symbol [2] longest codeword (255: > 64)
                          // [3] entries of table2
    int* status;
};

struct HuffDecodeArgs {
    const uint8_t* payload;  // any alignment; 8 readable bytes past the end are required
    unsigned long long payload_bits;
    const uint32_t* table;
    const uint32_t* table2;
    const uint32_t* child;
    const uint32_t* node_sym;
    const uint32_t* walk;                 // packed children (k_huff_table), when walk_smem
    int walk_smem;                        // 1: dict <= 16384, the walk array is copied to shared memory
    uint32_t nodes;                       // node count of the tree
    const unsigned long long* start_bit;  // per chunk, relative to start_bit[0] (indexed path)
    const uint16_t* chunk_len;            // indexed path: bits of each chunk
    uint32_t* chunk_zero;                 // indexed path: zero codes per chunk (may be null)
    const unsigned long long* out_begin;  // per chunk, or null: chunk * chunk_syms
    const uint32_t* nsym;                 // per chunk, or null: chunk_syms
    size_t nchunks;
    uint32_t chunk_syms;
    uint16_t* codes;
    size_t n;
    uint32_t max_nodes;                   // node indices past this are a corrupt tree
    const uint32_t* win;                  // k_huff_table's image for the split decoder, or null
    const uint32_t* tree_info;            // k_huff_table's info ([2] longest codeword), or null
    int* status;
};

struct HuffSyncArgs {
    const uint8_t* payload;
    unsigned long long payload_bits;
    const uint32_t* table;
    const uint32_t* table2;
    const uint32_t* child;
    const uint32_t* node_sym;
    size_t nchunks;
    uint32_t chunk_bits;
    unsigned long long* start;   // nchunks
    unsigned long long* exit_a;  // nchunks
    uint32_t* count;             // nchunks
    uint32_t max_nodes;
    int* status;
};

int launch_huff_build(HuffBuildArgs a, cudaStream_t st);
// Batches: one CTA per field; in_smem for every field when huff_build_in_smem(dict) (the others
// need HuffBuildArgs::scratch).  Encode: tasks of (field, 512-code chunk range); all fields' chunk
// bits are scanned at once (all_bits / all_off hold total_chunks + 1 entries, the fields' ranges
// in field order; each field's chunk_bits / chunk_off point into them).
bool huff_build_in_smem(int dict);
int launch_huff_build_batch(const HuffBuildArgs* args, uint32_t nfields, bool in_smem, int dict_max, cudaStream_t st,
                            int num_sms);
int launch_huff_encode_batch(const HuffEncodeArgs* args, uint32_t nfields, const BatchTask* tasks, uint32_t ntasks,
                             int cb_dict_max, uint16_t* all_bits, unsigned long long* all_off, size_t total_chunks,
                             unsigned long long* scan_status, uint32_t* scan_counter, int* batch_status,
                             cudaStream_t st, int num_sms);
void huff_encode_prepare(HuffEncodeArgs& a);
void huff_build_prepare();  // one-time kernel attributes of launch_huff_build (call outside capture)
size_t huff_build_scratch_bytes(int dict);  // also the shared memory of a build there
int launch_huff_encode(HuffEncodeArgs a, cudaStream_t st, int num_sms);
int launch_huff_table(HuffTableArgs a, cudaStream_t st);
// Many fields: decode tables one CTA per field; decoding over tasks of (field, range of the field's
// index), split (huff_split_batch): all by the split decoder, else 256 chunks each, every field's tree by the
// decoder of its kind (the window decoder for codewords up to 32 bits, the general one beyond); const_tasks
// (one-symbol trees) by a constant fill.
// most_nodes: the largest tree's.
int launch_huff_table_batch(const HuffTableArgs* args, uint32_t nfields, cudaStream_t st, int num_sms);
int launch_huff_decode_batch(const HuffDecodeArgs* args, const BatchTask* tasks, uint32_t ntasks,
                             const BatchTask* const_tasks, uint32_t nconst, bool split, uint32_t most_nodes,
                             cudaStream_t st, int num_sms);
int launch_huff_decode(HuffDecodeArgs a, cudaStream_t st, int num_sms);
int launch_huff_const(uint16_t* codes, size_t n, const uint32_t* info, const int* status, cudaStream_t st, int num_sms);
int launch_huff_sync_init(HuffSyncArgs a, cudaStream_t st);
int launch_huff_sync_round(HuffSyncArgs a, const unsigned long long* exit_in, unsigned long long* exit_out,
                           int* changed, cudaStream_t st);
// cleared: tile_status and tile_counter are zero already.
int launch_scan_u16(const uint16_t* in, unsigned long long* out, size_t n, unsigned long long* tile_status,
                    uint32_t* tile_counter, unsigned long long* total, int* status, cudaStream_t st,
                    bool cleared = false);
int launch_scan_u32(const uint32_t* in, unsigned long long* out, size_t n, unsigned long long* tile_status,
                    uint32_t* tile_counter, unsigned long long* total, int* status, cudaStream_t st,
                    bool cleared = false);
// The decode tables and the exclusive scan of the decode index (tile_status, tile_counter zero).
int launch_huff_table_scan(HuffTableArgs a, const uint16_t* bits, unsigned long long* start, size_t n,
                           unsigned long long* tile_status, uint32_t* tile_counter, cudaStream_t st);
size_t scan_tmp_tiles(size_t n);
// Test hooks (vsz_debug_*): this unit's look-back spin limit; a scan whose first tile never runs.
int set_spin_limit_huffman(long long polls);
int debug_scan_stalled(size_t n, int* status_out);

}  // namespace vsz
