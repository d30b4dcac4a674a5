// Heap-tree Huffman codebook built on the host, for the stream-ordered host-build mode of
// vsz_compress (the library's tree thread answers k_tree_handoff between the histogram and the
// encoder).
//
// Same result as k_huff_build (huffman.cu): the reference's binary-heap priority queue replayed
// operation for operation (src/huffman.hh:169-192, 248-262; the first qremove() of a merge is the
// RIGHT child), preorder numbering of pad_tree_* (:374-423), codewords of build_code (:200-227),
// serialisation of convert_HuffTree_to_bytes_anyStates (:425-502).  The replay is a long chain of
// dependent, branchy memory operations on a few KB: one CPU core runs it several times faster than
// one GPU thread.
#include "host_tree.h"

#include <cstring>
#include <vector>

namespace vsz {

static inline uint32_t tree_width(uint32_t nc) { return nc <= 256 ? 1u : (nc <= 65536 ? 2u : 4u); }

size_t host_tree_bytes(uint32_t nc) {
    const size_t w = tree_width(nc);
    return 1 + 2 * w * nc + 4 * (size_t)nc + nc;
}

int host_huffman_build(const uint64_t* hist, int dict, uint64_t* cb_word, uint8_t* cb_len, uint32_t* info,
                       uint8_t* head, int hdr_dict) {
    std::vector<uint32_t> used;
    used.reserve((size_t)dict);
    for (int s = 0; s < dict; s++)
        if (hist[s]) used.push_back((uint32_t)s);
    const int nused = (int)used.size();
    std::memset(cb_word, 0, sizeof(uint64_t) * (size_t)dict);
    std::memset(cb_len, 0, (size_t)dict);
    info[0] = info[1] = info[2] = info[3] = 0u;
    if (nused == 0) return 1;  // the reference dereferences a null root here
    // children of internal nodes (creation order); the heap holds (freq, node) pairs so that its
    // comparisons read the entries themselves.  The operations and their order are the
    // reference's (qinsert huffman.hh:169, qremove :179), so ties resolve the same way.
    struct HeapEnt {
        uint64_t f;
        int32_t n;
    };
    std::vector<int32_t> lch((size_t)nused), rch((size_t)nused);
    // 1-based; entry 0 (frequency 0) stops qinsert at the root.  A removal reads up to entry 2 i + 1 for
    // a hole i <= nused, so 2 nused + 2 entries (value-initialised) cover every read.
    std::vector<HeapEnt> heap_v(2 * (size_t)nused + 8);
    HeapEnt* const heap = heap_v.data();
    auto qinsert = [&](uint32_t i, uint64_t fn, int n) {
        uint32_t j;
        while (heap[j = i >> 1].f > fn) {
            heap[i] = heap[j];
            i       = j;
        }
        heap[i] = HeapEnt{fn, n};
    };
    // qremove: the hole always sinks to the bottom (no early exit), moving up the smaller child, the
    // left one on a tie, and then takes the last element.  Its way down doesn't depend on that element,
    // so the two removals of a merge go down in one loop, the second two levels behind the first (it
    // reads level d + 1 when that has its final values): two chains of loads and selects in flight
    // (Grace, 1024 symbols: 58 -> 39 us, 300: 11 as before).
    auto sink = [&](uint32_t& i) {
        const uint32_t c = 2u * i + (uint32_t)(heap[2u * i + 1u].f < heap[2u * i].f);
        heap[i]          = heap[c];
        i                = c;
    };
    auto sink_last = [&](uint32_t& i, uint32_t end) {  // `end`: first index that is not an element
        const uint32_t l = 2u * i;
        if (l < end) {
            const uint32_t c = l + (uint32_t)((l + 1u < end) & (heap[l + 1u].f < heap[l].f));
            heap[i]          = heap[c];
            i                = c;
        }
    };
    for (int i = 0; i < nused; i++) qinsert((uint32_t)i + 1u, hist[used[i]], i);
    int nnodes = nused;
    for (uint32_t q1 = (uint32_t)nused; q1 > 1; q1--) {  // q1: the last element; q2: the one before
        const uint32_t q2  = q1 - 1u;
        const HeapEnt top1 = heap[1];
        HeapEnt top2;
        uint32_t i1 = 1, i2 = 1;
        if (q2 >= 8u) {
            // levels 0 .. full - 1 have both children below q2, the next has some, then there are none
            const int full = 30 - __builtin_clz(q2);
            sink(i1);
            top2 = heap[1];
            sink(i1);
            for (int s = 2; s < full; s++) {
                sink(i1);
                sink(i2);
            }
            sink_last(i1, q1);
            heap[i1] = heap[q1];
            sink(i2);
            sink(i2);
            sink_last(i2, q2);
        } else {
            while (2u * i1 < q1) sink_last(i1, q1);
            heap[i1] = heap[q1];
            top2     = heap[1];
            while (2u * i2 < q2) sink_last(i2, q2);
        }
        heap[i2]       = heap[q2];
        const int v    = nnodes++;
        lch[v - nused] = top2.n;
        rch[v - nused] = top1.n;
        qinsert(q2, top1.f + top2.f, v);
    }
    // subtree sizes bottom-up, then preorder index / codeword / depth top-down
    const int nint = nnodes - nused;
    std::vector<uint32_t> size((size_t)nnodes, 1u), pre((size_t)nnodes, 0u), depth((size_t)nnodes, 0u);
    std::vector<uint64_t> code((size_t)nnodes, 0ull);
    for (int k = 0; k < nint; k++) size[nused + k] = 1u + size[lch[k]] + size[rch[k]];
    uint32_t max_len = 0;
    for (int k = nint - 1; k >= 0; k--) {
        const int v = nused + k, l = lch[k], r = rch[k];
        pre[l]   = pre[v] + 1u;
        pre[r]   = pre[v] + 1u + size[l];
        code[l]  = code[v] << 1;
        code[r]  = (code[v] << 1) | 1ull;
        depth[l] = depth[r] = depth[v] + 1u;
        if (depth[l] > max_len) max_len = depth[l];
    }
    const uint32_t nc = (uint32_t)nnodes;
    // [BE nodeCount][BE dict][u8 0][L][R][C u32 LE][t]
    const uint32_t w = tree_width(nc);
    head[0] = (uint8_t)(nc >> 24);
    head[1] = (uint8_t)(nc >> 16);
    head[2] = (uint8_t)(nc >> 8);
    head[3] = (uint8_t)nc;
    const uint32_t dh = (uint32_t)(hdr_dict ? hdr_dict : dict);
    head[4] = (uint8_t)(dh >> 24);
    head[5] = (uint8_t)(dh >> 16);
    head[6] = (uint8_t)(dh >> 8);
    head[7] = (uint8_t)dh;
    head[8] = 0;
    uint8_t* pL = head + 9;
    uint8_t* pR = pL + (size_t)w * nc;
    uint8_t* pC = pR + (size_t)w * nc;
    uint8_t* pT = pC + 4 * (size_t)nc;
    std::memset(pL, 0, 2 * (size_t)w * nc);
    for (int v = 0; v < nnodes; v++) {
        const uint32_t idx = pre[v];
        uint32_t c = 0, lv = 0, rv = 0;
        const bool leaf = v < nused;
        if (leaf) {
            c          = used[v];
            cb_len[c]  = (uint8_t)(depth[v] > 255u ? 255u : depth[v]);
            cb_word[c] = code[v];
        } else {
            lv = pre[lch[v - nused]];
            rv = pre[rch[v - nused]];
        }
        for (uint32_t b = 0; b < w; b++) {
            pL[(size_t)idx * w + b] = (uint8_t)(lv >> (8 * b));
            pR[(size_t)idx * w + b] = (uint8_t)(rv >> (8 * b));
        }
        std::memcpy(pC + 4 * (size_t)idx, &c, 4);
        pT[idx] = leaf ? 1 : 0;
    }
    info[0] = nc;
    info[1] = (uint32_t)host_tree_bytes(nc);
    info[2] = max_len;
    info[3] = nc;
    return 0;
}

}  // namespace vsz
