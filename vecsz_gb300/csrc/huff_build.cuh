// Tree build of one field by one CTA (k_huff_build, and k_dq_compress_batch for the fields of a batch).
#pragma once

#include <cstdint>

#include "scan.cuh"
#include "vsz_device.cuh"
#include "vsz_huffman.h"

namespace vsz {

// ------------------------------------------------------------------------------------------
// K2: heap-tree build
// ------------------------------------------------------------------------------------------

constexpr int kKeyShift = 20;  // heap key = freq << 20 | node  (node < 2^20, freq < 2^44)
constexpr uint32_t kNodeMask = (1u << kKeyShift) - 1u;

// Working set of the tree build (shared memory when it fits, else the global scratch).
struct BuildWs {
    unsigned long long* heap;  // 2 dict + 8 (room for speculative reads below the heap end)
    uint32_t* used;            // dict: symbol of leaf i
    int32_t* lchild;           // dict: children of internal node k (node nused + k)
    int32_t* rchild;
    uint32_t* size;            // 2 dict: subtree sizes
    uint32_t* pre;             // 2 dict: preorder index (pad_tree_* numbering)
    unsigned long long* code;  // 2 dict: codeword, right-aligned
    uint32_t* depth;           // 2 dict
};

__host__ __device__ inline size_t build_ws_bytes(int dict) {
    size_t d = (size_t)dict;
    return 8 * (2 * d + 8) + 4 * d + 8 * d + 4 * 2 * d * 2 + 8 * 2 * d + 4 * 2 * d + 256;
}

__device__ inline BuildWs carve_build_ws(uint8_t* p, int dict) {
    size_t d = (size_t)dict;
    BuildWs w;
    w.heap   = reinterpret_cast<unsigned long long*>(p);
    p += 8 * (2 * d + 8);
    w.code   = reinterpret_cast<unsigned long long*>(p);
    p += 8 * 2 * d;
    w.used   = reinterpret_cast<uint32_t*>(p);
    p += 4 * d;
    w.lchild = reinterpret_cast<int32_t*>(p);
    p += 4 * d;
    w.rchild = reinterpret_cast<int32_t*>(p);
    p += 4 * d;
    w.size   = reinterpret_cast<uint32_t*>(p);
    p += 4 * 2 * d;
    w.pre    = reinterpret_cast<uint32_t*>(p);
    p += 4 * 2 * d;
    w.depth  = reinterpret_cast<uint32_t*>(p);
    return w;
}

// Heap key layouts: freq in the high bits, node in the low bits.  K32: 32 | 32 (histogram total
// below 2^32, the usual case: the frequency is the high register, one 32-bit compare); otherwise
// 44 | 20.  Only the frequency part is ever compared, as in the reference.
template <bool K32>
struct HeapKey {
    static __device__ __forceinline__ unsigned long long fq(unsigned long long k) {
        return K32 ? (unsigned long long)(uint32_t)(k >> 32) : (k >> kKeyShift);
    }
    static __device__ __forceinline__ unsigned long long make(unsigned long long f, uint32_t node) {
        return K32 ? ((f << 32) | node) : ((f << kKeyShift) | node);
    }
    static __device__ __forceinline__ uint32_t node(unsigned long long k) {
        return K32 ? (uint32_t)k : (uint32_t)(k & kNodeMask);
    }
};

// The heap array by address: entry i is at base + 8 i, its children's pair at 2 (base + 8 i) - base.
// In shared memory the addresses are 32 bits.
template <bool IN_SMEM>
struct HeapMem {
    using Addr = uintptr_t;
    static __device__ __forceinline__ Addr addr(unsigned long long* p) { return reinterpret_cast<Addr>(p); }
    static __device__ __forceinline__ unsigned long long load(Addr a) { return *reinterpret_cast<unsigned long long*>(a); }
    static __device__ __forceinline__ ulonglong2 load2(Addr a) { return *reinterpret_cast<ulonglong2*>(a); }
    static __device__ __forceinline__ void store(Addr a, unsigned long long v) {
        *reinterpret_cast<unsigned long long*>(a) = v;
    }
};
template <>
struct HeapMem<true> {
    using Addr = uint32_t;
    static __device__ __forceinline__ Addr addr(unsigned long long* p) {
        return static_cast<uint32_t>(__cvta_generic_to_shared(p));
    }
    static __device__ __forceinline__ unsigned long long load(Addr a) {
        unsigned long long v;
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
        return v;
    }
    static __device__ __forceinline__ ulonglong2 load2(Addr a) {
        ulonglong2 v;
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
        return v;
    }
    static __device__ __forceinline__ void store(Addr a, unsigned long long v) {
        asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
    }
};

// A removal's hole: its address and its children's pair's.
template <bool IN_SMEM>
struct Hole {
    typename HeapMem<IN_SMEM>::Addr a, kids;
};

// The hole takes the smaller of its children c (ties: the left) and moves there.
template <bool K32, bool IN_SMEM>
__device__ __forceinline__ void heap_sink(Hole<IN_SMEM>& h, typename HeapMem<IN_SMEM>::Addr base, const ulonglong2 c) {
    using K           = HeapKey<K32>;
    const auto grands = 2 * h.kids - base;  // the left child's children
    if constexpr (K32 && IN_SMEM) {
        const uint32_t fx = (uint32_t)(c.x >> 32), fy = (uint32_t)(c.y >> 32);
        const uint32_t to = h.a;
        h.a               = h.kids;
        h.kids            = grands;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.lt.u32 p, %3, %4;\n\t"
            "@p add.u32 %1, %1, 16;\n\t"
            "@p add.u32 %0, %0, 8;\n\t"
            "@p st.shared.u64 [%2], %5;\n\t"
            "@!p st.shared.u64 [%2], %6;\n\t}"
            : "+r"(h.a), "+r"(h.kids)
            : "r"(to), "r"(fy), "r"(fx), "l"(c.y), "l"(c.x)
            : "memory");
    } else {
        const bool right = K::fq(c.y) < K::fq(c.x);
        HeapMem<IN_SMEM>::store(h.a, right ? c.y : c.x);
        h.a    = h.kids + (right ? 8 : 0);
        h.kids = grands + (right ? 16 : 0);
    }
}

// The last step: the hole takes a child if it has one (`end` is the address after the last element's),
// then it takes `last`.  Returns where that went.
template <bool K32, bool IN_SMEM>
__device__ __forceinline__ typename HeapMem<IN_SMEM>::Addr heap_settle(const Hole<IN_SMEM>& h,
                                                                       typename HeapMem<IN_SMEM>::Addr end,
                                                                       const ulonglong2 c, unsigned long long last) {
    using K          = HeapKey<K32>;
    const bool has   = h.kids < end;
    const bool right = (h.kids + 8 < end) & (K::fq(c.y) < K::fq(c.x));
    const auto to    = has ? h.kids + (right ? 8 : 0) : h.a;
    HeapMem<IN_SMEM>::store(h.a, has ? (right ? c.y : c.x) : last);
    HeapMem<IN_SMEM>::store(to, last);
    return to;
}

// qinsert (src/huffman.hh:169-180) of `key` at the end `ii`.  Entry 0 = 0 stops it at the root.
template <bool K32, bool IN_SMEM>
__device__ __forceinline__ void heap_insert(typename HeapMem<IN_SMEM>::Addr base, uint32_t ii, unsigned long long key) {
    using K                     = HeapKey<K32>;
    using M                     = HeapMem<IN_SMEM>;
    const unsigned long long fk = K::fq(key);
    auto pos                    = base + 8 * ii;
    for (;;) {
        const auto up              = base + 8 * (ii >>= 1);
        const unsigned long long v = M::load(up);
        if (K::fq(v) <= fk) break;
        M::store(pos, v);
        pos = up;
    }
    M::store(pos, key);
}

// The reference's heap, operation for operation (src/huffman.hh:169-192, 248-262), by one thread.
// qremove: the hole sinks along the smaller child (ties: left) to the bottom, then takes the last
// element, without sifting it up; so its way down doesn't depend on that element, and the two
// removals of a merge go down together, the second two levels behind the first (it reads a level when
// that has its final values).  The time is that of one thread's dependent instructions, about 800
// cycles a merge: levels unrolled, addresses and not indexes carried along, no branch for the last
// level.  60 fields of up to 1024 symbols, slowest tree: 0.45 ms; slower were one removal after the
// other with loads a level ahead (0.64), three levels a step with their 14 frequencies loaded together
// (0.74), a warp taking five levels a step by ballots (0.98), two lanes with a removal each (1.39).
template <bool K32, bool IN_SMEM>
struct HeapReplay {
    using K    = HeapKey<K32>;
    using M    = HeapMem<IN_SMEM>;
    using Addr = typename M::Addr;
    Addr base;
    uint32_t q1;  // the last element
    int nnodes;
    int32_t *rc, *lc;

    // new_node(.., qremove(), qremove()) -- the first removal is the RIGHT child -- and its qinsert
    __device__ __forceinline__ void join(unsigned long long top1, unsigned long long top2) {
        *rc++ = (int32_t)K::node(top1);
        *lc++ = (int32_t)K::node(top2);
        heap_insert<K32, IN_SMEM>(base, q1 - 1u, K::make(K::fq(top1) + K::fq(top2), (uint32_t)nnodes));
        nnodes++;
        q1--;
    }

    // Merges while a hole of the second removal has two children on `full` levels from the root
    // (q1 - 1 >= 2 << full), full >= 2; a constant for LEVELS > 0.
    template <int LEVELS>
    __device__ __forceinline__ void merges(int levels) {
        const int full       = LEVELS > 0 ? LEVELS : levels;
        const uint32_t least = 2u << full;  // of q1 - 1
        while (q1 > least) {
            const Addr aq1 = base + 8 * q1, aq2 = aq1 - 8;
            Hole<IN_SMEM> h1{base + 8, base + 16}, h2 = h1;
            const unsigned long long top1 = M::load(base + 8), last1 = M::load(aq1), old2 = M::load(aq2);
            // levels 0 .. full - 1 have both children below q1 - 1, the next has some, then there are none
            const ulonglong2 c23 = M::load2(base + 16), c45 = M::load2(base + 32), c67 = M::load2(base + 48);
            const bool right     = K::fq(c23.y) < K::fq(c23.x);
            const unsigned long long top2 = right ? c23.y : c23.x;
            heap_sink<K32, IN_SMEM>(h1, base, c23);
            heap_sink<K32, IN_SMEM>(h1, base, right ? c67 : c45);
#pragma unroll
            for (int s = 2; s < full; s++) {
                const ulonglong2 c1 = M::load2(h1.kids), c2 = M::load2(h2.kids);
                heap_sink<K32, IN_SMEM>(h1, base, c1);
                heap_sink<K32, IN_SMEM>(h2, base, c2);
            }
            const ulonglong2 c1 = M::load2(h1.kids), c2 = M::load2(h2.kids);
            const Addr to1 = heap_settle<K32, IN_SMEM>(h1, aq1, c1, last1);
            heap_sink<K32, IN_SMEM>(h2, base, c2);
            heap_sink<K32, IN_SMEM>(h2, base, M::load2(h2.kids));
            heap_settle<K32, IN_SMEM>(h2, aq2, M::load2(h2.kids), to1 == aq2 ? last1 : old2);
            join(top1, top2);
        }
    }

    __device__ __forceinline__ unsigned long long remove(uint32_t q) {  // q: the last element
        const unsigned long long top = M::load(base + 8), last = M::load(base + 8 * q);
        uint32_t i = 1;
        for (uint32_t l = 2; l < q; l = 2 * i) {
            const unsigned long long x = M::load(base + 8 * l), y = M::load(base + 8 * l + 8);
            const bool right = l + 1 < q && K::fq(y) < K::fq(x);
            M::store(base + 8 * i, right ? y : x);
            i = l + (right ? 1u : 0u);
        }
        M::store(base + 8 * i, last);
        return top;
    }

    // Returns the number of nodes created.
    __device__ __forceinline__ int run(const BuildWs& w, int nused) {
        base   = M::addr(w.heap);
        rc     = w.rchild;
        lc     = w.lchild;
        nnodes = nused;
        q1     = (uint32_t)nused;
        // leaves: qinsert(new_node(freq, i)) in symbol order
        unsigned long long f = w.code[0];
        for (int i = 0; i < nused; i++) {
            const unsigned long long key = K::make(f, (uint32_t)i);
            f                            = w.code[i + 1];  // w.code has twice the entries
            heap_insert<K32, IN_SMEM>(base, (uint32_t)i + 1u, key);
        }
        for (int full = 30 - __clz(nused); full > 9; full--) merges<0>(full);
        merges<9>(0);
        merges<8>(0);
        merges<7>(0);
        merges<6>(0);
        merges<5>(0);
        merges<4>(0);
        merges<3>(0);
        merges<2>(0);
        while (q1 > 1u) {
            const unsigned long long top1 = remove(q1), top2 = remove(q1 - 1u);
            join(top1, top2);
        }
        return nnodes;
    }
};

template <bool IN_SMEM>
__device__ __forceinline__ void build_field(const HuffBuildArgs& a, uint8_t* s_build_dyn) {
    __shared__ uint32_t s_info[4];
    __shared__ int s_fail;
    __shared__ uint32_t s_scan[33];
    __shared__ unsigned long long s_fsum[8];
    if (*a.status != VSZ_OK) return;  // an earlier stage failed (uniform: one CTA)
    const int dict = a.dict;
    uint8_t* ws    = s_build_dyn;
    // pairs of heap entries are 16 bytes; build_ws_bytes has 256 to spare
    if (!IN_SMEM) ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(a.scratch) + 15u) & ~(uintptr_t)15);
    BuildWs w      = carve_build_ws(ws, dict);
    if (threadIdx.x == 0) s_fail = 0;
    for (int i = threadIdx.x; i < 2 * dict + 8; i += blockDim.x) w.heap[i] = 0ull;
    for (int i = threadIdx.x; i < dict; i += blockDim.x) {
        a.cb_word[i] = 0ull;
        a.cb_len[i]  = 0;
    }
    // ---- used symbols in symbol order (src/huffman.hh:248-254), block-wide compaction
    const int per = (dict + blockDim.x - 1) / blockDim.x;
    const int s0  = threadIdx.x * per;
    uint32_t cnt  = 0;
    unsigned long long fsum = 0;
    for (int k = 0; k < per; k++) {
        int sym = s0 + k;
        if (sym < dict) {
            unsigned long long f = __ldcg(&a.hist[sym]);  // other CTAs' atomics
            cnt += (f != 0ull);
            fsum += f;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
    if ((threadIdx.x & 31) == 0) s_fsum[threadIdx.x >> 5] = fsum;
    uint32_t tot;
    uint32_t off = block_exclusive_scan<uint32_t>(cnt, s_scan, &tot);
    for (int k = 0; k < per; k++) {
        int sym = s0 + k;
        if (sym < dict) {
            unsigned long long f = __ldcg(&a.hist[sym]);  // other CTAs' atomics
            if (f != 0ull) {
                w.used[off]   = (uint32_t)sym;
                w.code[off++] = f;  // leaf frequencies, until the codewords are computed
            }
        }
    }
    __syncthreads();
    const int nused = (int)tot;

    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) total += s_fsum[i];
        int nnodes = nused, fail = 0;
        if (nused == 0) fail = VSZ_ERR_INVALID;
        else if (total >= (1ull << (64 - kKeyShift))) fail = VSZ_ERR_UNSUPPORTED;
        else if (total < (1ull << 32)) nnodes = HeapReplay<true, IN_SMEM>{}.run(w, nused);
        else nnodes = HeapReplay<false, IN_SMEM>{}.run(w, nused);
        const uint32_t node_count = fail ? 0u : (uint32_t)nnodes;
        s_fail    = fail;
        s_info[0] = node_count;
        s_info[1] = (uint32_t)tree_bytes_size(node_count);
        s_info[2] = 0u;
        s_info[3] = (uint32_t)nnodes;
    }
    __syncthreads();
    if (!s_fail) {
        // every node on its own, by the way up to the root (the last node created; a one-leaf tree:
        // the leaf): subtree sizes, then the preorder index of pad_tree_* (src/huffman.hh:374-423) and
        // the codeword of build_code (:200-227)
        const int nn = (int)s_info[0], root = nn - 1;
        uint32_t* parent = reinterpret_cast<uint32_t*>(w.heap);  // parent << 1 | right; the heap is done with
        for (int v = threadIdx.x; v < nn; v += blockDim.x) w.size[v] = 0u;
        for (int k = threadIdx.x; k < nn - nused; k += blockDim.x) {
            parent[w.lchild[k]] = (uint32_t)(nused + k) << 1;
            parent[w.rchild[k]] = ((uint32_t)(nused + k) << 1) | 1u;
        }
        __syncthreads();
        for (int v = threadIdx.x; v < nn; v += blockDim.x) {
            for (int u = v;; u = (int)(parent[u] >> 1)) {
                atomicAdd(&w.size[u], 1u);
                if (u == root) break;
            }
        }
        __syncthreads();
        uint32_t longest = 0;
        for (int v = threadIdx.x; v < nn; v += blockDim.x) {
            uint32_t pre = 0, depth = 0;
            unsigned long long code = 0;
            for (int u = v; u != root;) {
                const uint32_t p = parent[u];
                pre += 1u;
                if (p & 1u) {
                    pre += w.size[w.lchild[(p >> 1) - nused]];
                    if (depth < 64) code |= 1ull << depth;
                }
                depth++;
                u = (int)(p >> 1);
            }
            w.pre[v]   = pre;
            w.depth[v] = depth;
            w.code[v]  = code;
            longest    = max(longest, depth);
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_info[2], longest);
    }
    __syncthreads();
    if (s_fail) {
        if (threadIdx.x == 0) set_status(a.status, s_fail);
        return;
    }
    const uint32_t nc = s_info[0];
    const int nused_c = nused;
    const int wdt     = tree_index_width(nc);
    // [BE nodeCount][BE dict][u8 0][L][R][C u32 LE][t]  (src/huffman.hh:649-653, 438-444)
    uint8_t* o = a.out;
    if (threadIdx.x == 0) {
        o[0] = (uint8_t)(nc >> 24);
        o[1] = (uint8_t)(nc >> 16);
        o[2] = (uint8_t)(nc >> 8);
        o[3] = (uint8_t)nc;
        uint32_t dh = (uint32_t)(a.hdr_dict ? a.hdr_dict : dict);
        o[4] = (uint8_t)(dh >> 24);
        o[5] = (uint8_t)(dh >> 16);
        o[6] = (uint8_t)(dh >> 8);
        o[7] = (uint8_t)dh;
        o[8] = 0;
    }
    uint8_t* pL = o + 9;
    uint8_t* pR = pL + (size_t)wdt * nc;
    uint8_t* pC = pR + (size_t)wdt * nc;
    uint8_t* pT = pC + 4 * (size_t)nc;
    for (uint32_t v = threadIdx.x; v < nc; v += blockDim.x) {
        const uint32_t idx = w.pre[v];
        const bool leaf    = (int)v < nused_c;
        uint32_t l = 0, r = 0, c = 0;
        if (leaf) {
            c = w.used[v];
            a.cb_len[c]  = (uint8_t)(w.depth[v] > 255u ? 255u : w.depth[v]);
            a.cb_word[c] = w.code[v];
        } else {
            l = w.pre[w.lchild[v - nused_c]];
            r = w.pre[w.rchild[v - nused_c]];
        }
        for (int b = 0; b < wdt; b++) {
            pL[(size_t)idx * wdt + b] = (uint8_t)(l >> (8 * b));
            pR[(size_t)idx * wdt + b] = (uint8_t)(r >> (8 * b));
        }
        pC[4 * (size_t)idx + 0] = (uint8_t)c;
        pC[4 * (size_t)idx + 1] = (uint8_t)(c >> 8);
        pC[4 * (size_t)idx + 2] = (uint8_t)(c >> 16);
        pC[4 * (size_t)idx + 3] = (uint8_t)(c >> 24);
        pT[idx]                 = leaf ? 1 : 0;
    }
    if (threadIdx.x < 4) a.info[threadIdx.x] = s_info[threadIdx.x];
}

}  // namespace vsz
