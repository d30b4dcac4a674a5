// Dual-quantization decompress on sm_103a: outlier placement + reverse Lorenzo + dequantization.
//
// Replaces, from szcompressor/vecSZ:
//   outlier scatter           src/vecsz_interface.hh:313-317
//   x_lorenzo_{1,2,3}d1l      src/dualquant.hh:915-1043
//
// Per element, in the reference's FP32 operation order (zero halo per block, or with padding the
// block's pad values from the archive's pad section, src/dualquant.hh:946-1016):
//   s = code == 0 ? outlier : (float)(pred + (float)(code - R))
//   pred: 1D s[x-1]; 2D (N + W) - NW; 3D XYZ - XY - XZ - YZ + X + Y + Z, left to right
//   xhat = (float)((double) s * 2eb)                 (dequant(), vsz_device.cuh)
// The outliers are placed first, as the reference's scatter does: k_outlier_scatter writes each one
// to its element of the output, where the reverse Lorenzo kernels read it (code 0) before they
// write the reconstruction there.  So no kernel ranks the zero codes of its rows; the placement
// reads only the chunks of 512 codes that hold some.
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "vsz_device.cuh"
#include "vsz_kernels.h"

namespace vsz {

constexpr int kDSeg = 256;  // decompress row segment (one warp of 8-wide blocks)

// ------------------------------------------------------------------------------------------
// Outlier placement.  zero codes per chunk of kOutChunk codes are known (the Huffman decoder counts
// them, or k_count_zeros_chunk); their exclusive scan gives each chunk's first outlier.  A warp
// takes a chunk with zero codes 64 codes at a time: ballots rank them, and the outliers, which
// lie at any byte offset of the archive, are read as two aligned words and a funnel shift -- so
// reads and writes are contiguous across the warp where outliers are dense.
// ------------------------------------------------------------------------------------------
constexpr int kOutChunk = 512;

__device__ __forceinline__ float outlier_at(const uint8_t* o, unsigned long long i, unsigned sh) {
    // o: the section rounded down to a word; sh: the bits skipped
    const uint32_t* w = reinterpret_cast<const uint32_t*>(o) + i;
    const uint32_t lo = __ldg(w);
    return __uint_as_float(sh ? __funnelshift_r(lo, __ldg(w + 1), sh) : lo);
}

// The cnt outliers of chunk c, the first of them outlier `rank`, by one warp.  The codes and the
// outliers (through s_val) are loaded together, all loads before the first store (the compiler
// cannot move them across it): a load latency a chunk instead of sixteen.
__device__ __forceinline__ void scatter_chunk(const OutlierArgs& a, size_t c, unsigned long long rank, uint32_t cnt,
                                              float* s_val) {
    constexpr int K     = kOutChunk / 64;
    const unsigned lane = lane_id(), lt = lanemask_lt();
    const unsigned sh   = (unsigned)(reinterpret_cast<uintptr_t>(a.outliers) & 3u) * 8u;
    const uint8_t* o    = a.outliers - sh / 8u;
    const size_t i0     = c * kOutChunk + 2u * lane;
    const bool whole    = (c + 1) * kOutChunk <= a.n && (reinterpret_cast<uintptr_t>(a.codes) & 3u) == 0;
    uint32_t w[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const size_t i = i0 + 64u * k;
        if (whole) w[k] = *reinterpret_cast<const uint32_t*>(a.codes + i);
        else w[k] = (i < a.n ? a.codes[i] : 1u) | ((i + 1 < a.n ? a.codes[i + 1] : 1u) << 16);
    }
    // a corrupt archive has fewer outliers than zero codes
    cnt = (uint32_t)min((unsigned long long)cnt, rank < a.n_out ? a.n_out - rank : 0ull);
    const uint32_t* ow = reinterpret_cast<const uint32_t*>(o) + rank;
    const unsigned next = sh ? 1u : 0u;  // aligned outliers are one word each
    for (uint32_t i0v = 0; i0v < cnt; i0v += 256) {
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {  // no branch, so that nothing waits for one of them
            const uint32_t i = min(i0v + 32u * q + lane, cnt - 1u);
            lo[q] = __ldg(ow + i);
            hi[q] = __ldg(ow + i + next);
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t i = i0v + 32u * q + lane;
            if (i < cnt) s_val[i] = __uint_as_float(__funnelshift_r(lo[q], hi[q], sh));
        }
    }
    __syncwarp();
    const bool pairs = (reinterpret_cast<uintptr_t>(a.out) & 7u) == 0;
    uint32_t run     = 0;  // outliers before step k
#pragma unroll
    for (int k = 0; k < K; k++) {
        const bool z0     = !(w[k] & 0xffffu), z1 = !(w[k] >> 16);
        const unsigned m0 = __ballot_sync(0xffffffffu, z0), m1 = __ballot_sync(0xffffffffu, z1);
        const uint32_t r  = run + __popc(m0 & lt) + __popc(m1 & lt), r1 = r + (z0 ? 1u : 0u);
        float* d          = a.out + i0 + 64u * k;
        if (z0 && z1 && r1 < cnt && pairs) {
            *reinterpret_cast<float2*>(d) = make_float2(s_val[r], s_val[r1]);
        } else {
            if (z0 && r < cnt) d[0] = s_val[r];
            if (z1 && r1 < cnt) d[1] = s_val[r1];
        }
        run += __popc(m0) + __popc(m1);
    }
    __syncwarp();  // s_val is the next chunk's
}

// One field, over the scan of its counts: CTAs of 8 warps, a warp per chunk and step.  The zero codes
// must be as many as the outliers (or, not exact, at most as many).  A scan in the same kernel, by
// look-back over tiles of 64 chunks, left it waiting on the look-back's chain (512^3: 0.05 ms, a scan
// of its own and this 0.02).
__global__ void __launch_bounds__(256) k_outlier_scatter(OutlierArgs a) {
    __shared__ float s_val[8][kOutChunk];
    if (__syncthreads_or(*a.status != VSZ_OK)) return;  // uniform
    const unsigned long long all = *a.total;
    if (a.exact ? all != a.n_out : all > a.n_out) {
        if (threadIdx.x == 0 && blockIdx.x == 0) set_status(a.status, VSZ_ERR_CORRUPT);
        return;
    }
    if (all == 0) return;
    const unsigned warp = threadIdx.x >> 5, lane = lane_id();
    // 32 counts at a time; a warp's chunks are a CTA apart, so that dense ones spread
    for (size_t c0 = (size_t)blockIdx.x * 8 + warp; c0 < a.nchunks; c0 += (size_t)gridDim.x * 8 * 32) {
        const size_t c   = c0 + (size_t)lane * gridDim.x * 8;
        const uint32_t z = c < a.nchunks ? a.chunk_zero[c] : 0u;
        const unsigned long long off = z ? a.chunk_off[c] : 0ull;
        for (unsigned m = __ballot_sync(0xffffffffu, z != 0u); m; m &= m - 1u) {
            const int q = __ffs(m) - 1;
            scatter_chunk(a, __shfl_sync(0xffffffffu, c, q), __shfl_sync(0xffffffffu, off, q),
                          __shfl_sync(0xffffffffu, z, q), s_val[warp]);
        }
    }
}

// Many fields: tasks of (field, chunk range), one CTA each, over the scan of all fields' counts.
__global__ void __launch_bounds__(256)
    k_outlier_scatter_batch(const OutlierArgs* __restrict__ args, const BatchTask* __restrict__ tasks, uint32_t ntasks) {
    __shared__ float s_val[8][kOutChunk];
    const unsigned warp = threadIdx.x >> 5;
    for (uint32_t t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const BatchTask tk   = tasks[t];
        const OutlierArgs& a = args[tk.field];
        if (*a.status != VSZ_OK) continue;  // set by earlier kernels only
        for (size_t c = tk.u0 + warp; c < tk.u1; c += 8) {
            const uint32_t z = a.chunk_zero[c];  // offsets are relative to the field's first chunk
            if (z) scatter_chunk(a, c, a.chunk_off[c] - a.chunk_off[0], z, s_val[warp]);
        }
    }
}

// Zero codes per chunk, for codes that no decoder of this library counted: a warp per chunk, two 16-byte
// loads a lane where the codes are so aligned (268 MB of codes 70 -> 51 us).
__global__ void __launch_bounds__(256) k_count_zeros_chunk(const uint16_t* __restrict__ codes, size_t n, size_t nchunks,
                                                           uint32_t* __restrict__ chunk_zero) {
    const unsigned lane = lane_id();
    const size_t wtot   = (size_t)gridDim.x * (blockDim.x >> 5);
    const bool vec      = (reinterpret_cast<uintptr_t>(codes) & 15u) == 0;
    static_assert(kOutChunk == 2 * 8 * 32, "two loads of 8 codes a lane");
    for (size_t c = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); c < nchunks; c += wtot) {
        uint32_t z = 0;
        if (vec && (c + 1) * kOutChunk <= n) {
            const uint4* p = reinterpret_cast<const uint4*>(codes + c * kOutChunk);
            const uint4 a = p[lane], b = p[lane + 32];
            z = __vseteq2(a.x, 0u) + __vseteq2(a.y, 0u) + __vseteq2(a.z, 0u) + __vseteq2(a.w, 0u) +  // per half
                __vseteq2(b.x, 0u) + __vseteq2(b.y, 0u) + __vseteq2(b.z, 0u) + __vseteq2(b.w, 0u);
            z = (z & 0xffffu) + (z >> 16);
        } else {
#pragma unroll
            for (int k = 0; k < kOutChunk / 32; k++) {
                const size_t i = c * kOutChunk + 32u * k + lane;
                z += (i < n && codes[i] == 0) ? 1u : 0u;
            }
        }
        z = __reduce_add_sync(0xffffffffu, z);
        if (lane == 0) chunk_zero[c] = z;
    }
}

int launch_count_zeros_chunk(const uint16_t* codes, size_t n, uint32_t* chunk_zero, cudaStream_t st, int num_sms) {
    const size_t nchunks = (n + kOutChunk - 1) / kOutChunk;
    if (nchunks == 0) return VSZ_OK;
    const size_t want = (nchunks + 7) / 8, cap = (size_t)num_sms * 16;
    k_count_zeros_chunk<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(codes, n, nchunks, chunk_zero);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

int launch_outlier_scatter(const OutlierArgs& a, cudaStream_t st, int num_sms) {
    if (a.nchunks == 0) return VSZ_OK;
    const size_t want = (a.nchunks + 7) / 8, cap = (size_t)num_sms * 5;  // resident CTAs
    k_outlier_scatter<<<(unsigned)(want < cap ? want : cap), 256, 0, st>>>(a);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

int launch_outlier_scatter_batch(const OutlierArgs* args, const BatchTask* tasks, uint32_t ntasks, cudaStream_t st,
                                 int num_sms) {
    if (ntasks == 0) return VSZ_OK;
    const uint32_t cap = (uint32_t)num_sms * 8;
    k_outlier_scatter_batch<<<ntasks < cap ? ntasks : cap, 256, 0, st>>>(args, tasks, ntasks);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

// ------------------------------------------------------------------------------------------
// Fast path, block size 8: one lane reconstructs one whole Lorenzo block (8 x by 8 y, plane by
// plane in z) -- the x, y and z recurrences never leave the thread.  A warp covers 32 consecutive
// blocks (one 256-wide row segment), so code loads (16 B) and value stores (32 B) of a row are
// contiguous across the warp.  Codes are prefetched one row ahead into registers; the previous
// plane of every lane's block lives in shared memory [row][column][lane] (lane-minor, so
// conflict-free).  Rows are processed in a rolled loop (8 columns unrolled): the body stays small
// enough for the instruction cache (two rows per iteration measured fastest).
// ------------------------------------------------------------------------------------------

// Any zero 16-bit half in a word (exact: a borrow out of the low half needs the low half zero).
__device__ __forceinline__ uint32_t zero_halves(uint32_t w) { return (w - 0x00010001u) & ~w & 0x80008000u; }

// Strict archives: an outlier is the input value; the Lorenzo chain continues from its
// prequantized value, by the compressor's rule for that column.
template <int NDIM>
__device__ __forceinline__ float strict_prequant(float v, uint32_t col, const DqDecArgs& a, const Consts& c) {
    if (NDIM == 3 && col >= a.xtail) return prequant_scalar(v, c.r_d);
    return prequant_vec(v, c.r_f);
}

// The outliers that k_outlier_scatter put in a row's 8 elements (zm: which of them).
template <bool VEC>
__device__ __forceinline__ void load_outliers(const float* p, uint32_t zm, float ov[8]) {
    if (VEC) {  // 16-byte rows: the other elements hold nothing yet and are not looked at
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        ov[0] = a.x, ov[1] = a.y, ov[2] = a.z, ov[3] = a.w;
        ov[4] = b.x, ov[5] = b.y, ov[6] = b.z, ov[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) ov[k] = (zm & (1u << k)) ? p[k] : 0.f;
    }
}

// The same from the archive, for blocks that the separable pass has already written over: by rank,
// the outliers before the chunk plus the zero codes from the chunk's start to the row segment's
// (q; at most 511 codes, counted by the warp) plus those of the lanes before.  All lanes call it.
__device__ __forceinline__ void redo_outliers(const DqDecArgs& a, size_t q, uint32_t zm, float ov[8]) {
    if (!__any_sync(0xffffffffu, zm != 0u)) return;
    const unsigned lane = lane_id();
    const uint32_t cnt  = __popc(zm);
    uint32_t incl       = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (unsigned)o) incl += t;
    }
    const size_t lo = (q & ~(size_t)(kOutChunk - 1)) + (size_t)lane * 16;
    uint32_t zc     = 0;
#pragma unroll
    for (int t = 0; t < 16; t++)
        if (lo + t < q) zc += (a.codes[lo + t] == 0);
    zc = __reduce_add_sync(0xffffffffu, zc);
    unsigned long long r = a.chunk_off[q / kOutChunk] - a.chunk_off[0] + zc + (incl - cnt);
    const unsigned sh    = (unsigned)(reinterpret_cast<uintptr_t>(a.outliers) & 3u) * 8u;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        ov[k] = 0.f;
        if (!(zm & (1u << k))) continue;
        if (r < a.n_outliers) ov[k] = outlier_at(a.outliers - sh / 8u, r, sh);
        else set_status(a.status, VSZ_ERR_CORRUPT);
        r++;
    }
}

typedef float DqPlane[8][8][32];  // one warp's plane of 8 x 8 blocks, [row][column][lane]
typedef float4 DqPlaneV[8][2][32];  // the same bytes for the separable pass: [row][half][lane] x 4 columns

// Units ui = first, first + stride, ... < end of one field (one warp each; `wib` = this warp's
// plane in s_prev).  REDO: the units the separable kernel listed instead (end = their count,
// read by the caller: final in stream order).
template <int NDIM, bool VEC, bool PAD, bool REDO>
__device__ __forceinline__ void dq_b8_units(const DqDecArgs& a, uint32_t first, uint32_t end, uint32_t stride,
                                            DqPlane* s_prev, unsigned wib) {
    const Consts c = *a.consts;
    if (c.status != VSZ_OK || *a.status != VSZ_OK) return;
    const int R           = a.R;
    // (float)(code - R) exactly: 2^23 + code as float bits, minus 2^23 + R (both exact, R < 2^16)
    const float rbias     = 8388608.0f + (float)R;
    const uint32_t rpair  = (uint32_t)R | ((uint32_t)R << 16);
    const unsigned lane   = lane_id();

    // Narrow rows (a.ygrp > 1, rows of at most 16 blocks): the warp takes ygrp consecutive
    // y-blocks of one z-block, a group of nbx8 lanes per y-block (lanes past ygrp * nbx8 idle), so
    // that its lanes are not spent on columns past the row's end.  A lane still reconstructs one
    // whole block.
    const uint32_t G   = (REDO || PAD || NDIM == 1) ? 1u : a.ygrp;
    const uint32_t gw  = G > 1 ? a.nbx8 : 32u;  // lanes per group
    const uint32_t grp = G > 1 ? lane / gw : 0u;
    const uint32_t gl0 = grp * gw;              // the group's first lane
    const uint32_t lbx = lane - gl0;            // this lane's block along x in its segment
    // unit indices fit 32 bits (n <= 2^36 elements, 2048 per unit): 32-bit divisions only.
    for (uint32_t ui = first; ui < end; ui += stride) {
        const uint32_t u  = REDO ? a.redo[1 + ui] : ui;
        uint32_t xs, yb, zb;
        if (G > 1) {  // units: (group of G y-blocks, z-block)
            xs = 0;
            yb = (u % a.nyb_g) * G + grp;
            zb = (NDIM == 3) ? u / a.nyb_g : 0u;
        } else {
            xs = u % a.nxs;
            const uint32_t r = u / a.nxs;
            yb = (NDIM >= 2) ? r % a.nyb : 0u;
            zb = (NDIM == 3) ? r / a.nyb : 0u;
        }
        const bool blk_in = grp < G && (NDIM < 2 || yb < a.nyb);  // my block exists
        const uint32_t x0 = xs * kDSeg + lbx * 8;
        const uint32_t y0 = yb * 8, z0 = zb * 8;
        const int ny = (NDIM >= 2) ? (blk_in ? (int)min(8u, a.d1 - y0) : 0) : 1;
        const int nz = (NDIM == 3) ? (int)min(8u, a.d2 - z0) : 1;
        const bool col_in = blk_in && x0 < a.d0;  // VEC: d0 % 8 == 0, so all 8 columns or none
        // halo of my block (zero without padding): x-, y- and z-halo cells; in 3D the (x-1, y-1)
        // cell of a halo row is the y-halo's, in 2D the x-halo's
        float hx = 0.f, hy = 0.f, hz = 0.f;
        if (PAD && col_in) {
            const Halo hv = halo_of(a.pad, NDIM, x0 / 8, yb, zb);
            hx = hv.x;
            hy = hv.y;
            hz = hv.z;
        }

        // the 8 codes of this lane's columns (VEC: one 16-byte load), a row ahead of their use;
        // cells outside the field read as R (no zero codes, so they never enter the outlier path)
        auto load_row = [&](int zz, int y) -> uint4 {
            const size_t row = (size_t)(z0 + zz) * a.d1 + (y0 + y);
            if (VEC) {
                if (!(col_in && y < ny && zz < nz)) return make_uint4(rpair, rpair, rpair, rpair);
                return __ldcs(reinterpret_cast<const uint4*>(a.codes + row * a.d0 + x0));
            }
            const bool rin       = y < ny && zz < nz;
            const uint16_t* crow = a.codes + row * a.d0;
            uint32_t t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = (rin && x0 + k < a.d0) ? (uint32_t)crow[x0 + k] : (uint32_t)R;
            return make_uint4(t[0] | (t[1] << 16), t[2] | (t[3] << 16), t[4] | (t[5] << 16), t[6] | (t[7] << 16));
        };
        uint4 cv_next = load_row(0, 0);

        if (NDIM == 3) {
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int k = 0; k < 8; k++) s_prev[wib][i][k][lane] = hz;
        }

        for (int zz = 0; zz < nz; zz++) {
            float Cm[8];  // row y - 1 of this plane (the halo row above the block)
            float Zm[8], Zn[8];  // 3D: row y - 1 and row y of plane z - 1
#pragma unroll
            for (int k = 0; k < 8; k++) Cm[k] = hy;
#pragma unroll 2
            for (int y = 0; y < 8; y++) {
                const bool row_in = y < ny;
                const size_t row  = ((size_t)(z0 + zz) * a.d1 + (y0 + y));
                const bool all_in = row_in && (x0 + 7 < a.d0);
                const uint4 cv    = cv_next;
                cv_next           = (y < 7) ? load_row(zz, y + 1) : load_row(zz + 1, 0);
                const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
                auto code_at = [&](int k) -> uint32_t { return (cw[k >> 1] >> (16 * (k & 1))) & 0xffffu; };
                auto in_at   = [&](int k) -> bool { return all_in || (row_in && x0 + (uint32_t)k < a.d0); };
                // outliers of this lane's columns.  Cells outside the field read code R (never 0), so no
                // range test is needed here or in the row pass: their values only ever feed other
                // cells outside the field.
                uint32_t zm = 0;
                if (zero_halves(cv.x) | zero_halves(cv.y) | zero_halves(cv.z) | zero_halves(cv.w)) {
#pragma unroll
                    for (int k = 0; k < 8; k++) zm |= (code_at(k) == 0u) ? (1u << k) : 0u;
                }
                float ov[8];
                if (REDO) redo_outliers(a, row * a.d0 + (size_t)xs * kDSeg, zm, ov);
                else if (zm) load_outliers<VEC>(a.out + row * a.d0 + x0, zm, ov);
                // ---- reverse Lorenzo along the row; an element with code 0 takes its outlier
                float C[8];
                auto row_pass = [&](auto with_outliers) {
                    float pZ = 0.f, pYZ = 0.f;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        float pred;
                        if (NDIM == 1) {
                            pred = k ? C[k - 1] : hx;
                        } else if (NDIM == 2) {
                            const float X  = k ? C[k - 1] : hx;
                            const float XY = k ? Cm[k - 1] : hx;
                            pred           = __fsub_rn(__fadd_rn(Cm[k], X), XY);  // (N + W) - NW
                        } else {
                            // previous plane: this row (z-1, y) from shared memory, the row above
                            // (z-1, y-1) kept from the row before; both rolled along x
                            const float Z   = s_prev[wib][y][k][lane];
                            const float YZ  = y ? Zm[k] : (zz ? hy : hz);
                            Zn[k]           = Z;
                            const float XYZ = k ? pYZ : (zz ? (y ? hx : hy) : hz);
                            const float XZ  = k ? pZ : (zz ? hx : hz);
                            pZ              = Z;
                            pYZ             = YZ;
                            const float XY  = k ? Cm[k - 1] : (y ? hx : hy);
                            const float X   = k ? C[k - 1] : hx;
                            pred = __fadd_rn(__fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(__fsub_rn(XYZ, XY), XZ), YZ), X), Cm[k]),
                                             Z);
                        }
                        const uint32_t cd = code_at(k);
                        float s = __fadd_rn(pred, __fsub_rn(__uint_as_float(0x4B000000u | cd), rbias));
                        if (decltype(with_outliers)::value) {
                            if (zm & (1u << k)) {
                                s = ov[k];
                                if (a.strict) s = strict_prequant<NDIM>(s, x0 + (uint32_t)k, a, c);
                            }
                        }
                        C[k] = s;
                    }
                };
                if (zm) row_pass(std::true_type{});
                else row_pass(std::false_type{});
                float* orow = a.out + row * a.d0;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float xo[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) xo[k] = dequant(C[4 * h + k], c.c_d, c.c_hi, c.c_lo, c.dq_fast);
                    if (a.strict && zm) {  // strict outliers are output as stored
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            if (zm & (1u << (4 * h + k))) xo[k] = ov[4 * h + k];
                        }
                    }
                    if (VEC && all_in) {
                        __stcs(reinterpret_cast<float4*>(orow + x0 + 4 * h), make_float4(xo[0], xo[1], xo[2], xo[3]));
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (in_at(4 * h + k)) orow[x0 + 4 * h + k] = xo[k];
                    }
                }
                if (NDIM == 3 && y > 0) {  // row y-1 of this plane is no longer needed as "plane z-1"
#pragma unroll
                    for (int k = 0; k < 8; k++) s_prev[wib][y - 1][k][lane] = Cm[k];
                }
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    Cm[k] = C[k];
                    if (NDIM == 3) Zm[k] = Zn[k];
                }
                if (NDIM == 1) break;
            }
            if (NDIM == 3) {
#pragma unroll
                for (int k = 0; k < 8; k++) s_prev[wib][7][k][lane] = Cm[k];
            }
        }
    }
}

template <int NDIM, bool VEC, bool PAD = false, bool REDO = false>
__global__ void __launch_bounds__(128, 6) k_dq_decompress_b8(DqDecArgs a) {
    extern __shared__ __align__(16) uint8_t s_dq_dyn[];
    const unsigned wib = threadIdx.x >> 5;  // warp in block (4 warps)
    const uint32_t end = REDO ? a.redo[0] : (uint32_t)a.nunits;
    dq_b8_units<NDIM, VEC, PAD, REDO>(a, blockIdx.x * (blockDim.x >> 5) + wib, end, gridDim.x * (blockDim.x >> 5),
                                      reinterpret_cast<DqPlane*>(s_dq_dyn), wib);
}

// ------------------------------------------------------------------------------------------
// Separable pass, 3D, block 8, zero halo (no padding), not strict.  With a zero halo the Lorenzo
// inverse is the block's 3D inclusive prefix sum of the residuals q = code - R, so an element takes
// three adds -- A = A(z-1) + q, B = B(y-1) + A, s = s(x-1) + B -- instead of the predictor's seven.
// While every value of the block stays below 2^21 in magnitude, every partial sum of the
// reference's order and of this one is an integer below 2^24, exact in FP32, so both give the same
// bits.  An outlier sets s; B and A are corrected from it (B = s - s(x-1), A = B - B(y-1)).  A warp
// with a block whose values leave that range (or meet a NaN or an infinity) lists its unit in
// a.redo, and the reference-order kernel redoes it afterwards.
// ------------------------------------------------------------------------------------------
// Units u = first, first + stride, ... < end of one field; s_A: A of the previous plane.
__device__ __forceinline__ void dq_b8s_units(const DqDecArgs& a, uint32_t first, uint32_t end, uint32_t stride,
                                             DqPlane* s_A, unsigned wib) {
    const Consts c = *a.consts;
    if (c.status != VSZ_OK || *a.status != VSZ_OK) return;
    const int R                = a.R;
    const float rbias          = 8388608.0f + (float)R;
    const uint32_t rpair       = (uint32_t)R | ((uint32_t)R << 16);
    const unsigned lane        = lane_id();
    // rows start on 32-byte boundaries (d0 % 8 == 0) when the output does
    const bool out32           = (reinterpret_cast<uintptr_t>(a.out) & 31u) == 0;

    for (uint32_t u = first; u < end; u += stride) {
        const uint32_t xs = u % a.nxs;
        const uint32_t r  = u / a.nxs;
        const uint32_t yb = r % a.nyb;
        const uint32_t zb = r / a.nyb;
        const uint32_t x0 = xs * kDSeg + lane * 8;
        const uint32_t y0 = yb * 8, z0 = zb * 8;
        const int ny      = (int)min(8u, a.d1 - y0);
        const int nz      = (int)min(8u, a.d2 - z0);
        const bool col_in = x0 < a.d0;  // d0 % 8 == 0: all 8 columns or none
        auto load_row = [&](int zz, int y) -> uint4 {
            if (!(col_in && y < ny && zz < nz)) return make_uint4(rpair, rpair, rpair, rpair);
            const size_t row = (size_t)(z0 + zz) * a.d1 + (y0 + y);
            return __ldcs(reinterpret_cast<const uint4*>(a.codes + row * a.d0 + x0));
        };
        uint4 cv_next = load_row(0, 0);
        DqPlaneV* sAv = reinterpret_cast<DqPlaneV*>(s_A);  // a row's 8 A values: two 16-byte accesses
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) sAv[wib][i][h][lane] = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t big = 0;  // largest |value| of the block, as float bits (NaN and infinity above all)

        for (int zz = 0; zz < nz; zz++) {
            float Bm[8];  // B of the row above (zero above the block)
#pragma unroll
            for (int k = 0; k < 8; k++) Bm[k] = 0.f;
#pragma unroll 2
            for (int y = 0; y < 8; y++) {
                const bool row_in = y < ny;
                const size_t row  = ((size_t)(z0 + zz) * a.d1 + (y0 + y));
                const bool all_in = row_in && col_in;
                const uint4 cv    = cv_next;
                cv_next           = (y < 7) ? load_row(zz, y + 1) : load_row(zz + 1, 0);
                {  // the row 4 ahead into L2 (rows of this unit only): the load one row ahead then hits L2
                    const int za = y < 4 ? zz : zz + 1, ya = (y + 4) & 7;
                    if (col_in && za < nz && ya < ny) {
                        const size_t rowa = (size_t)(z0 + za) * a.d1 + (y0 + ya);
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.codes + rowa * a.d0 + x0));
                    }
                }
                const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
                auto code_at = [&](int k) -> uint32_t { return (cw[k >> 1] >> (16 * (k & 1))) & 0xffffu; };
                uint32_t zm = 0;  // outliers of this lane's columns
                if (zero_halves(cv.x) | zero_halves(cv.y) | zero_halves(cv.z) | zero_halves(cv.w)) {
#pragma unroll
                    for (int k = 0; k < 8; k++) zm |= (code_at(k) == 0u) ? (1u << k) : 0u;
                }
                float C[8], Ar[8];  // Ar: A of the row in the previous plane, then of this one
                {
                    const float4 a0 = sAv[wib][y][0][lane], a1 = sAv[wib][y][1][lane];
                    Ar[0] = a0.x, Ar[1] = a0.y, Ar[2] = a0.z, Ar[3] = a0.w;
                    Ar[4] = a1.x, Ar[5] = a1.y, Ar[6] = a1.z, Ar[7] = a1.w;
                }
                auto row_pass = [&](auto with_outliers) {
                    float ov[8];
                    if (decltype(with_outliers)::value) load_outliers<true>(a.out + row * a.d0 + x0, zm, ov);
                    float sl = 0.f;  // s of the element to the left (zero left of the block)
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const float q = __fsub_rn(__uint_as_float(0x4B000000u | code_at(k)), rbias);
                        float A       = __fadd_rn(Ar[k], q);
                        float B       = __fadd_rn(Bm[k], A);
                        float sv      = __fadd_rn(sl, B);
                        if (decltype(with_outliers)::value) {
                            if (zm & (1u << k)) {
                                sv = ov[k];
                                B = __fsub_rn(sv, sl);
                                A = __fsub_rn(B, Bm[k]);
                            }
                        }
                        Ar[k]                = A;
                        Bm[k]                = B;
                        sl                   = sv;
                        C[k]                 = sv;
                        big                  = max(big, __float_as_uint(sv) & 0x7fffffffu);
                    }
                };
                if (zm) row_pass(std::true_type{});
                else row_pass(std::false_type{});
                sAv[wib][y][0][lane] = make_float4(Ar[0], Ar[1], Ar[2], Ar[3]);
                sAv[wib][y][1][lane] = make_float4(Ar[4], Ar[5], Ar[6], Ar[7]);
                if (all_in) {
                    float* orow = a.out + row * a.d0;
                    float xo[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) xo[k] = dequant_small(C[k], c);
                    if (out32) {  // the lane's 8 values are one 32-byte sector: one 256-bit store
                        asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(orow + x0),
                                     "f"(xo[0]), "f"(xo[1]), "f"(xo[2]), "f"(xo[3]), "f"(xo[4]), "f"(xo[5]), "f"(xo[6]),
                                     "f"(xo[7])
                                     : "memory");
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            __stcs(reinterpret_cast<float4*>(orow + x0 + 4 * h),
                                   make_float4(xo[4 * h], xo[4 * h + 1], xo[4 * h + 2], xo[4 * h + 3]));
                    }
                }
            }
        }
        // 0x4A000000 = 2^21: a block with a larger value (or a NaN / infinity) is redone
        if (__any_sync(0xffffffffu, big >= 0x4A000000u) && lane == 0) {
            const uint32_t i = atomicAdd(a.redo, 1u);
            a.redo[1 + i]    = u;
        }
    }
}

// A check result kept in the caller's workspace: c_d's bits, the mode and exception, and a check
// word, so that bytes left there by anything else are not taken for a result.
constexpr unsigned long long kDqCacheMagic = 0x9e3779b97f4a7c15ull;
__device__ __forceinline__ unsigned long long dq_cache_check(unsigned long long key, unsigned long long v0,
                                                             unsigned long long v1) {
    return (key * kDqCacheMagic) ^ (v0 + 0x632be59bd9b4e019ull) ^ (v1 * 0xc2b2ae3d27d4eb4full) ^ 0x5bd1e995ull;
}

// Checks, for every integer 0 < s < 2^21, the two-operation dequantization of dequant_small()
// against the reference's (float)((double)s * c_d), and sets c->dq_mul (negative s follow: both
// forms are odd).  scratch: 3 words, zero on entry (mismatches, one mismatching s, block ticket);
// the last block to finish sets the mode and zeroes scratch[0] again.  cache (4 words, or null):
// the last result for this workspace; a hit for the same c_d skips the check.
__global__ void __launch_bounds__(256) k_dq_mul_verify(Consts* __restrict__ c, uint32_t* __restrict__ scratch,
                                                       unsigned long long* __restrict__ cache) {
    __shared__ uint32_t s_bad;
    const Consts k = *c;
    const unsigned long long key = (unsigned long long)__double_as_longlong(k.c_d);
    if (cache && k.status == VSZ_OK) {
        const unsigned long long ck = cache[0], v0 = cache[1], v1 = cache[2], chk = cache[3];
        if (ck == key && chk == dq_cache_check(ck, v0, v1) && (v0 & 0xffu) <= 2u) {  // uniform over the grid
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                c->dq_mul   = (int)(v0 & 0xffu);
                c->dq_exc   = __uint_as_float((uint32_t)(v0 >> 32));
                c->dq_exc_y = __uint_as_float((uint32_t)v1);
            }
            return;
        }
    }
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    uint32_t bad = 0, which = 0;
    if (k.status == VSZ_OK) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x + 1; i < (1u << 21); i += gridDim.x * blockDim.x) {
            const float s   = (float)i;  // exact
            const float y1  = __fmaf_rn(s, k.c_hi, __fmul_rn(s, k.c_lo));
            const float y2  = __double2float_rn(__dmul_rn((double)i, k.c_d));
            const bool diff = __float_as_uint(y1) != __float_as_uint(y2);
            bad += diff ? 1u : 0u;
            which = diff ? i : which;
        }
    }
    if (bad) {
        atomicAdd(&s_bad, bad);
        atomicExch(&scratch[1], which);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (s_bad) atomicAdd(&scratch[0], s_bad);
    __threadfence();
    if (atomicAdd(&scratch[2], 1u) != gridDim.x - 1) return;
    __threadfence();
    const uint32_t nbad = atomicAdd(&scratch[0], 0u), s1 = atomicAdd(&scratch[1], 0u);
    const int mode      = k.status != VSZ_OK ? 0 : nbad == 0 ? 1 : nbad == 1 ? 2 : 0;
    const float exc   = mode == 2 ? (float)s1 : 0.f;
    const float exc_y = mode == 2 ? __double2float_rn(__dmul_rn((double)s1, k.c_d)) : 0.f;
    c->dq_exc   = exc;
    c->dq_exc_y = exc_y;
    c->dq_mul   = mode;
    scratch[0]  = 0u;  // the separable pass counts its redo units here
    if (cache && k.status == VSZ_OK) {
        const unsigned long long v0 = (unsigned long long)mode | ((unsigned long long)__float_as_uint(exc) << 32);
        const unsigned long long v1 = __float_as_uint(exc_y);
        cache[0] = key;
        cache[1] = v0;
        cache[2] = v1;
        cache[3] = dq_cache_check(key, v0, v1);
    }
}

__global__ void __launch_bounds__(128, 6) k_dq_decompress_b8s(DqDecArgs a) {
    extern __shared__ __align__(16) uint8_t s_dq_dyn[];
    const unsigned wib = threadIdx.x >> 5;
    dq_b8s_units(a, blockIdx.x * (blockDim.x >> 5) + wib, (uint32_t)a.nunits, gridDim.x * (blockDim.x >> 5),
                 reinterpret_cast<DqPlane*>(s_dq_dyn), wib);
}

// ------------------------------------------------------------------------------------------
// Wavefront pass, 3D, block 8, no padding: single fields of at most kW8MaxN elements, and the 3D fields of
// batches that hold at most 2^25 elements of them (kDbatchW8MaxN).  The block-8
// kernels give each lane a whole 8 x 8 x 8 block, 512 elements one after another; a field with
// fewer warp units than the GPU holds then takes that chain's latency (0.1-0.3 ms) whatever its
// size.  Here a block has 8 lanes, one per row y, and lane y runs one plane behind lane y - 1: at
// step t it reconstructs row (y, z = t - y) from its own row of plane z - 1 (in registers) and
// lane y - 1's rows of planes z and z - 1 (shuffled one lane up after each step).  15 steps of 8
// elements per lane instead of 512; the predictor is the reference's, in its FP32 order, so the
// values are the same bits.  A warp holds 4 blocks along x.
//
// With few warps in flight a step waits for whatever it loads, so a lane's codes of all its planes are
// staged in shared memory first (one load latency a unit, not one a step), and rows with outliers
// prefetched then: 64^3 24 -> 20 us, 333x241x187 85 -> 77.
// ------------------------------------------------------------------------------------------
typedef uint4 W8Codes[8][32];  // one warp's codes: [plane][lane]

// Units u = first, first + stride, ... < end of one field (one warp each); s_codes: this warp's.
template <bool VEC>
__device__ __forceinline__ void dq_w8_units(const DqDecArgs& a, uint32_t first, uint32_t end, uint32_t stride,
                                            W8Codes& s_codes) {
    const Consts c = *a.consts;
    if (c.status != VSZ_OK || *a.status != VSZ_OK) return;
    const int R           = a.R;
    const float rbias     = 8388608.0f + (float)R;
    const uint32_t rpair  = (uint32_t)R | ((uint32_t)R << 16);
    const unsigned lane   = lane_id();
    const int y           = (int)(lane & 7u);  // row of the block
    const uint32_t nxq    = (a.nbx8 + 3) / 4;  // groups of 4 blocks along x
    // unit indices fit 32 bits: there are no more units than elements, 2^25 at most (a unit of four whole
    // blocks holds 2048)
    for (uint32_t u = first; u < end; u += stride) {
        const uint32_t xq = u % nxq, r = u / nxq;
        const uint32_t yb = r % a.nyb, zb = r / a.nyb;
        const uint32_t bx = xq * 4 + (lane >> 3);
        const uint32_t x0 = bx * 8, z0 = zb * 8, yr = yb * 8 + (uint32_t)y;
        const int nz        = (int)min(8u, a.d2 - z0);  // the same for the whole warp
        const bool row_in   = bx < a.nbx8 && yr < a.d1;  // this lane's row exists (in every plane)
        const bool all_in   = row_in && x0 + 7 < a.d0;
        auto row_of = [&](int zz) -> size_t { return (size_t)(z0 + zz) * a.d1 + yr; };
        // the 8 codes of the lane's row in plane zz (cells outside the field read R: never an
        // outlier, and their values only feed other cells outside the field)
        auto load_row = [&](int zz) -> uint4 {
            if (!(row_in && zz < nz)) return make_uint4(rpair, rpair, rpair, rpair);
            const uint16_t* crow = a.codes + row_of(zz) * a.d0;
            if (VEC) return __ldcs(reinterpret_cast<const uint4*>(crow + x0));
            uint32_t t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = (x0 + k < a.d0) ? (uint32_t)crow[x0 + k] : (uint32_t)R;
            return make_uint4(t[0] | (t[1] << 16), t[2] | (t[3] << 16), t[4] | (t[5] << 16), t[6] | (t[7] << 16));
        };
        float Zp[8], Y[8], Yp[8];  // own row of plane z - 1; rows y - 1 of planes z and z - 1
#pragma unroll
        for (int k = 0; k < 8; k++) Zp[k] = Y[k] = Yp[k] = 0.f;
        if (VEC) {
#pragma unroll
            for (int zz = 0; zz < 8; zz++) {
                if (row_in && zz < nz) cp_async16_zfill(&s_codes[zz][lane], a.codes + row_of(zz) * a.d0 + x0, 16u);
                else s_codes[zz][lane] = make_uint4(rpair, rpair, rpair, rpair);
            }
            cp_async_commit();
            cp_async_wait<0>();
        } else {
#pragma unroll 2
            for (int zz = 0; zz < 8; zz++) s_codes[zz][lane] = load_row(zz);
        }
        // (a lane reads back what it wrote itself)
        if (a.n_outliers) {
#pragma unroll
            for (int zz = 0; zz < 8; zz++) {
                const uint4 cz = s_codes[zz][lane];
                if (zero_halves(cz.x) | zero_halves(cz.y) | zero_halves(cz.z) | zero_halves(cz.w))
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(a.out + row_of(zz) * a.d0 + x0));
            }
        }
        for (int t = 0; t < nz + 7; t++) {
            float up[8];  // lane y - 1's newest row (row y - 1 of the plane this lane takes now)
#pragma unroll
            for (int k = 0; k < 8; k++) up[k] = __shfl_up_sync(0xffffffffu, Zp[k], 1);
            const int zz = t - y;
            if (zz >= 0 && zz < nz) {
                const uint4 cw4 = s_codes[zz][lane];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    Yp[k] = Y[k];
                    Y[k]  = y ? up[k] : 0.f;
                }
                const uint32_t cw[4] = {cw4.x, cw4.y, cw4.z, cw4.w};
                auto code_at = [&](int k) -> uint32_t { return (cw[k >> 1] >> (16 * (k & 1))) & 0xffffu; };
                uint32_t zm = 0;
                if (zero_halves(cw4.x) | zero_halves(cw4.y) | zero_halves(cw4.z) | zero_halves(cw4.w)) {
#pragma unroll
                    for (int k = 0; k < 8; k++) zm |= (code_at(k) == 0u) ? (1u << k) : 0u;
                }
                float C[8], ov[8];
                if (zm) load_outliers<VEC>(a.out + row_of(zz) * a.d0 + x0, zm, ov);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const float X   = k ? C[k - 1] : 0.f;
                    const float XY  = k ? Y[k - 1] : 0.f;
                    const float XZ  = k ? Zp[k - 1] : 0.f;
                    const float XYZ = k ? Yp[k - 1] : 0.f;
                    const float pred =
                        __fadd_rn(__fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(__fsub_rn(XYZ, XY), XZ), Yp[k]), X), Y[k]), Zp[k]);
                    float s = __fadd_rn(pred, __fsub_rn(__uint_as_float(0x4B000000u | code_at(k)), rbias));
                    if (zm & (1u << k)) {
                        s = ov[k];
                        if (a.strict) s = strict_prequant<3>(s, x0 + (uint32_t)k, a, c);
                    }
                    C[k] = s;
                }
                float xo[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    xo[k] = dequant(C[k], c.c_d, c.c_hi, c.c_lo, c.dq_fast);
                    if (a.strict && (zm & (1u << k))) xo[k] = ov[k];  // strict outliers are output as stored
                }
                float* orow = a.out + row_of(zz) * a.d0;
                if (VEC && all_in) {
                    __stcs(reinterpret_cast<float4*>(orow + x0), make_float4(xo[0], xo[1], xo[2], xo[3]));
                    __stcs(reinterpret_cast<float4*>(orow + x0 + 4), make_float4(xo[4], xo[5], xo[6], xo[7]));
                } else if (row_in) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        if (x0 + (uint32_t)k < a.d0) orow[x0 + k] = xo[k];
                }
#pragma unroll
                for (int k = 0; k < 8; k++) Zp[k] = C[k];
            }
        }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(128, 4) k_dq_decompress_w8(DqDecArgs a) {
    __shared__ W8Codes s_codes[4];
    dq_w8_units<VEC>(a, blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), (uint32_t)a.nunits,
                     gridDim.x * (blockDim.x >> 5), s_codes[threadIdx.x >> 5]);
}

void dq_w8_geometry(DqDecArgs& a) { a.nunits = (unsigned long long)((a.nbx8 + 3) / 4) * a.nyb * ((a.d2 + 7) / 8); }

bool dq_w8_applies(const DqDecArgs& a, int ndim) {
    if (ndim != 3 || a.pad.vals || a.n > kW8MaxN) return false;
    if (getenv("VSZ_DQ_NO_WAVEFRONT") != nullptr) return false;
    // the separable pass catches up with the wavefront between 256x256x128 (82 us against 45) and 256^3
    // (59 against 65); the reference-order pass over aligned rows at 384x384x256 (163 against 171)
    return a.n <= kW8MaxSeparableN || !dq_b8_separable(a, ndim);
}

// ------------------------------------------------------------------------------------------
// General block sizes (16, 32, 64; also 8): one thread per block row, skewed pipeline.
// Thread t (row y = t of the block) visits its elements in (z, x) order one step behind thread
// t - 1, so every neighbour it reads was written in an earlier step; planes alternate between
// two shared-memory buffers.  A CTA runs G = 128 / bs blocks side by side.
// 1D: one thread per block, sequential along x.
// ------------------------------------------------------------------------------------------
template <int NDIM, int BS, bool PAD = false>
__global__ void __launch_bounds__(128) k_dq_decompress_gen(DqDecArgs a) {
    constexpr int G = (128 / BS) > 0 ? (128 / BS) : 1;
    extern __shared__ float s_buf[];  // G blocks x 2 planes x BS x BS
    const Consts c = *a.consts;
    if (c.status != VSZ_OK || *a.status != VSZ_OK) return;  // uniform across the grid
    const int R = a.R;
    if (NDIM == 1) {
        size_t b = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
        size_t x0 = b * BS;
        if (x0 >= a.d0) return;
        const float hx = PAD ? halo_of(a.pad, 1, (uint32_t)(x0 / BS), 0, 0).x : 0.f;
        float prev = 0.f;
        for (int k = 0; k < BS; k++) {
            size_t x = x0 + k;
            if (x >= a.d0) break;
            uint32_t cd = a.codes[x];
            float s, xo;
            if (cd == 0u) {
                s  = a.out[x];
                xo = s;  // strict: the stored input value
                if (a.strict) s = strict_prequant<1>(s, (uint32_t)x, a, c);
                else xo = dequant(s, c.c_d, c.c_hi, c.c_lo, c.dq_fast);
            } else {
                s  = __fadd_rn(k ? prev : hx, (float)((int)cd - R));
                xo = dequant(s, c.c_d, c.c_hi, c.c_lo, c.dq_fast);
            }
            prev     = s;
            a.out[x] = xo;
        }
        return;
    }
    const int g = threadIdx.x / BS, t = threadIdx.x % BS;
    const unsigned long long blk = (unsigned long long)blockIdx.x * G + g;
    const bool active = blk < a.nunits;
    const uint32_t bx = active ? (uint32_t)(blk % a.nbx) : 0u;
    const unsigned long long rr = active ? blk / a.nbx : 0ull;
    const uint32_t by = (uint32_t)(rr % a.nyb);
    const uint32_t bz = (NDIM == 3) ? (uint32_t)(rr / a.nyb) : 0u;
    const uint32_t x0 = bx * BS, y = by * BS + t, z0 = bz * BS;
    float hx = 0.f, hy = 0.f, hz = 0.f;  // halo of this block (zero without padding)
    if (PAD && active) {
        const Halo hv = halo_of(a.pad, NDIM, bx, by, bz);
        hx = hv.x;
        hy = hv.y;
        hz = hv.z;
    }
    float* S0 = s_buf + (size_t)g * 2 * BS * BS;
    float* S1 = S0 + BS * BS;
    for (int i = t; i < 2 * BS * BS; i += BS) S0[i] = 0.f;
    __syncthreads();
    const int nsteps = (NDIM == 3) ? (BS * BS + BS - 1) : (2 * BS - 1);
    for (int step = 0; step < nsteps; step++) {
        const int q = step - t;
        const int lim = (NDIM == 3) ? BS * BS : BS;
        if (active && q >= 0 && q < lim) {
            const int zl = (NDIM == 3) ? q / BS : 0, xl = (NDIM == 3) ? q % BS : q;
            const uint32_t z = z0 + zl, x = x0 + xl;
            float* Sc = (zl & 1) ? S1 : S0;  // plane z
            float* Sp = (zl & 1) ? S0 : S1;  // plane z - 1
            const bool in = (x < a.d0) && (y < a.d1) && (NDIM < 3 || z < a.d2);
            float s = 0.f;
            if (in) {
                const size_t row     = (size_t)z * a.d1 + y;
                const uint16_t* crow = a.codes + row * a.d0;
                uint32_t cd = crow[x];
                float pred;
                // halo cells: 2D (x-1, y-1) is the x-halo's, 3D the y-halo's; z - 1 = halo: hz
                const float X  = xl ? Sc[t * BS + xl - 1] : hx;
                const float Y  = t ? Sc[(t - 1) * BS + xl] : hy;
                const float XY = (t && xl) ? Sc[(t - 1) * BS + xl - 1]
                                           : (NDIM == 2 ? (xl ? hy : hx) : (t ? hx : hy));
                if (NDIM == 2) {
                    pred = __fsub_rn(__fadd_rn(Y, X), XY);
                } else {
                    const bool zp   = zl > 0;
                    const float XYZ = (zp && t && xl) ? Sp[(t - 1) * BS + xl - 1] : (zp ? (t ? hx : hy) : hz);
                    const float XZ  = (zp && xl) ? Sp[t * BS + xl - 1] : (zp ? hx : hz);
                    const float YZ  = (zp && t) ? Sp[(t - 1) * BS + xl] : (zp ? hy : hz);
                    const float Z   = zp ? Sp[t * BS + xl] : hz;
                    pred = __fadd_rn(__fadd_rn(__fadd_rn(__fsub_rn(__fsub_rn(__fsub_rn(XYZ, XY), XZ), YZ), X), Y), Z);
                }
                float xo;
                if (cd == 0u) {
                    s  = a.out[row * a.d0 + x];
                    xo = s;  // strict: the stored input value
                    if (a.strict) s = strict_prequant<NDIM>(s, x, a, c);
                    else xo = dequant(s, c.c_d, c.c_hi, c.c_lo, c.dq_fast);
                } else {
                    s  = __fadd_rn(pred, (float)((int)cd - R));
                    xo = dequant(s, c.c_d, c.c_hi, c.c_lo, c.dq_fast);
                }
                a.out[row * a.d0 + x] = xo;
            }
            Sc[t * BS + xl] = s;
        }
        __syncthreads();
    }
}

// Zero codes per 256-wide row segment, for callers that hold codes but no decoder counts.
__global__ void __launch_bounds__(256) k_count_zeros(const uint16_t* __restrict__ codes, uint32_t d0, size_t nrows,
                                                     uint32_t nxs, uint32_t* __restrict__ seg_zero) {
    const unsigned lane = lane_id();
    const size_t nseg   = nrows * nxs;
    const size_t wtot   = (size_t)gridDim.x * (blockDim.x >> 5);
    for (size_t sgi = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); sgi < nseg; sgi += wtot) {
        size_t row = sgi / nxs;
        uint32_t xs = (uint32_t)(sgi - row * nxs);
        const uint16_t* crow = codes + row * d0;
        uint32_t z = 0;
        for (uint32_t x = xs * kDSeg + lane; x < min(d0, (xs + 1) * kDSeg); x += 32) z += (crow[x] == 0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
        if (lane == 0) seg_zero[sgi] = z;
    }
}

int launch_count_zeros(const uint16_t* codes, uint32_t d0, size_t nrows, uint32_t* seg_zero, cudaStream_t st,
                       int num_sms) {
    uint32_t nxs = (d0 + kDSeg - 1) / kDSeg;
    size_t nseg  = nrows * nxs;
    if (nseg == 0) return VSZ_OK;
    long long want = (long long)((nseg + 7) / 8), cap = (long long)num_sms * 16;
    int grid = (int)(want < cap ? want : cap);
    k_count_zeros<<<grid, 256, 0, st>>>(codes, d0, nrows, nxs, seg_zero);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

template <int NDIM, int BS, bool PAD>
static int launch_gen(const DqDecArgs& a, cudaStream_t st) {
    constexpr int G = (128 / BS) > 0 ? (128 / BS) : 1;
    if (NDIM == 1) {
        size_t nblk = (a.d0 + BS - 1) / BS;
        k_dq_decompress_gen<1, BS, PAD><<<(unsigned)((nblk + 127) / 128), 128, 0, st>>>(a);
        count_launch();
    } else {
        size_t smem = (size_t)G * 2 * BS * BS * sizeof(float);
        static std::atomic<unsigned long long> attr{0};
        smem_limit_once(k_dq_decompress_gen<NDIM, BS, PAD>, (int)smem, attr);
        unsigned grid = (unsigned)((a.nunits + G - 1) / G);
        k_dq_decompress_gen<NDIM, BS, PAD><<<grid, G * BS, smem, st>>>(a);
        count_launch();
    }
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

void dq_b8_geometry(DqDecArgs& a, int ndim) {
    a.nxs   = (a.d0 + kDSeg - 1) / kDSeg;
    a.nyb   = (a.d1 + 7) / 8;
    a.nbx8  = (a.d0 + 7) / 8;
    a.ygrp  = 1;
    a.nyb_g = a.nyb;
    unsigned long long nzb = (ndim == 3) ? (a.d2 + 7) / 8 : 1;
    a.nunits = (unsigned long long)a.nxs * (ndim >= 2 ? a.nyb : 1) * nzb;
}

void dq_b8_narrow(DqDecArgs& a, int ndim) {
    if (ndim < 2 || a.nbx8 == 0 || a.nbx8 > 16) return;
    a.ygrp  = 32 / a.nbx8;
    a.nyb_g = (a.nyb + a.ygrp - 1) / a.ygrp;
    const unsigned long long nzb = (ndim == 3) ? (a.d2 + 7) / 8 : 1;
    a.nunits = (unsigned long long)a.nyb_g * nzb;
}

bool dq_b8_vec(const DqDecArgs& a) {
    return (a.d0 % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.codes) & 15u) == 0) &&
           ((reinterpret_cast<uintptr_t>(a.out) & 15u) == 0);
}

bool dq_b8_separable(const DqDecArgs& a, int ndim) {
    return ndim == 3 && dq_b8_vec(a) && a.redo && !a.strict && !a.pad.vals && a.n_outliers * 64 < a.n;
}

// ---- many fields (block size 8, no padding): tasks of (field, unit range), taken one at a time
// by whichever warp is free (`next`: the launch's task counter, zero at launch), so that warps do
// not idle behind uneven tasks.  Per field the result is the single-field kernels'.
__device__ __forceinline__ uint32_t dq_next_task(uint32_t* next) {
    uint32_t t = 0;
    if (lane_id() == 0) t = atomicAdd(next, 1u);
    return __shfl_sync(0xffffffffu, t, 0);
}

template <int NDIM, bool VEC>
__global__ void __launch_bounds__(128, 6)
    k_dq_decompress_b8_batch(const DqDecArgs* __restrict__ args, const BatchTask* __restrict__ tasks, uint32_t ntasks,
                             uint32_t* __restrict__ next) {
    extern __shared__ __align__(16) uint8_t s_dq_dyn[];
    const unsigned wib = threadIdx.x >> 5;
    for (uint32_t t = dq_next_task(next); t < ntasks; t = dq_next_task(next)) {
        const BatchTask tk = tasks[t];  // the field's arguments are read in place (a copy spills)
        dq_b8_units<NDIM, VEC, false, false>(args[tk.field], (uint32_t)tk.u0, (uint32_t)tk.u1, 1u,
                                             reinterpret_cast<DqPlane*>(s_dq_dyn), wib);
    }
}

__global__ void __launch_bounds__(128, 6)
    k_dq_decompress_b8s_batch(const DqDecArgs* __restrict__ args, const BatchTask* __restrict__ tasks, uint32_t ntasks,
                              uint32_t* __restrict__ next) {
    extern __shared__ __align__(16) uint8_t s_dq_dyn[];
    const unsigned wib = threadIdx.x >> 5;
    for (uint32_t t = dq_next_task(next); t < ntasks; t = dq_next_task(next)) {
        const BatchTask tk = tasks[t];
        dq_b8s_units(args[tk.field], (uint32_t)tk.u0, (uint32_t)tk.u1, 1u, reinterpret_cast<DqPlane*>(s_dq_dyn), wib);
    }
}

// Small batches: every class in one launch, the task naming its class (tk.pad, kDqDec*).  A launch per
// class runs them one after another, each too small to fill the GPU, and 3D fields take the wavefront
// pass here (60 mixed fields, 20 M elements of them 3D: 594 -> 343 us).  In large batches (see
// vsz_dbatch_create) the block kernels keep their own launches: one kernel of them all spills (632).
__global__ void __launch_bounds__(128, 5)
    k_dq_decompress_small_batch(const DqDecArgs* __restrict__ args, const BatchTask* __restrict__ tasks, uint32_t ntasks,
                                uint32_t* __restrict__ next) {
    __shared__ W8Codes s_codes[4];
    W8Codes& codes = s_codes[threadIdx.x >> 5];
    for (uint32_t t = dq_next_task(next); t < ntasks; t = dq_next_task(next)) {
        const BatchTask tk = tasks[t];  // the field's arguments are read in place (a copy spills)
        const DqDecArgs& a = args[tk.field];
        const uint32_t u0 = (uint32_t)tk.u0, u1 = (uint32_t)tk.u1;
        switch (tk.pad) {
            case kDqDec1D: dq_b8_units<1, false, false, false>(a, u0, u1, 1u, nullptr, 0); break;
            case kDqDec1D + kDqDecVec: dq_b8_units<1, true, false, false>(a, u0, u1, 1u, nullptr, 0); break;
            case kDqDec2D: dq_b8_units<2, false, false, false>(a, u0, u1, 1u, nullptr, 0); break;
            case kDqDec2D + kDqDecVec: dq_b8_units<2, true, false, false>(a, u0, u1, 1u, nullptr, 0); break;
            case kDqDec3D: dq_w8_units<false>(a, u0, u1, 1u, codes); break;
            default: dq_w8_units<true>(a, u0, u1, 1u, codes); break;
        }
    }
}

// The units the separable pass listed, one CTA per field (tasks carry only the field).
__global__ void __launch_bounds__(128, 6)
    k_dq_decompress_redo_batch(const DqDecArgs* __restrict__ args, const BatchTask* __restrict__ tasks, uint32_t ntasks) {
    extern __shared__ __align__(16) uint8_t s_dq_dyn[];
    const unsigned wib = threadIdx.x >> 5;
    for (uint32_t t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const DqDecArgs& a = args[tasks[t].field];  // read in place: fewer registers than a copy
        dq_b8_units<3, true, false, true>(a, wib, a.redo[0], 4u, reinterpret_cast<DqPlane*>(s_dq_dyn), wib);
    }
}

int launch_dq_decompress_small_batch(const DqDecArgs* args, const BatchTask* tasks, uint32_t ntasks, uint32_t* next,
                                     cudaStream_t st, int num_sms) {
    if (ntasks == 0) return VSZ_OK;
    const uint32_t want = (ntasks + 3) / 4, cap = (uint32_t)num_sms * 5;  // resident CTAs of 4 warps
    k_dq_decompress_small_batch<<<want < cap ? want : cap, 128, 0, st>>>(args, tasks, ntasks, next);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

int launch_dq_decompress_batch(const DqDecArgs* args, const BatchTask* tasks, uint32_t ntasks, int ndim, bool vec,
                               bool sep, uint32_t* next, cudaStream_t st, int num_sms) {
    if (ntasks == 0) return VSZ_OK;
    const uint32_t cap  = (uint32_t)num_sms * 6;  // resident CTAs of 4 warps
    const uint32_t want = (ntasks + 3) / 4;
    const uint32_t grid = want < cap ? want : cap;
    const size_t smem   = (ndim == 3) ? 4 * sizeof(DqPlane) : 0;
    static std::atomic<unsigned long long> attr[8];
    auto go = [&](auto kern, int slot) {
        if (smem > 48 * 1024) smem_limit_once(kern, (int)smem, attr[slot]);
        kern<<<grid, 128, smem, st>>>(args, tasks, ntasks, next);
        count_launch();
    };
    if (sep) go(k_dq_decompress_b8s_batch, 0);
    else if (ndim == 3) vec ? go(k_dq_decompress_b8_batch<3, true>, 1) : go(k_dq_decompress_b8_batch<3, false>, 2);
    else if (ndim == 2) vec ? go(k_dq_decompress_b8_batch<2, true>, 3) : go(k_dq_decompress_b8_batch<2, false>, 4);
    else vec ? go(k_dq_decompress_b8_batch<1, true>, 5) : go(k_dq_decompress_b8_batch<1, false>, 6);
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

int launch_dq_redo_batch(const DqDecArgs* args, const BatchTask* tasks, uint32_t ntasks, cudaStream_t st,
                         int num_sms) {
    if (ntasks == 0) return VSZ_OK;
    const uint32_t cap  = (uint32_t)num_sms * 6;
    const uint32_t grid = ntasks < cap ? ntasks : cap;
    static std::atomic<unsigned long long> attr{0};
    smem_limit_once(k_dq_decompress_redo_batch, (int)(4 * sizeof(DqPlane)), attr);
    k_dq_decompress_redo_batch<<<grid, 128, 4 * sizeof(DqPlane), st>>>(args, tasks, ntasks);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
}

// Fields from this size on check the two-operation dequantization before the separable pass.
constexpr size_t kDqVerifyMin = (size_t)1 << 22;

int launch_dq_decompress(DqDecArgs a, int ndim, int bs, bool force_general, cudaStream_t st, int num_sms) {
    if (a.n == 0) return VSZ_OK;
    if (bs == 8 && !force_general) {
        dq_b8_geometry(a, ndim);
        const bool vec = dq_b8_vec(a);
        if (dq_w8_applies(a, ndim)) {  // small 3D field: the wavefront pass
            dq_w8_geometry(a);
            const long long want = (long long)((a.nunits + 3) / 4), cap = (long long)num_sms * 16;
            const int grid = (int)(want < cap ? want : cap);
            if (vec) k_dq_decompress_w8<true><<<grid, 128, 0, st>>>(a);
            else k_dq_decompress_w8<false><<<grid, 128, 0, st>>>(a);
            count_launch();
            return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
        }
        if (!a.pad.vals && !dq_b8_separable(a, ndim)) dq_b8_narrow(a, ndim);  // the reference-order kernel
        long long want = (long long)((a.nunits + 3) / 4);
        long long cap  = (long long)num_sms * 16;
        int grid = (int)(want < cap ? want : cap);
        if (grid < 1) grid = 1;
        static std::atomic<unsigned long long> attr[12];
        const bool pad = a.pad.vals != nullptr;
        auto go = [&](auto kern, int nd) {
            const size_t smem = (nd == 3) ? 4 * 8 * 8 * 32 * 4 : 0;  // previous plane per warp
            if (smem > 48 * 1024)
                smem_limit_once(kern, (int)smem, attr[(nd - 1) * 4 + (vec ? 1 : 0) + (pad ? 2 : 0)]);
            kern<<<grid, 128, smem, st>>>(a);
            count_launch();
        };
        if (pad) {
            if (ndim == 3) vec ? go(k_dq_decompress_b8<3, true, true>, 3) : go(k_dq_decompress_b8<3, false, true>, 3);
            else if (ndim == 2) vec ? go(k_dq_decompress_b8<2, true, true>, 2) : go(k_dq_decompress_b8<2, false, true>, 2);
            else vec ? go(k_dq_decompress_b8<1, true, true>, 1) : go(k_dq_decompress_b8<1, false, true>, 1);
        } else if (dq_b8_separable(a, ndim)) {
            // separable pass, then the reference-order kernel over the units it listed.  A large
            // field first checks the cheaper dequantization (a few microseconds, all SMs).
            const bool verify = a.consts_rw && a.n >= kDqVerifyMin;
            if (!a.redo_cleared && cudaMemsetAsync(a.redo, 0, (verify ? 3 : 1) * sizeof(uint32_t), st) != cudaSuccess)
                return VSZ_ERR_CUDA;
            if (verify) {
                k_dq_mul_verify<<<(unsigned)num_sms * 4, 256, 0, st>>>(a.consts_rw, a.redo, a.dq_cache);
                count_launch();
            }
            go(k_dq_decompress_b8s, 3);
            go(k_dq_decompress_b8<3, true, false, true>, 3);
        } else {
            if (ndim == 3) vec ? go(k_dq_decompress_b8<3, true>, 3) : go(k_dq_decompress_b8<3, false>, 3);
            else if (ndim == 2) vec ? go(k_dq_decompress_b8<2, true>, 2) : go(k_dq_decompress_b8<2, false>, 2);
            else vec ? go(k_dq_decompress_b8<1, true>, 1) : go(k_dq_decompress_b8<1, false>, 1);
        }
        return cudaGetLastError() == cudaSuccess ? VSZ_OK : VSZ_ERR_CUDA;
    }
    a.nxs = (a.d0 + kDSeg - 1) / kDSeg;
    a.nbx = (a.d0 + bs - 1) / bs;
    a.nyb = (a.d1 + bs - 1) / bs;
    unsigned long long nzb = (ndim == 3) ? (a.d2 + bs - 1) / bs : 1;
    a.nunits = (unsigned long long)a.nbx * a.nyb * nzb;
    auto go = [&](auto bs_c) -> int {
        constexpr int B = decltype(bs_c)::value;
        if (a.pad.vals) {
            if (ndim == 3) return launch_gen<3, B, true>(a, st);
            if (ndim == 2) return launch_gen<2, B, true>(a, st);
            return launch_gen<1, B, true>(a, st);
        }
        if (ndim == 3) return launch_gen<3, B, false>(a, st);
        if (ndim == 2) return launch_gen<2, B, false>(a, st);
        return launch_gen<1, B, false>(a, st);
    };
    switch (bs) {
        case 8: return go(std::integral_constant<int, 8>{});
        case 16: return go(std::integral_constant<int, 16>{});
        case 32: return go(std::integral_constant<int, 32>{});
        case 64: return go(std::integral_constant<int, 64>{});
        default: return VSZ_ERR_UNSUPPORTED;
    }
}

}  // namespace vsz
