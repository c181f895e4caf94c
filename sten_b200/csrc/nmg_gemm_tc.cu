// Two-pass tensor-core matmul for large token counts: expand once, multiply at dense rate.
//
// The n:m blocks of the format run along the output-feature axis, so the tensor cores execute the dense product
// whatever the kernel does; what differs is how often a weight tile is expanded.  The fused kernel (nmg_spmm_tc.cu)
// expands every tile once per 256-token tile of the output, which costs about a third of its main loop; that is the
// right trade for few tokens, where the compressed weight is the HBM traffic.  With thousands of tokens it is cheaper
// to expand the weight ONCE into a transient dense 16-bit matrix in the caller's workspace (an HBM-bound pass of
// about 2.5 bytes per weight element) and run a plain TMA-fed tcgen05 matmul over it:
//
//   expand_dense_kernel   (val, idx) -> dense W [M][K] (forward) or W^T [K][M] (transposed product), 16-bit; fp32
//                         weights become three bf16 planes (exact hi / mid / lo split).  Works for every (n, m, g).
//   split_rows_kernel     fp32 only, first: the activation's planes (split_columns_kernel from a K-major activation).
//   expand_rows_kernel    the same for W with n <= 2 and chunks of whole 16-byte pieces, the usual weight: whole rows.
//   gemm_tc_kernel        persistent, one CTA per SM, in pairs but for 16-bit outputs of one feature tile.  Warp 0 issues the TMA loads of both operands, warp 1 the
//                         MMAs (128 x 256 x 16, fp32 accumulators in TMEM), warps 4..11 drain accumulators.  16-bit
//                         mode double-buffers the accumulator (2 x 256 TMEM columns) so that the drain of one tile
//                         overlaps the MMAs of the next; in fp32 mode a buffer is a chunk of k-blocks, and
//                         the drain warps keep the running sum of the chunks in registers.
//
// All device-side waits are bounded: a wait that runs out sets the status word and the role leaves its loop; the
// CTA then meets at the common exit where TMEM is released.
#include <cstdlib>

#include "nmg_expand.cuh"
#include "nmg_spmm_simt.cuh"
#include "nmg_tc_common.cuh"
#include "nmg_tiles.h"

namespace nmg {

// =========================================================================================================
// Expansion pass
// =========================================================================================================
// Move `cnt` (1..8) consecutive elements of a shared-memory line to the destination planes and clear them in shared
// memory.  VEC: cnt == 8 and both sides are 16-byte aligned.
// PLAIN (fp32 only): the destination is an fp32 matrix, not three bf16 planes (the densifier's use of this pass).
template <typename T, bool VEC, bool PLAIN> __device__ __forceinline__ void expand_flush(const ExpandParams &p, T *line, int64_t off, int cnt) {
    if constexpr (sizeof(T) == 4 && PLAIN) {
        float *d = static_cast<float *>(p.dst) + off;
        if (VEC) {
            *reinterpret_cast<float4 *>(d) = *reinterpret_cast<const float4 *>(line);
            *reinterpret_cast<float4 *>(d + 4) = *reinterpret_cast<const float4 *>(line + 4);
            *reinterpret_cast<float4 *>(line) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4 *>(line + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            for (int i = 0; i < cnt; i++) { d[i] = line[i]; line[i] = 0.f; }
        }
    } else if constexpr (sizeof(T) == 2) {
        T *d = static_cast<T *>(p.dst) + off;
        if (VEC) {
            *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(line);
            *reinterpret_cast<uint4 *>(line) = make_uint4(0, 0, 0, 0);
        } else {
            for (int i = 0; i < cnt; i++) { d[i] = line[i]; line[i] = DT<T>::from_f32(0.f); }
        }
    } else {
        __nv_bfloat16 *d = static_cast<__nv_bfloat16 *>(p.dst) + off;
        if (VEC) {
            const float4 a = *reinterpret_cast<const float4 *>(line), b = *reinterpret_cast<const float4 *>(line + 4);
            *reinterpret_cast<float4 *>(line) = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4 *>(line + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t w[3][4];
            split3_pair(a.x, a.y, w[0][0], w[1][0], w[2][0]);
            split3_pair(a.z, a.w, w[0][1], w[1][1], w[2][1]);
            split3_pair(b.x, b.y, w[0][2], w[1][2], w[2][2]);
            split3_pair(b.z, b.w, w[0][3], w[1][3], w[2][3]);
#pragma unroll
            for (int c = 0; c < 3; c++) *reinterpret_cast<uint4 *>(d + c * p.plane_elems) = make_uint4(w[c][0], w[c][1], w[c][2], w[c][3]);
        } else {
            for (int i = 0; i < cnt; i++) {
                __nv_bfloat16 x[3];
                split3(line[i], x);
                line[i] = 0.f;
                for (int c = 0; c < 3; c++) d[c * p.plane_elems + i] = x[c];
            }
        }
    }
}

// Work item = (column chunk kc, R consecutive row-blocks).  The item's dense tile lives in shared memory, in the
// orientation of the destination (TR = false: lines are weight rows, cc columns long; TR = true: lines are weight
// columns, R * m rows long).  It starts as zeros; the item's non-zeros are scattered into it straight from global
// memory (coalesced reads of val and idx, one thread per slot), and the tile is then moved out with 16-byte accesses
// that also restore the zeros.
// N_ = n for the vectorised scatter (1 or 2), 0 for the generic one.
template <typename T, bool TR, int N_, bool PLAIN = false>
__global__ void __launch_bounds__(EXPAND_THREADS) expand_dense_kernel(const ExpandParams prm) {
    extern __shared__ __align__(16) char smem[];
    constexpr bool VEC_OK = N_ > 0;
    const int n = N_ > 0 ? N_ : prm.n, m = prm.m, g = prm.g, cc = prm.cc, R = prm.R, pitch = prm.pitch;
    const int lines = TR ? cc : R * m;
    T *tile = reinterpret_cast<T *>(smem);                                  // [lines][pitch]
    int8_t *ord = reinterpret_cast<int8_t *>(tile + (size_t)lines * pitch);  // [C][n]
    // The matmul kernel that follows may become resident and run its prologue while this grid drains, and reads nothing this grid
    // writes before its dependents_wait; this one's prologue runs beside the kernel ahead.
    dependents_launch();
    for (int i = threadIdx.x; i < prm.C * n; i += EXPAND_THREADS) ord[i] = prm.order[i];  // a constant of the library
    for (int i = threadIdx.x; i < lines * pitch; i += EXPAND_THREADS) tile[i] = DT<T>::from_f32(0.f);
    dependents_wait();

    const T *val = static_cast<const T *>(prm.val);
    const int64_t groups = (prm.nb + R - 1) / R;
    const int64_t items = groups * prm.nc;
    const int vec_per_line = pitch / 8;  // pitch is a multiple of 8

    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const int64_t kc = item / groups, mb0 = (item - kc * groups) * R;
        const int rj = (int)(prm.nb - mb0 < R ? prm.nb - mb0 : R);  // row-blocks in this item
        __syncthreads();  // the tile is all zeros again
        expand_scatter_item<T, TR, N_>(prm, tile, ord, kc, mb0, rj);
        __syncthreads();
        const int64_t col0 = kc * cc, r0 = mb0 * m;
        // line l, elements e .. e+7 -> dst[(TR ? col0 + l : r0 + l)][(TR ? r0 : col0) + e]
        const int64_t line_lim = TR ? prm.K - col0 : prm.M - r0;   // lines inside the weight
        const int64_t elem_lim = TR ? prm.M - r0 : prm.K - col0;   // elements of a line inside the weight
        const int ne = TR ? rj * m : cc;                            // elements of a line this item owns
        const bool aligned = ((TR ? r0 : col0) % 8) == 0;           // ld is a multiple of 8, the workspace is 256-byte aligned
        for (int v = threadIdx.x; v < lines * vec_per_line; v += EXPAND_THREADS) {
            const int l = v / vec_per_line, e = (v - l * vec_per_line) * 8;
            T *line = tile + l * pitch + e;
            if (l >= line_lim || e >= ne || e >= elem_lim) {  // outside the weight: nothing to store, but keep the tile clean
                if constexpr (sizeof(T) == 2) *reinterpret_cast<uint4 *>(line) = make_uint4(0, 0, 0, 0);
                else { *reinterpret_cast<float4 *>(line) = make_float4(0.f, 0.f, 0.f, 0.f); *reinterpret_cast<float4 *>(line + 4) = make_float4(0.f, 0.f, 0.f, 0.f); }
                continue;
            }
            const int64_t off = ((TR ? col0 : r0) + l) * prm.ld + (TR ? r0 : col0) + e;
            // A full vector may run past the item's elements only into the row's padding (last chunk / last group:
            // ld = round_up(extent, 8)), never into elements another item owns.
            if (aligned && (e + 8 <= ne || ne >= elem_lim)) {
                expand_flush<T, true, PLAIN>(prm, line, off, 8);
            } else {
                int cnt = ne - e < 8 ? ne - e : 8;
                if (elem_lim - e < cnt) cnt = (int)(elem_lim - e);
                expand_flush<T, false, PLAIN>(prm, line, off, cnt);
                // elements of the vector past cnt were never written by this item's valid slots; clear them anyway
                for (int i = cnt; i < 8; i++) line[i] = DT<T>::from_f32(0.f);
            }
        }
    }
}

// The same pass for the common case: rows in the weight's orientation, n <= 2, chunks of whole 16-byte pieces.  HBM-bound work
// (4096 x 4096 bf16 2:4: 25 MB in, 34 MB out, 9 us at the copy rate) that the general kernel did in 19 us: its items were one
// chunk wide (192-byte pieces of a row for 2:4), every piece cost divisions and bounds arithmetic, and a CTA's loads waited for
// its stores.  Here an item is R row-blocks x Q chunks, about 512 columns of as many rows as give every thread one piece of
// eight slots, so that rows leave in whole lines; what a thread does with its piece -- row-block, pattern rows, place in the
// tile -- is the same for every item and computed once; the next item's loads are in flight while a tile is moved out.
// STRIPS (PLAIN only): rows of the destination are not 16-byte aligned.  A kernel of its own: together the two took 64 to 78 registers for
// 16-bit n = 2, as the compiler pleased, and with 78 three CTAs fit an SM where four do: densify 8192 x 8192 bf16 38.0 .. 39.9 -> 34.5 us.
template <typename T, int N_, bool PLAIN, bool STRIPS>
__global__ void __launch_bounds__(EXPAND_THREADS) expand_rows_kernel(const ExpandParams prm) {
    extern __shared__ __align__(16) char smem[];
    const int m = prm.m, g = prm.g, cc = prm.cc, R = prm.R, Q = prm.Q, cols = Q * cc, rows = R * m;
    T *tile = reinterpret_cast<T *>(smem);                                 // [rows][cols]
    int8_t *ord = reinterpret_cast<int8_t *>(tile + (size_t)rows * cols);  // [C][n]
    dependents_launch();                                                   // see expand_dense_kernel

    constexpr int VL = N_ * (int)sizeof(T) / 2;  // 16-byte loads of values per 8 slots
    const int per_chunk = R * cc / 8, tid = (int)threadIdx.x;
    const bool has = tid < Q * per_chunk;
    const int uq = tid / per_chunk, e8 = (tid - uq * per_chunk) * 8, uj = e8 / cc, uslot = e8 - uj * cc;  // chunk, row-block, slot in its tile
    const T *val = static_cast<const T *>(prm.val);
    const int groups = (int)((prm.nb + R - 1) / R), spans = (int)((prm.nc + Q - 1) / Q);
    const int64_t items = (int64_t)groups * spans;
    uint4 iv, vv[VL];
    auto load = [&](int64_t item) {
        const int span = (int)(item / groups), grp = (int)(item - (int64_t)span * groups);
        iv = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);  // column -1: no slot
        if (!has || span * Q + uq >= prm.nc || grp * R + uj >= prm.nb) return;
        const int64_t slot = ((int64_t)(span * Q + uq) * prm.nb + grp * R + uj) * cc + uslot;
        iv = *reinterpret_cast<const uint4 *>(prm.idx + slot);
#pragma unroll
        for (int i = 0; i < VL; i++) vv[i] = reinterpret_cast<const uint4 *>(val + slot * N_)[i];
    };
    for (int i = tid; i < prm.C * N_; i += EXPAND_THREADS) ord[i] = prm.order[i];
    for (int i = tid; i < rows * cols * (int)sizeof(T) / 16; i += EXPAND_THREADS) reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0, 0, 0, 0);
    dependents_wait();
    if (blockIdx.x < items) load(blockIdx.x);
    __syncthreads();
    const bool same_pattern = (g & 7) == 0;  // 8 consecutive slots then belong to one pattern
    T *ubase = tile + uj * m * cols + uq * cc;
    int urow[N_];
#pragma unroll
    for (int t = 0; t < N_; t++) urow[t] = (same_pattern && has) ? (int)ord[(uslot / g) * N_ + t] * cols : 0;
    constexpr int V = (PLAIN || sizeof(T) == 2) ? 16 / (int)sizeof(T) : 8;  // elements per move
    const int vpl = cols / V, total = rows * vpl, dl = EXPAND_THREADS / vpl, de = EXPAND_THREADS - dl * vpl;
    const int l0 = tid / vpl, e0 = tid - l0 * vpl;

    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const int16_t *ci = reinterpret_cast<const int16_t *>(&iv);
        const T *vals = reinterpret_cast<const T *>(vv);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int c = ci[k];
            if ((unsigned)c >= (unsigned)cc) continue;  // no slot, or a malformed index: never dereferenced
#pragma unroll
            for (int t = 0; t < N_; t++) ubase[(same_pattern ? urow[t] : (int)ord[((uslot + k) / g) * N_ + t] * cols) + c] = vals[k * N_ + t];
        }
        __syncthreads();
        if (item + gridDim.x < items) load(item + gridDim.x);
        const int span = (int)(item / groups), grp = (int)(item - (int64_t)span * groups);
        const int64_t r0 = (int64_t)grp * rows, c0 = (int64_t)span * cols;
        const int row_lim = (int)(prm.M - r0 < rows ? prm.M - r0 : rows), col_lim = (int)(prm.K - c0 < cols ? prm.K - c0 : cols);
        if constexpr (STRIPS) {  // rows of the destination are not 16-byte aligned: neighbouring threads store neighbouring elements
            const int dle = EXPAND_THREADS / cols, dee = EXPAND_THREADS - dle * cols;
            for (int v = tid, l = tid / cols, e = tid - l * cols; v < rows * cols; v += EXPAND_THREADS) {
                if (l < row_lim && e < col_lim) static_cast<T *>(prm.dst)[(r0 + l) * prm.ld + c0 + e] = tile[v];
                tile[v] = DT<T>::from_f32(0.f);
                l += dle;
                if ((e += dee) >= cols) { e -= cols; l++; }
            }
            __syncthreads();
        } else {
            // A vector that starts inside the weight may run past K only into the row's padding (ld = round_up(K, 8)).
            // Pieces in flight per thread against registers, us with 1 / 2: densify bf16 2:8 8192 x 8192 34.4 / 35.0, f16 1:4 4096 x 4096 9.7 / 9.2;
            // the pass and the matmul behind it, bf16 1:8 4096 x 4096, 4096 tokens 104.1 / 105.1.
            constexpr int FLUSH = PLAIN && sizeof(T) == 2 && N_ == 1 ? 2 : 1;
#pragma unroll FLUSH
            for (int v = tid, l = l0, e = e0; v < total; v += EXPAND_THREADS) {
                T *line = tile + v * V;
                const int64_t off = (r0 + l) * prm.ld + c0 + e * V;
                const bool inside = l < row_lim && e * V < col_lim;
                if constexpr (V * sizeof(T) == 16) {
                    if (inside) *reinterpret_cast<uint4 *>(static_cast<T *>(prm.dst) + off) = *reinterpret_cast<const uint4 *>(line);
                    *reinterpret_cast<uint4 *>(line) = make_uint4(0, 0, 0, 0);
                } else {
                    if (inside) expand_flush<T, true, PLAIN>(prm, line, off, V);
                    else {
                        reinterpret_cast<uint4 *>(line)[0] = make_uint4(0, 0, 0, 0);
                        reinterpret_cast<uint4 *>(line)[1] = make_uint4(0, 0, 0, 0);
                    }
                }
                l += dl;
                if ((e += de) >= vpl) { e -= vpl; l++; }
            }
            __syncthreads();
        }
    }
}
// R and Q of the rows kernel, false when it does not serve the weight
static bool expand_rows_plan(const Geo &geo, size_t es, int *R, int *Q, size_t *smem) {
    if (geo.n < 1 || geo.n > 2 || geo.cc % 8 != 0 || geo.nb > 0x3fffffff || geo.nc > 0x3fffffff) return false;
    int q = 512 / geo.cc;
    if (q < 1) q = 1;
    if (q > geo.nc) q = (int)geo.nc;
    const int cols = q * geo.cc;
    int r = EXPAND_THREADS * 8 / cols;                                  // one piece per thread
    const int fit = (int)(32 * 1024 / ((size_t)geo.m * cols * es));     // seven CTAs per SM
    if (r > fit) r = fit;
    if (r < 1) r = 1;
    const size_t bytes = (size_t)r * geo.m * cols * es;
    if (bytes > 64 * 1024 || r * cols / 8 > EXPAND_THREADS) return false;
    *R = r; *Q = q;
    *smem = bytes + (size_t)geo.C * geo.n + 16;
    return true;
}

static int expand_pitch(const Geo &geo, bool tr, int R) { return (int)round_up(tr ? (int64_t)R * geo.m : (int64_t)geo.cc, 8) + 8; }
static size_t expand_smem_bytes(const Geo &geo, size_t es, bool tr, int R) {
    const size_t lines = tr ? (size_t)geo.cc : (size_t)R * geo.m;
    return lines * expand_pitch(geo, tr, R) * es + (size_t)geo.C * geo.n + 16;
}
static int expand_rows_per_item(const Geo &geo, size_t es, bool tr) {
    int R = 64 / geo.m;
    if (R < 1) R = 1;
    while (R > 1 && expand_smem_bytes(geo, es, tr, R) > 64 * 1024) R >>= 1;
    return R;
}

// =========================================================================================================
// fp32 activations: three bf16 planes and a factor per row
// =========================================================================================================
struct SplitParams {
    const float *src;
    __nv_bfloat16 *dst;     // [SPLIT_PLANES][rows][ld]
    float *factors;         // [rows] TINY_FACTOR for rows split times TINY_SCALE; anything else counts as one (a row of zeros may have no entry)
    int64_t rows, cols, ld_src, ld;
};
__device__ __forceinline__ void store_split(const SplitParams &p, int64_t r, int64_t c, const float (&f)[8], float scale) {
    uint4 w[SPLIT_PLANES];
    split3_pair(f[0] * scale, f[1] * scale, w[0].x, w[1].x, w[2].x);
    split3_pair(f[2] * scale, f[3] * scale, w[0].y, w[1].y, w[2].y);
    split3_pair(f[4] * scale, f[5] * scale, w[0].z, w[1].z, w[2].z);
    split3_pair(f[6] * scale, f[7] * scale, w[0].w, w[1].w, w[2].w);
    __nv_bfloat16 *d = p.dst + r * p.ld + c;
#pragma unroll
    for (int t = 0; t < SPLIT_PLANES; t++) *reinterpret_cast<uint4 *>(d + t * p.rows * p.ld) = w[t];
}

// One row per CTA, or one per warp where a warp's registers hold it (ROWS = 4).  HBM-bound: 4 bytes read and 6 written per value.  The
// part that the registers hold nearly always settles that the row is not tiny; only if it does not is the rest read twice.
constexpr int SPLIT_THREADS = 128;
template <int ROWS> __global__ void __launch_bounds__(SPLIT_THREADS) split_rows_kernel(const SplitParams p) {
    dependents_launch();
    dependents_wait();
    constexpr int LANES = SPLIT_THREADS / ROWS, HELD = 4;
    const int sub = threadIdx.x / LANES, tid = threadIdx.x - sub * LANES;
    const int64_t r = (int64_t)blockIdx.x * ROWS + sub;
    if (ROWS > 1 && r >= p.rows) return;  // whole warps
    const float *row = p.src + r * p.ld_src;
    const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
    auto load = [&](int64_t c, float (&f)[8]) {
        if (vec && c + 8 <= p.cols) {
            const float4 a = *reinterpret_cast<const float4 *>(row + c), b = *reinterpret_cast<const float4 *>(row + c + 4);
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) f[i] = c + i < p.cols ? row[c + i] : 0.f;
        }
    };
    auto any = [&](bool v) -> bool { return ROWS > 1 ? __any_sync(0xffffffffu, v) : __syncthreads_or(v); };
    float held[HELD][8];
    bool big = false;
#pragma unroll
    for (int h = 0; h < HELD; h++) {
        const int64_t c = ((int64_t)h * LANES + tid) * 8;
        if (c >= p.ld) break;
        load(c, held[h]);
    }
#pragma unroll
    for (int h = 0; h < HELD; h++) {
        const int64_t c = ((int64_t)h * LANES + tid) * 8;
        if (c >= p.ld) break;
#pragma unroll
        for (int i = 0; i < 8; i++) big |= not_tiny(held[h][i]);
    }
    big = any(big);
    constexpr int64_t FIRST = (int64_t)HELD * LANES * 8;  // not held from here on
    for (int64_t c0 = FIRST; c0 < p.ld && !big; c0 += LANES * 8) {
        float f[8];
        bool b = false;
        if (c0 + tid * 8 < p.ld) {
            load(c0 + tid * 8, f);
#pragma unroll
            for (int i = 0; i < 8; i++) b |= not_tiny(f[i]);
        }
        big = any(b);
    }
    if (tid == 0) p.factors[r] = big ? 1.f : TINY_FACTOR;
    const float scale = big ? 1.f : TINY_SCALE;
#pragma unroll
    for (int h = 0; h < HELD; h++) {
        const int64_t c = ((int64_t)h * LANES + tid) * 8;
        if (c >= p.ld) break;
        store_split(p, r, c, held[h], scale);
    }
    for (int64_t c = FIRST + tid * 8; c < p.ld; c += LANES * 8) {
        float f[8];
        load(c, f);
        store_split(p, r, c, f, scale);
    }
}

// The same from a K-major activation src[red][ld_src >= tokens], transposed through a 64 x 32 tile on the way.  A CTA looks at the rest of
// a token's row only if its own part holds values of it and none that settles the matter.
constexpr int COLS_THREADS = 256, COLS_RED = 64, COLS_WARPS = COLS_THREADS / 32;
__global__ void __launch_bounds__(COLS_THREADS) split_columns_kernel(const SplitParams p) {
    __shared__ float tile[COLS_RED][33];                                        // [reduction][token]
    __shared__ __align__(16) unsigned found_big[COLS_WARPS], found_any[COLS_WARPS];  // bits by token
    dependents_launch();
    dependents_wait();
    const int64_t k0 = (int64_t)blockIdx.x * COLS_RED, t0 = (int64_t)blockIdx.y * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t = t0 + lane;
    auto at = [&](int64_t k) -> float { return k < p.cols && t < p.rows ? p.src[k * p.ld_src + t] : 0.f; };
    auto all = [](const unsigned *found) -> unsigned {
        const uint4 a = reinterpret_cast<const uint4 *>(found)[0], b = reinterpret_cast<const uint4 *>(found)[1];
        return a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w;
    };
    static_assert(COLS_WARPS == 8, "two 16-byte reads");
    bool b = false, any = false;
#pragma unroll
    for (int i = 0; i < COLS_RED / COLS_WARPS; i++) {
        const float v = at(k0 + warp + i * COLS_WARPS);
        tile[warp + i * COLS_WARPS][lane] = v;
        b |= not_tiny(v);
        any |= v != 0.f;
    }
    const unsigned bm = __ballot_sync(0xffffffffu, b), am = __ballot_sync(0xffffffffu, any);
    if (lane == 0) {
        found_big[warp] = bm;
        found_any[warp] = am;
    }
    __syncthreads();
    unsigned big = all(found_big);
    const unsigned own = all(found_any);
    for (int64_t k = 0; k < p.cols && (own & ~big); k += COLS_RED) {  // the same for all threads
        b = false;
#pragma unroll
        for (int i = 0; i < COLS_RED / COLS_WARPS; i++) b |= not_tiny(at(k + warp + i * COLS_WARPS));
        const unsigned m = __ballot_sync(0xffffffffu, b);
        __syncthreads();  // what was found before has been read
        if (lane == 0) found_big[warp] = m;
        __syncthreads();
        big |= all(found_big);
    }
    if (threadIdx.x < 32 && t < p.rows && ((own >> lane) & 1)) p.factors[t] = ((big >> lane) & 1) ? 1.f : TINY_FACTOR;  // CTAs that write agree
    const int r = threadIdx.x >> 3, c8 = (threadIdx.x & 7) * 8;  // token within the tile, reduction offset
    if (t0 + r < p.rows && k0 + c8 < p.ld) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = tile[c8 + i][r];
        store_split(p, t0 + r, k0 + c8, f, ((own & ~big) >> r) & 1 ? TINY_SCALE : 1.f);
    }
}

// =========================================================================================================
// Dense-operand matmul
// =========================================================================================================
static_assert(TILE_COLS == TC_BN, "one accumulator");
constexpr int GEMM_DRAIN_WARPS = 8;   // two per TMEM lane quarter, each takes half of the accumulator's columns
constexpr int GEMM_THREADS = 32 * (4 + GEMM_DRAIN_WARPS);  // TMA warp, MMA warp, two idle ones, drain warps
constexpr int GEMM_RING_BYTES = TC_STAGES * (TC_A_BYTES + TC_B_BYTES);  // 192 KB of operand stages in either mode

constexpr int GEMM_MAX_OUTS = 8;
struct GemmParams {
    const void *bias;  // [out_feats] or NULL
    void *outs[GEMM_MAX_OUTS];  // the result is written to every one of these (same shape and pitch): outs[0] is the
    int n_out;                  // caller's buffer, the others are typically the same buffer on peer GPUs
    void *mc_out;               // NVSwitch multicast address mapping onto all of outs[], or NULL: one multimem.st reaches every GPU
    const void *residual;       // added after the activation, same orientation as the output, or NULL
    int64_t ld_res;
    int act;                    // NMG_EPI_NONE / NMG_EPI_GELU applied to (product + bias)
    int bias_cols;              // bias runs along the accumulator's columns ("tokens" below) instead of its rows
    int out_tma;                // staged output with one destination: the staging tile leaves as one tiled bulk store per group
    int res_vec;                // staged output: the residual is read in the same 16-byte pieces as the output is written
    int64_t out_feats, red, ntok, ld_out;
    int out_token_major;
    int out_staged;    // feature-major output whose rows are 16-byte aligned: go through the staging tile
    int out_tm_vec;    // token-major output (and residual) whose rows are 16-byte aligned: transposed in the staging tile, 16-byte stores
    GemmTiles tiles;       // one CTA per tile of 128 features, or a pair per 256
    int band;              // width of the tile order's bands, in feature tiles
    unsigned *wave_ctr;    // zeroed counter for the producers' soft rendezvous before every tile, or NULL
    const float *factors;  // fp32: of the activation's rows, see SplitParams
    int chunk_kb;          // fp32: k-blocks per chunk of the accumulator, see tc_dense_gemm
    int a_rows, b_rows;                // rows of a plane
    int *status;
};
constexpr int GEMM_STAGING_BYTES = GEMM_DRAIN_WARPS * 4096;  // per drain warp: 32 feature rows x 128 bytes

struct GemmMaps {
    CUtensorMap a;       // row operand, its planes below one another, box 64 x 128, 128-byte swizzle
    CUtensorMap b;       // column operand, box 64 x bn (64 x bn / 2 for CTA pairs)
    CUtensorMap b_tail;  // the same with the box of the narrow tiles
    CUtensorMap out;     // out_tma: the output, box 128 bytes x 32 rows, 128-byte swizzle (fp32: 64 bytes, 64-byte swizzle)
};

// PAIR = false: one CTA per 128-feature x 256-token tile.
// PAIR = true: two CTAs of a cluster share a 256-feature x 256-token tile.  Each loads the weight rows
// of its own 128 features and only half of the activation tile (128 tokens); the MMA (cta_group::2, M = 256, issued by the
// even CTA) reads both halves from both shared memories.  An SM then takes in 32 KB per 64 reduction elements instead of
// 48 KB, which is what keeps the tensor core fed from L2.  full[s] lives in the even ("leader") CTA and receives the TMA
// bytes of both; empty[s] and acc_full[b] exist in both CTAs and are signalled by multicast commits; acc_free[b] lives in
// the leader and collects the drain warps of both CTAs.  No load is multicast.
// fp32 (always pairs): a stage is one k-block of all six planes, 96 KB, and its six products run from it (a stage per product, 48 KB per
// 512 clocks and SM, is over what L2 delivers).
// TMA_OUT = true: the one-destination staged output, leaving as tiled bulk stores; only that output path is compiled,
// which keeps the drain warps' code and register needs small.  TMA_OUT = false: every other output form.
template <typename T, bool PAIR, bool TMA_OUT>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_tc_kernel(const GemmParams prm, const __grid_constant__ GemmMaps maps) {
    constexpr bool SPLIT = sizeof(T) == 4;
    constexpr int TERMS = SPLIT ? SPLIT_TERMS : 1;
    using E = typename TcMode<T>::elem;
    static_assert(PAIR || !SPLIT, "fp32 runs on CTA pairs");
    constexpr int NBUF = 2;  // accumulator tiles in flight between the MMA issuer and the drain warps
    constexpr uint32_t TMEM_COLS = NBUF * TC_ACC_COLS;
    constexpr int PLANES = SPLIT ? SPLIT_PLANES : 1;
    constexpr int B_BYTES = PAIR ? TC_B_BYTES / 2 : TC_B_BYTES;  // room of one plane; the widest tile fills it
    constexpr int OFF_B = PLANES * TC_A_BYTES, STAGE_BYTES = OFF_B + PLANES * B_BYTES;
    constexpr int STAGES = GEMM_RING_BYTES / STAGE_BYTES;  // 4, 6 for pairs, 2 for fp32
    constexpr int TILE_FEATS = PAIR ? 2 * TC_BM : TC_BM;

    extern __shared__ char smem_raw[];
    char *smem = reinterpret_cast<char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    char *staging = smem + GEMM_RING_BYTES;
    char *misc = staging + GEMM_STAGING_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(misc);   // pairs: meaningful in the leader only
    uint64_t *empty = full + STAGES;
    uint64_t *acc_full = empty + STAGES;  // [2] MMA issuer -> drain warps: unit complete in accumulator b
    uint64_t *acc_free = acc_full + 2;    // [2] drain warps -> MMA issuer: accumulator b may be overwritten (pairs: leader only)
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 192);
    static_assert((2 * STAGES + 4) * 8 <= 192, "barrier block too small");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    const bool leader = rank == 0;
    const int unit_id = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;      // CTA (or pair) index
    const int nunits = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    // A "unit" is what the MMA issuer hands to the drain warps: a whole tile (16-bit) or a chunk of k-blocks (fp32).
    const int ntiles = prm.tiles.count(), nwide = prm.tiles.wide();
    const int my_tiles = (unit_id < ntiles) ? (ntiles - unit_id + nunits - 1) / nunits : 0;
    const int nkb = (int)((prm.red + TC_BK - 1) / TC_BK);  // iterations per tile
    const int chunk_it = SPLIT ? prm.chunk_kb : nkb;
    const int nchunks = (nkb + chunk_it - 1) / chunk_it;

    dependents_launch();
    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_free[b], GEMM_DRAIN_WARPS * (PAIR ? 2 : 1));  // lane 0 of each drain warp (of both CTAs)
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        if constexpr (PAIR) tmem_alloc_pair(tmem_slot, TMEM_COLS);
        else tmem_alloc(tmem_slot, TMEM_COLS);
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // barriers of both CTAs are initialised before anyone arrives remotely
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t full_leader = PAIR ? map_to_rank(smem_u32(&full[0]), 0) : 0u;
    const uint32_t acc_free_leader = PAIR ? map_to_rank(smem_u32(&acc_free[0]), 0) : 0u;

    auto wait = [&](uint64_t *bar, uint32_t parity, int code) -> bool {
        if constexpr (PAIR) return mbar_wait_cluster_bounded(bar, parity, prm.status, code);
        else return mbar_wait_bounded(bar, parity, prm.status, code);
    };
    auto narrow = [&](int ti) -> bool { return PAIR && unit_id + ti * nunits >= nwide; };
    auto tile_origin = [&](int ti, int &feat0, int &tok0, int &bn) {  // feat0: first feature of THIS CTA's 128 rows; bn: columns
        int tile_f, tile_t;
        const bool nar = narrow(ti);
        tile_of_cta(unit_id + ti * nunits - (nar ? nwide : 0), nar ? prm.tiles.f_narrow : prm.tiles.f_wide, nar ? prm.tiles.t_narrow : prm.tiles.t_wide, tile_f, tile_t,
                    prm.band);
        bn = !PAIR ? TC_BN : nar ? prm.tiles.bn_tail : prm.tiles.bn;
        feat0 = (tile_f + (nar ? prm.tiles.f_wide : 0)) * TILE_FEATS + (int)rank * TC_BM;
        tok0 = tile_t * bn;
    };

    // fp32: the running sums take 128 registers of a drain warp.  Shares of the launch's 384 x 168: 128 x 56 + 256 x 224.
    if (warp < 4) {
    if constexpr (SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        // The warp stays converged and issues under elect_one (see there).
        int it = 0;
        bool ok = true;
        // Everything this kernel reads that an earlier kernel of the stream wrote (the expanded weight, the
        // activations) arrives through the loads below: wait here for the preceding grid to complete and flush.
        dependents_wait();
        unsigned arrivals = 0;
        for (int ti = 0; ti < my_tiles && ok; ti++) {
            int feat0, tok0, bn;
            tile_origin(ti, feat0, tok0, bn);
            const CUtensorMap *bmap = narrow(ti) ? &maps.b_tail : &maps.b;
            if (prm.wave_ctr && ti > 0) {
                // CTAs whose tiles share operand panels read them from HBM once only while they stream through the
                // reduction in step; left alone they drift apart over the waves (measured: 2.2 MB of DRAM reads per
                // 256 x 256 x 16384 tile in the first dozen waves, 3.9 MB averaged over 55).  So the producers meet,
                // softly, before each tile: everyone that has a tile ti counts in.
                const int left = ntiles - ti * nunits;
                arrivals += (unsigned)((left < nunits ? left : nunits) * (PAIR ? 2 : 1));
                if (lane == 0) soft_rendezvous(prm.wave_ctr, arrivals, (uint64_t)nkb * 40);
                __syncwarp();
            }
            for (int kb = 0; kb < nkb; kb++, it++) {
                const int s = it % STAGES;
                const uint32_t ph = (uint32_t)((it / STAGES) & 1);
                if (!(ok = __all_sync(0xffffffffu, wait(&empty[s], ph ^ 1, 21)))) break;
                if (elect_one()) {
                    char *stage = smem + s * STAGE_BYTES;
                    if constexpr (PAIR) {
                        const int half = bn / 2;
                        if (leader) mbar_expect_tx(&full[s], (uint32_t)(2 * PLANES * (TC_A_BYTES + half * TC_BK * 2)));  // both CTAs report to this barrier
#pragma unroll
                        for (int c = 0; c < PLANES; c++) {
                            tma_load_2d_pair(stage + c * TC_A_BYTES, &maps.a, kb * TC_BK, c * prm.a_rows + feat0, full_leader + s * 8);
                            tma_load_2d_pair(stage + OFF_B + c * B_BYTES, bmap, kb * TC_BK, c * prm.b_rows + tok0 + (int)rank * half, full_leader + s * 8);
                        }
                    } else {
                        mbar_expect_tx(&full[s], STAGE_BYTES);
                        tma_load_2d(stage, &maps.a, kb * TC_BK, feat0, &full[s]);
                        tma_load_2d(stage + TC_A_BYTES, &maps.b, kb * TC_BK, tok0, &full[s]);
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (of the leader for pairs)
        if (leader) {
            dependents_wait();  // the limits of the waits below count from here, not while kernels ahead run
            const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint64_t desc0 = make_sw128_desc(smem_u32(smem));
            bool ok = true;
            int it = 0, unit = 0;
            for (int ti = 0; ti < my_tiles && ok; ti++) {
                uint32_t idesc = make_idesc<E>(!PAIR ? TC_BN : narrow(ti) ? prm.tiles.bn_tail : prm.tiles.bn);
                if constexpr (PAIR) idesc = (idesc & ~(0x1fu << 24)) | ((uint32_t)(256 >> 4) << 24);  // M = 256 across the pair
                int kb = 0;
                for (int c = 0; c < nchunks && ok; c++, unit++) {
                    const int b = unit % NBUF, use = unit / NBUF;
                    if (use > 0) ok = __all_sync(0xffffffffu, wait(&acc_free[b], (uint32_t)((use - 1) & 1), 26));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_u + (uint32_t)(b * TC_ACC_COLS);
                    const int kend = (kb + chunk_it < nkb) ? kb + chunk_it : nkb;
                    for (bool first = true; kb < kend; kb++, it++, first = false) {
                        const int s = it % STAGES;
                        const uint32_t ph = (uint32_t)((it / STAGES) & 1);
                        if (!(ok = __all_sync(0xffffffffu, wait(&full[s], ph, 22)))) break;
                        tc_fence_after();
                        if (elect_one()) {
                            const uint64_t stage_a = desc0 + (uint64_t)(uint32_t)(s * (STAGE_BYTES / 16)), stage_b = stage_a + OFF_B / 16;
#pragma unroll
                            for (int t = 0; t < TERMS; t++) {
                                // bias_cols: the operands' roles are exchanged, the order of the products is not (equal results either way)
                                const int ap = !SPLIT ? 0 : prm.bias_cols ? split_x(t) : split_w(t), bp = !SPLIT ? 0 : prm.bias_cols ? split_w(t) : split_x(t);
                                const uint64_t adesc = stage_a + (uint32_t)(ap * (TC_A_BYTES / 16)), bdesc = stage_b + (uint32_t)(bp * (B_BYTES / 16));
#pragma unroll
                                for (int k = 0; k < TC_BK / 16; k++) {  // 16 elements = 32 bytes = 2 descriptor units per step
                                    if constexpr (PAIR) tc2_mma_f16(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (first && t == 0 && k == 0) ? 0u : 1u);
                                    else tc_mma_f16(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (first && k == 0) ? 0u : 1u);
                                }
                            }
                            if constexpr (PAIR) tc2_commit_both(&empty[s]);
                            else tc_commit(&empty[s]);  // arrives when the MMAs above have read the stage
                        }
                        __syncwarp();
                    }
                    // arrives when the unit's MMAs have written TMEM (also on the error path)
                    if (elect_one()) {
                        if constexpr (PAIR) tc2_commit_both(&acc_full[b]);
                        else tc_commit(&acc_full[b]);
                    }
                    __syncwarp();
                }
            }
        }
    }
    } else {
        if constexpr (SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        // ------------------------------------------------------------------ drain warps: promotion and epilogue
        // Feature-major output (out[feature][token]) leaves through a per-warp staging tile: the warp's 32 features x
        // 128 bytes of tokens, 16-byte chunks XOR-swizzled by row.  TMEM hands every lane one feature row; the staging
        // tile turns that into stores whose 8 neighbouring lanes cover 128 contiguous bytes of one output row, which
        // is what both HBM and NVLink want, and the same registers are stored to every destination buffer.
        constexpr int CHUNK_TOK = 16 / (int)sizeof(T);         // tokens per 16-byte chunk
        constexpr int GROUP_TOK = 128 / (int)sizeof(T);        // tokens per staged row: 64 (16-bit) or 32 (fp32)
        constexpr int GROUP_SLICES = GROUP_TOK / 32;           // 32-column TMEM slices per staged group
        constexpr bool RES_AHEAD = TMA_OUT && sizeof(T) == 2;  // residual fetched one slice ahead (fp32 rows would take 2 x 32 registers)
        constexpr int RQ = RES_AHEAD ? 4 : 1;                  // 16-byte pieces of one slice row of the residual
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        constexpr int SLICES = (TC_BN / 32) / (GEMM_DRAIN_WARPS / 4);  // 32-column slices per warp, at most
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
        char *stage_w = staging + (warp - 4) * 4096;
        const T *res = static_cast<const T *>(prm.residual);
        const bool gelu = prm.act == NMG_EPI_GELU;
        // The bias and the residual are read with ordinary loads, possibly before the first accumulator is ready: like the
        // producer's loads they must not run ahead of the grid this one was launched behind.
        dependents_wait();
        int unit = 0;
        bool ok = true;
        uint32_t run[SPLIT ? SLICES : 1][32];  // fp32: sum of the tile's finished chunks
        for (int ti = 0; ti < my_tiles && ok; ti++) {
            int feat0, tok0, bn;
            tile_origin(ti, feat0, tok0, bn);
            // this warp's first slice and how many it has: whole staged groups, the first half of the warps takes the odd one
            const int per_warp = (bn / GROUP_TOK + 1) / 2 * GROUP_SLICES, sl0 = ((warp - 4) >> 2) * per_warp;
            const int nsl = min(per_warp, bn / 32 - sl0);
            const int64_t feat = (int64_t)feat0 + q * 32 + lane;
            const bool feat_ok = feat < prm.out_feats;
            const float bias = (prm.bias && !prm.bias_cols && feat_ok) ? DT<T>::to_f32(static_cast<const T *>(prm.bias)[feat]) : 0.f;
            // column bias: lane l keeps the value of column l of each of this warp's slices; the slice's loop fetches
            // element j's value from lane j
            float bcol[SLICES];
#pragma unroll
            for (int i = 0; i < SLICES; i++) {
                const int64_t col = (int64_t)tok0 + (sl0 + i) * 32 + lane;
                bcol[i] = (prm.bias && prm.bias_cols && col < prm.ntok) ? DT<T>::to_f32(static_cast<const T *>(prm.bias)[col]) : 0.f;
            }
            // The residual of a slice (this lane's row, 32 elements) is fetched in 16-byte pieces one slice ahead of its
            // use, like the accumulator, when the bulk-store path runs and the residual's rows allow it.
            auto res_vec_ok = [&](int64_t tokc) -> bool { return TMA_OUT && prm.res_vec && tokc + 32 <= prm.ntok; };
            auto res_fetch = [&](int sl, uint4 (&qr)[RQ]) {
                if constexpr (RES_AHEAD) {
                    const int64_t tokc = (int64_t)tok0 + sl * 32;
                    if (res && feat_ok && res_vec_ok(tokc)) {
#pragma unroll
                        for (int v = 0; v < RQ; v++) qr[v] = reinterpret_cast<const uint4 *>(res + feat * prm.ld_res + tokc)[v];
                    }
                }
            };
            for (int c = 0; c < nchunks; c++, unit++) {
                const int b = unit % NBUF, use = unit / NBUF;
                if (!(ok = wait(&acc_full[b], (uint32_t)(use & 1), 25))) break;
                tc_fence_after();
                const bool last = c == nchunks - 1;
                auto release = [&]() {  // this warp's TMEM reads of the unit are done: the issuer may reuse the accumulator once all warps say so
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (PAIR) mbar_arrive_remote(acc_free_leader + b * 8);
                        else mbar_arrive(&acc_free[b]);
                    }
                };
                // handle(sl, r, qr): slice sl of the unit is in registers r (this lane's feature row, 32 tokens); qr holds the
                // same 32 elements of the residual when res_fetch found them loadable in 16-byte pieces
                auto handle = [&](int sl, uint32_t (&r)[32], const uint4 (&qr)[RQ]) {
                    if (!(SPLIT && TMA_OUT) && sl == sl0 + nsl - 1) release();
                    const int64_t tokc = (int64_t)tok0 + sl * 32;
                    if constexpr (SPLIT) {  // tiny rows of the activation: this lane's row, or columns of the slice
                        const bool rows = prm.bias_cols != 0;
                        const int64_t at = rows ? feat : tokc + lane;
                        const float f = at < (rows ? prm.out_feats : prm.ntok) && prm.factors[at] == TINY_FACTOR ? TINY_FACTOR : 1.f;
                        if (__any_sync(0xffffffffu, f != 1.f)) {
#pragma unroll
                            for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * (rows ? f : __shfl_sync(0xffffffffu, f, j)));
                        }
                    }
                    // activation(product + bias), kept as fp32 bits in r.  The activation sits in one warp-uniform branch
                    // around its own unrolled loop: the 32 evaluations are independent and interleave, where a test per
                    // element would run them one after the other at full dependent latency.
                    if (prm.bias_cols) {
                        float bc = bcol[0];
#pragma unroll
                        for (int i = 1; i < SLICES; i++) bc = (sl - sl0 == i) ? bcol[i] : bc;
#pragma unroll
                        for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __shfl_sync(0xffffffffu, bc, j));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + bias);
                    }
                    if (gelu) {
#pragma unroll
                        for (int j = 0; j < 32; j += 2) gelu_erf_pair(r[j], r[j + 1]);
                    }
                    if constexpr (TMA_OUT) {
                        if (res && feat_ok) {
                            if (res_vec_ok(tokc)) {
                                if constexpr (RES_AHEAD) {
                                    const T *e = reinterpret_cast<const T *>(qr);
#pragma unroll
                                    for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + DT<T>::to_f32(e[j]));
                                } else {
                                    const uint4 *src = reinterpret_cast<const uint4 *>(res + feat * prm.ld_res + tokc);
#pragma unroll
                                    for (int v = 0; v < 8; v++) {
                                        const uint4 w = src[v];
                                        r[4 * v] = __float_as_uint(__uint_as_float(r[4 * v]) + __uint_as_float(w.x));
                                        r[4 * v + 1] = __float_as_uint(__uint_as_float(r[4 * v + 1]) + __uint_as_float(w.y));
                                        r[4 * v + 2] = __float_as_uint(__uint_as_float(r[4 * v + 2]) + __uint_as_float(w.z));
                                        r[4 * v + 3] = __float_as_uint(__uint_as_float(r[4 * v + 3]) + __uint_as_float(w.w));
                                    }
                                }
                            } else {
                                for (int j = 0; j < 32; j++)
                                    if (tokc + j < prm.ntok) r[j] = __float_as_uint(__uint_as_float(r[j]) + DT<T>::to_f32(res[feat * prm.ld_res + tokc + j]));
                            }
                        }
                        if constexpr (sizeof(T) == 4) {
                            // Two halves of 32 rows x 64 bytes (64-byte swizzle), used in turn: a store reads one while the other is filled.
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                char *half = stage_w + h * 2048 + lane * 64;
                                if (lane == 0) tma_store_wait_read<1>();
                                __syncwarp();
#pragma unroll
                                for (int v = 0; v < 4; v++)
                                    *reinterpret_cast<uint4 *>(half + ((v ^ ((lane >> 1) & 3)) << 4)) =
                                        make_uint4(r[16 * h + 4 * v], r[16 * h + 4 * v + 1], r[16 * h + 4 * v + 2], r[16 * h + 4 * v + 3]);
                                fence_proxy_async_smem();
                                __syncwarp();
                                if (lane == 0) tma_store_2d(&maps.out, stage_w + h * 2048, (int)tokc + 16 * h, feat0 + q * 32);
                            }
                            return;
                        }
                        // registers -> staging row `lane` (16-byte chunks XOR-swizzled by row: the 128-byte swizzle of the
                        // output's tensor map), once the previous group's bulk store has read the tile
                        constexpr int CH = 32 / CHUNK_TOK;  // chunks per slice: 4 (16-bit) or 8 (fp32)
                        const int ch0 = (sl % GROUP_SLICES) * CH;
                        if ((sl % GROUP_SLICES) == 0) {
                            if (lane == 0) tma_store_wait_read();
                            __syncwarp();
                        }
#pragma unroll
                        for (int v = 0; v < CH; v++) {
                            uint4 w;
                            if constexpr (sizeof(T) == 4) {
                                w = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
                            } else {  // one packed conversion per pair
                                w = make_uint4(pack2<T>(__uint_as_float(r[8 * v]), __uint_as_float(r[8 * v + 1])),
                                               pack2<T>(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3])),
                                               pack2<T>(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5])),
                                               pack2<T>(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7])));
                            }
                            *reinterpret_cast<uint4 *>(stage_w + lane * 128 + (((ch0 + v) ^ (lane & 7)) << 4)) = w;
                        }
                        if ((sl % GROUP_SLICES) != GROUP_SLICES - 1) return;
                        // The staging tile is exactly one swizzled box of 32 rows x 128 bytes: hand it to the copy engine,
                        // which clips it at the tensor's edges, and go on with the next slice.
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) tma_store_2d(&maps.out, stage_w, tok0 + (sl / GROUP_SLICES) * GROUP_TOK, feat0 + q * 32);
                        return;
                    } else {
                    if (prm.out_tm_vec) {
                        // Token-major output through the staging tile.  TMEM hands every lane one feature and 32 tokens;
                        // out[token][feature] wants neighbouring lanes on neighbouring features, which scalar stores
                        // give only 2 bytes at a time.  The slice is transposed in shared memory ([token][32 features])
                        // and leaves -- after the residual, fetched in the same 16-byte pieces before the transposition
                        // so that its latency is covered, is added -- in 16-byte stores.
                        constexpr int CPR = 32 * (int)sizeof(T) / 16;  // 16-byte chunks per staged row: 4 (16-bit) or 8 (fp32)
                        const int64_t fbase = (int64_t)feat0 + q * 32 + (lane % CPR) * CHUNK_TOK;  // CHUNK_TOK = elements per chunk
                        const bool whole = fbase + CHUNK_TOK <= prm.out_feats;
                        uint4 rv[CPR];
                        if (res) {
#pragma unroll
                            for (int i = 0; i < CPR; i++) {
                                const int64_t tok = tokc + i * (32 / CPR) + lane / CPR;
                                rv[i] = make_uint4(0u, 0u, 0u, 0u);
                                if (tok < prm.ntok && whole) rv[i] = *reinterpret_cast<const uint4 *>(res + tok * prm.ld_res + fbase);
                            }
                        }
                        T *st = reinterpret_cast<T *>(stage_w);
#pragma unroll
                        for (int j = 0; j < 32; j++) st[j * 32 + lane] = DT<T>::from_f32(__uint_as_float(r[j]));
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < CPR; i++) {
                            const int row = i * (32 / CPR) + lane / CPR;
                            const int64_t tok = tokc + row;
                            if (tok >= prm.ntok || fbase >= prm.out_feats) continue;
                            uint4 w = *reinterpret_cast<const uint4 *>(stage_w + row * 32 * (int)sizeof(T) + (lane % CPR) * 16);
                            if (res) {
                                __align__(16) T a[CHUNK_TOK], b[CHUNK_TOK];
                                *reinterpret_cast<uint4 *>(a) = w;
                                *reinterpret_cast<uint4 *>(b) = rv[i];
                                if (!whole)  // ragged end of the feature axis
                                    for (int k = 0; k < CHUNK_TOK; k++) b[k] = fbase + k < prm.out_feats ? res[tok * prm.ld_res + fbase + k] : DT<T>::from_f32(0.f);
#pragma unroll
                                for (int k = 0; k < CHUNK_TOK; k++) a[k] = DT<T>::from_f32(DT<T>::to_f32(a[k]) + DT<T>::to_f32(b[k]));
                                w = *reinterpret_cast<const uint4 *>(a);
                            }
                            T *dst = static_cast<T *>(prm.outs[0]) + tok * prm.ld_out + fbase;
                            if (whole) *reinterpret_cast<uint4 *>(dst) = w;
                            else {
                                const T *e = reinterpret_cast<const T *>(&w);
                                for (int k = 0; k < CHUNK_TOK && fbase + k < prm.out_feats; k++) dst[k] = e[k];
                            }
                        }
                        __syncwarp();  // the staging rows are free for the next slice
                        return;
                    }
                    // the other output forms take the residual element by element, again under one uniform branch
                    const bool res_late = prm.out_staged && prm.res_vec;
                    if (res && feat_ok && !res_late) {
                        if (prm.out_token_major) {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (tokc + j < prm.ntok) r[j] = __float_as_uint(__uint_as_float(r[j]) + DT<T>::to_f32(res[(tokc + j) * prm.ld_res + feat]));
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j++)
                                if (tokc + j < prm.ntok) r[j] = __float_as_uint(__uint_as_float(r[j]) + DT<T>::to_f32(res[feat * prm.ld_res + tokc + j]));
                        }
                    }
                    if (!prm.out_staged) {
                        if (tokc >= prm.ntok || !feat_ok) return;
                        if (prm.out_token_major && prm.n_out == 1 && tokc + 32 <= prm.ntok) {
                            // full slice of the F.linear layout: one conversion, one pointer step and one store per element
                            T *p = static_cast<T *>(prm.outs[0]) + tokc * prm.ld_out + feat;
#pragma unroll
                            for (int j = 0; j < 32; j++, p += prm.ld_out) *p = DT<T>::from_f32(__uint_as_float(r[j]));
                            return;
                        }
                        for (int d = 0; d < prm.n_out; d++) {
                            T *out = static_cast<T *>(prm.outs[d]);
#pragma unroll
                            for (int j = 0; j < 32; j++) {
                                const int64_t tok = tokc + j;
                                if (tok < prm.ntok) {
                                    const T o = DT<T>::from_f32(__uint_as_float(r[j]));
                                    if (prm.out_token_major) out[tok * prm.ld_out + feat] = o;
                                    else out[feat * prm.ld_out + tok] = o;
                                }
                            }
                        }
                        return;
                    }
                    // registers -> staging row `lane`
                    constexpr int CH = 32 / CHUNK_TOK;  // chunks per slice: 4 (16-bit) or 8 (fp32)
                    const int ch0 = (sl % GROUP_SLICES) * CH;
#pragma unroll
                    for (int v = 0; v < CH; v++) {
                        uint4 w;
                        if constexpr (sizeof(T) == 4) {
                            w = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
                        } else {  // one packed conversion per pair
                            w = make_uint4(pack2<T>(__uint_as_float(r[8 * v]), __uint_as_float(r[8 * v + 1])),
                                           pack2<T>(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3])),
                                           pack2<T>(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5])),
                                           pack2<T>(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7])));
                        }
                        *reinterpret_cast<uint4 *>(stage_w + lane * 128 + (((ch0 + v) ^ (lane & 7)) << 4)) = w;
                    }
                    if ((sl % GROUP_SLICES) != GROUP_SLICES - 1) return;
                    __syncwarp();
                    // staging -> every destination: lane handles chunk (lane & 7) of rows (lane >> 3) + 4 i
                    const int64_t tokg = (int64_t)tok0 + (sl / GROUP_SLICES) * GROUP_TOK + (lane & 7) * CHUNK_TOK;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int row = i * 4 + (lane >> 3);
                        const int64_t f = (int64_t)feat0 + q * 32 + row;
                        if (f >= prm.out_feats || tokg >= prm.ntok) continue;
                        uint4 w = *reinterpret_cast<const uint4 *>(stage_w + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
                        if (res && res_late) {  // the loads of the eight rows are independent of one another and of the staging tile
                            __align__(16) T a[CHUNK_TOK], b[CHUNK_TOK];
                            *reinterpret_cast<uint4 *>(a) = w;
                            if (tokg + CHUNK_TOK <= prm.ntok) *reinterpret_cast<uint4 *>(b) = *reinterpret_cast<const uint4 *>(res + f * prm.ld_res + tokg);
                            else
                                for (int k = 0; k < CHUNK_TOK; k++) b[k] = tokg + k < prm.ntok ? res[f * prm.ld_res + tokg + k] : DT<T>::from_f32(0.f);
#pragma unroll
                            for (int k = 0; k < CHUNK_TOK; k++) a[k] = DT<T>::from_f32(DT<T>::to_f32(a[k]) + DT<T>::to_f32(b[k]));
                            w = *reinterpret_cast<const uint4 *>(a);
                        }
                        if (tokg + CHUNK_TOK <= prm.ntok) {
                            if (prm.mc_out) {  // the switch replicates the 16 bytes to every GPU of the multicast group
                                multimem_st_v4(static_cast<T *>(prm.mc_out) + f * prm.ld_out + tokg, w);
                                continue;
                            }
                            for (int d = 0; d < prm.n_out; d++)
                                *reinterpret_cast<uint4 *>(static_cast<T *>(prm.outs[d]) + f * prm.ld_out + tokg) = w;
                        } else {  // ragged end of the token axis
                            const T *e = reinterpret_cast<const T *>(&w);
                            for (int d = 0; d < prm.n_out; d++)
                                for (int k = 0; k < CHUNK_TOK && tokg + k < prm.ntok; k++)
                                    (static_cast<T *>(prm.outs[d]) + f * prm.ld_out + tokg)[k] = e[k];
                        }
                    }
                    __syncwarp();  // the staging rows are free for the next group
                    }  // !TMA_OUT
                };
                // TMEM reads are software-pipelined: the load of the next slice is in flight while this one is converted
                // and stored; tmem_ld_fence ties the wait to the registers so no use can move above it.
                uint32_t ra[32], rb[32];
                uint4 qa[RQ], qb[RQ];
                const uint32_t acc_addr = lane_base + (uint32_t)(b * TC_ACC_COLS);
                if constexpr (SPLIT) {
                    if (TMA_OUT || nchunks > 1) {
                        // Promotion: the chunk joins the running sum.  With the last one the accumulator is handed back and the epilogue
                        // works on the registers (TMA_OUT), or the total returns to TMEM for it.
#pragma unroll
                        for (int i = 0; i < SLICES; i++) {
                            if (i >= nsl) break;
                            tmem_ld32(acc_addr + (uint32_t)((sl0 + i) * 32), ra);
#pragma unroll
                            for (int j = 0; j < 32; j++) run[i][j] = c > 0 ? __float_as_uint(__fadd_rn(__uint_as_float(run[i][j]), __uint_as_float(ra[j]))) : ra[j];
                            if (!TMA_OUT && last) tmem_st32(acc_addr + (uint32_t)((sl0 + i) * 32), run[i]);
                        }
                        if (TMA_OUT || !last) release();
                        if (!last) continue;
                        if constexpr (TMA_OUT) {
#pragma unroll
                            for (int i = 0; i < SLICES; i++)
                                if (i < nsl) handle(sl0 + i, run[i], qa);
                            continue;
                        }
                    }
                }
                const int sl_end = sl0 + nsl;
                tmem_ld32_issue(acc_addr + (uint32_t)(sl0 * 32), ra);
                res_fetch(sl0, qa);
#pragma unroll 1
                for (int sl = sl0; sl < sl_end; sl += 2) {
                    tmem_ld_fence(ra);
                    if (sl + 1 < sl_end) {
                        tmem_ld32_issue(acc_addr + (uint32_t)((sl + 1) * 32), rb);
                        res_fetch(sl + 1, qb);
                    }
                    handle(sl, ra, qa);
                    if (sl + 1 >= sl_end) break;
                    tmem_ld_fence(rb);
                    if (sl + 2 < sl_end) {
                        tmem_ld32_issue(acc_addr + (uint32_t)((sl + 2) * 32), ra);
                        res_fetch(sl + 2, qa);
                    }
                    handle(sl + 1, rb, qb);
                }
            }
        }
        // the bulk stores must have read their shared-memory source before the CTA's shared memory is given up; their
        // global writes are complete when the grid is
        if (TMA_OUT && lane == 0) tma_store_wait_read();
    }
    __syncthreads();
    if constexpr (PAIR) cluster_sync_all();  // the peer no longer reads this CTA's shared memory or signals its barriers
    if (warp == 1) {
        tc_fence_after();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
        else tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------------ host side
static int64_t dense_ld(int64_t red) { return round_up(red, 8); }  // row stride is a multiple of 16 bytes for TMA

bool tc_dense_supported(const Geo &geo, int dtype) {
    const size_t es = dtype == NMG_F32 ? 4 : 2;
    if (geo.cc > 32767 || geo.C > 65535) return false;
    return expand_smem_bytes(geo, es, false, 1) <= 200 * 1024 && expand_smem_bytes(geo, es, true, 1) <= 200 * 1024;
}

static size_t planes_bytes(int64_t rows, int64_t red) { return ((size_t)SPLIT_PLANES * (size_t)rows * (size_t)dense_ld(red) * 2 + 255) & ~(size_t)255; }

size_t tc_dense_workspace_bytes(const Geo &geo, int dtype, bool transposed) {
    const int64_t rows = transposed ? geo.K : geo.M, red = transposed ? geo.M : geo.K;
    return (dtype == NMG_F32 ? SPLIT_PLANES : 1) * (size_t)rows * (size_t)dense_ld(red) * 2 + 512;
}
size_t tc_split_act_bytes(int64_t tokens, int64_t red) { return planes_bytes(tokens, red) + (size_t)tokens * 4 + 512; }

int tc_split_act(const void *act, int64_t ld_act, bool act_k_major, int64_t tokens, int64_t red, char *buf, DenseAct *out, cudaStream_t st) {
    if (tokens > 65535 * 16) NMG_FAIL(NMG_ERR_UNSUPPORTED, "too many tokens for the split pre-pass");
    SplitParams p{};
    p.src = static_cast<const float *>(act);
    p.dst = reinterpret_cast<__nv_bfloat16 *>(buf);
    p.factors = reinterpret_cast<float *>(buf + planes_bytes(tokens, red));
    p.rows = tokens; p.cols = red; p.ld_src = ld_act; p.ld = dense_ld(red);
    *out = DenseAct{buf, p.ld, p.factors};
    if (act_k_major)
        return launch_early(split_columns_kernel, dim3((unsigned)((p.ld + COLS_RED - 1) / COLS_RED), (unsigned)((tokens + 31) / 32)), COLS_THREADS, 0, st, p);
    if (p.ld <= 1024) return launch_early(split_rows_kernel<4>, (unsigned)((tokens + 3) / 4), SPLIT_THREADS, 0, st, p);
    return launch_early(split_rows_kernel<1>, (unsigned)tokens, SPLIT_THREADS, 0, st, p);
}

template <typename T, bool TR, int N_, bool PLAIN> static int expand_launch_n(const ExpandParams &p, size_t smem, int64_t items, cudaStream_t st) {
    int sms = 148, rc_sms;
    if ((rc_sms = device_sms(&sms))) return rc_sms;
    const int64_t cap = (int64_t)sms * 16;
    NMG_ALLOW_SMEM(smem, expand_dense_kernel<T, TR, N_, PLAIN>);
    return launch_early(expand_dense_kernel<T, TR, N_, PLAIN>, (unsigned)(items < cap ? items : cap), EXPAND_THREADS, smem, st, p);
}
template <typename T, int N_, bool PLAIN, bool STRIPS = false> static int expand_rows_launch_n(const ExpandParams &p, size_t smem, cudaStream_t st) {
    int sms = 148, rc;
    if ((rc = device_sms(&sms))) return rc;
    if (PLAIN && !STRIPS && !p.vec) return expand_rows_launch_n<T, N_, PLAIN, PLAIN>(p, smem, st);
    NMG_ALLOW_SMEM(smem, expand_rows_kernel<T, N_, PLAIN, STRIPS>);
    int per_sm = (int)((size_t)227 * 1024 / (smem + 1024));
    if (per_sm > 8) per_sm = 8;
    const int64_t items = ((p.nb + p.R - 1) / p.R) * ((p.nc + p.Q - 1) / p.Q), cap = (int64_t)sms * per_sm;
    return launch_early(expand_rows_kernel<T, N_, PLAIN, STRIPS>, (unsigned)(items < cap ? items : cap), EXPAND_THREADS, smem, st, p);
}
template <typename T, bool PLAIN> static int expand_rows_launch(const ExpandParams &p, size_t smem, cudaStream_t st) {
    return p.n == 1 ? expand_rows_launch_n<T, 1, PLAIN>(p, smem, st) : expand_rows_launch_n<T, 2, PLAIN>(p, smem, st);
}
template <typename T, bool TR, bool PLAIN = false> static int expand_launch(const ExpandParams &p, size_t smem, int64_t items, cudaStream_t st) {
    // the vectorised scatter reads 16-byte pieces of val / idx: tile bases are 16-byte aligned when cc is a multiple of 8
    const bool aligned = (reinterpret_cast<uintptr_t>(p.val) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.idx) & 15) == 0;
    if (aligned && p.n == 1) return expand_launch_n<T, TR, 1, PLAIN>(p, smem, items, st);
    if (aligned && p.n == 2) return expand_launch_n<T, TR, 2, PLAIN>(p, smem, items, st);
    return expand_launch_n<T, TR, 0, PLAIN>(p, smem, items, st);
}

template <typename T, bool PAIR, bool TMA_OUT> static int gemm_launch_as(const GemmParams &p, const GemmMaps &maps, cudaStream_t st) {
    const size_t smem = (size_t)GEMM_RING_BYTES + GEMM_STAGING_BYTES + 256 + 1024;
    int sms = 148, rc_sms;
    if ((rc_sms = device_sms(&sms))) return rc_sms;
    const int64_t tiles = p.tiles.count();
    NMG_ALLOW_SMEM(smem, gemm_tc_kernel<T, PAIR, TMA_OUT>);
    cudaLaunchConfig_t cfg = {};
    const int64_t units = PAIR ? sms / 2 : sms;  // persistent CTAs, or CTA pairs
    cfg.gridDim = dim3((unsigned)((tiles < units ? tiles : units) * (PAIR ? 2 : 1)));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // overlap the prologue with the expansion pass's tail
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR ? 2 : 1;
    NMG_CUDA(cudaLaunchKernelEx(&cfg, gemm_tc_kernel<T, PAIR, TMA_OUT>, p, maps));
    return NMG_OK;
}
template <typename T, bool PAIR> static int gemm_launch(const GemmParams &p, const GemmMaps &maps, cudaStream_t st) {
    return p.out_tma ? gemm_launch_as<T, PAIR, true>(p, maps, st) : gemm_launch_as<T, PAIR, false>(p, maps, st);
}

// (val, idx) -> the weight with its zeros restored, rows `ld` elements apart at `dst` (16-byte aligned, ld a multiple of 8).
// plain = false: the matmul's operand, 16-bit or three bf16 planes for fp32; plain = true: the
// weight in its own dtype (the densifier), where full stores must not run past the row: K a multiple of 8, or the rows kernel.
static int expand_to(const Geo &geo, int dtype, bool transposed, bool plain, const void *val, const int16_t *idx, void *dst, int64_t ld,
                     cudaStream_t st) {
    const int64_t rows = transposed ? geo.K : geo.M;
    const size_t es = dtype == NMG_F32 ? 4 : 2;
    int rc;
    PatternTable tab;
    if ((rc = get_pattern_table(geo.n, geo.m, &tab))) return rc;
    ExpandParams ep{};
    ep.val = val; ep.idx = idx; ep.order = tab.order; ep.dst = dst;
    ep.ld = ld; ep.plane_elems = rows * ld;
    ep.vec = geo.K % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
    ep.M = geo.M; ep.K = geo.K; ep.nb = geo.nb; ep.nc = geo.nc;
    ep.n = geo.n; ep.m = geo.m; ep.g = geo.g; ep.C = geo.C; ep.cc = geo.cc;
    size_t rsmem = 0;
    const bool aligned = ((reinterpret_cast<uintptr_t>(val) | reinterpret_cast<uintptr_t>(idx)) & 15) == 0;
    if (!transposed && aligned && expand_rows_plan(geo, es, &ep.R, &ep.Q, &rsmem)) {
        if (dtype == NMG_F16) return plain ? expand_rows_launch<__half, true>(ep, rsmem, st) : expand_rows_launch<__half, false>(ep, rsmem, st);
        if (dtype == NMG_BF16) return plain ? expand_rows_launch<__nv_bfloat16, true>(ep, rsmem, st) : expand_rows_launch<__nv_bfloat16, false>(ep, rsmem, st);
        return plain ? expand_rows_launch<float, true>(ep, rsmem, st) : expand_rows_launch<float, false>(ep, rsmem, st);
    }
    ep.R = expand_rows_per_item(geo, es, transposed);
    ep.pitch = expand_pitch(geo, transposed, ep.R);
    const size_t esmem = expand_smem_bytes(geo, es, transposed, ep.R);
    if (esmem > 200 * 1024) NMG_FAIL(NMG_ERR_UNSUPPORTED, "chunk of %d columns does not fit the expansion pass", geo.cc);
    const int64_t items = ((geo.nb + ep.R - 1) / ep.R) * geo.nc;
    if (dtype == NMG_F16) return transposed ? expand_launch<__half, true>(ep, esmem, items, st) : expand_launch<__half, false>(ep, esmem, items, st);
    if (dtype == NMG_BF16) return transposed ? expand_launch<__nv_bfloat16, true>(ep, esmem, items, st) : expand_launch<__nv_bfloat16, false>(ep, esmem, items, st);
    if (plain) return expand_launch<float, false, true>(ep, esmem, items, st);
    return transposed ? expand_launch<float, true>(ep, esmem, items, st) : expand_launch<float, false>(ep, esmem, items, st);
}

int tc_dense_expand(const Geo &geo, int dtype, bool transposed, const void *val, const int16_t *idx, char *dense, cudaStream_t st) {
    return expand_to(geo, dtype, transposed, false, val, idx, dense, dense_ld(transposed ? geo.M : geo.K), st);
}

// The densifier through the expansion pass: whole tiles are scattered into shared memory and leave as 16-byte stores, or, from
// the rows kernel and whatever the destination's alignment, element by element.
bool tc_expand_plain_supported(const Geo &geo, int dtype, const void *val, const int16_t *idx, const void *dense, int64_t ld) {
    const size_t es = dtype == NMG_F32 ? 4 : 2;
    int R, Q;
    size_t smem;
    if (geo.C <= 65535 && ((reinterpret_cast<uintptr_t>(val) | reinterpret_cast<uintptr_t>(idx)) & 15) == 0 && expand_rows_plan(geo, es, &R, &Q, &smem)) return true;
    if (geo.cc > 32767 || geo.C > 65535 || geo.K % 8 != 0 || ld % 8 != 0 || (reinterpret_cast<uintptr_t>(dense) & 15) != 0) return false;
    return expand_smem_bytes(geo, es, false, expand_rows_per_item(geo, es, false)) <= 200 * 1024;
}
int tc_expand_plain(const Geo &geo, int dtype, const void *val, const int16_t *idx, void *dense, int64_t ld, cudaStream_t st) {
    return expand_to(geo, dtype, false, true, val, idx, dense, ld, st);
}

// out = dense[rows][round_up(red, 8)] (16-bit, or the three bf16 planes of an fp32 weight) x activations (16-bit, or the planes of the split).
// CTA pairs (256 rows per tile) unless a 16-bit output has one tile of 128 features only.  source: expand this weight into `dense`
// first, right before the matmul, whose prologue overlaps the expansion's end only when nothing is queued between the two.
int tc_dense_gemm(int64_t rows, int64_t red, int dtype, const char *dense, const DenseAct &act, int64_t tokens, const void *bias,
                  void *const *outs, int n_outs, void *mc_out, int64_t ld_out, int out_token_major, cudaStream_t st, const Epilogue &epi, const DenseSource *source) {
    if (n_outs < 1 || n_outs > GEMM_MAX_OUTS) NMG_FAIL(NMG_ERR_INVALID, "between 1 and %d output buffers, got %d", GEMM_MAX_OUTS, n_outs);
    const int64_t ld = dense_ld(red);
    const int planes = dtype == NMG_F32 ? SPLIT_PLANES : 1;
    int rc;
    GemmMaps maps;
    const int edt = dtype == NMG_F32 ? NMG_BF16 : dtype;
    const size_t osz = dtype == NMG_F32 ? 4 : 2;
    const bool pair = dtype == NMG_F32 || rows > TC_BM;
    // Token-major output of a CTA-pair product: exchange the operands' roles.  The activations become the row operand (tokens
    // on the accumulator's lanes) and the weight the column operand; the output is then "feature-major" in the kernel's terms -- accumulator rows are output rows -- and leaves through the
    // staged 16-byte path with no transposition, the bias running along the columns.
    const bool swap = pair && out_token_major && n_outs == 1 && !mc_out && tokens > TC_BM && (ld_out * osz) % 16 == 0 &&
                      (reinterpret_cast<uintptr_t>(outs[0]) & 15) == 0;
    int sms = 148;
    if ((rc = device_sms(&sms))) return rc;
    const int64_t units = pair ? sms / 2 : sms, row_ext = swap ? tokens : rows, col_ext = swap ? rows : tokens;
    const int tile_feats = pair ? 2 * TC_BM : TC_BM;
    const int64_t tiles_f = (row_ext + tile_feats - 1) / tile_feats;
    if (tiles_f * ((col_ext + 63) / 64) > 0x3fffffff) NMG_FAIL(NMG_ERR_UNSUPPORTED, "too many output tiles for one launch");
    const GemmTiles tiles = gemm_tiles(tiles_f, col_ext, units, dtype == NMG_F32, pair);
    const uint64_t act_rows = (uint64_t)tokens * planes, w_rows = (uint64_t)rows * planes;
    const uint32_t col_box = (uint32_t)(pair ? tiles.bn / 2 : tiles.bn);
    if ((rc = encode_tmap_2d(swap ? &maps.b : &maps.a, edt, dense, (uint64_t)red, w_rows, (uint64_t)ld, TC_BK, swap ? col_box : TC_BM, 1))) return rc;
    if ((rc = encode_tmap_2d(swap ? &maps.a : &maps.b, edt, act.base, (uint64_t)red, act_rows, (uint64_t)act.ld, TC_BK, swap ? TC_BM : col_box, 1))) return rc;
    if (tiles.f_narrow == 0) maps.b_tail = maps.b;
    else if ((rc = encode_tmap_2d(&maps.b_tail, edt, swap ? dense : act.base, (uint64_t)red, swap ? w_rows : act_rows, (uint64_t)(swap ? ld : act.ld), TC_BK, (uint32_t)(tiles.bn_tail / 2), 1))) return rc;
    if (swap) {  // from here on "rows" are the accumulator's rows (tokens) and "tokens" its columns (output features)
        const int64_t t = rows;
        rows = tokens;
        tokens = t;
        out_token_major = 0;
    }
    int *status = nullptr;
    if ((rc = get_status_word(&status))) return rc;
    GemmParams gp{};
    gp.bias = bias;
    gp.n_out = n_outs;
    gp.bias_cols = swap ? 1 : 0;
    gp.factors = act.factors;
    // fp32: the drain warps keep up with short chunks, which leave fewer truncating additions in a row (tc_common).  3072 <- 768, 4096 tokens,
    // chunks of 4 / 2 / 1 k-blocks: 81.8 / 84.1 / 88.8 us and a relative error of 1.33e-6 / 5.4e-7 / 0.9e-7; up to 512 elements: within 1 %.
    gp.chunk_kb = red <= 8 * TC_BK ? 1 : 2;
    gp.a_rows = (int)row_ext; gp.b_rows = (int)col_ext;
    bool vec = !out_token_major && (ld_out * osz) % 16 == 0;
    for (int d = 0; d < n_outs; d++) {
        if (!outs[d]) NMG_FAIL(NMG_ERR_INVALID, "output buffer %d is NULL", d);
        gp.outs[d] = outs[d];
        vec = vec && (reinterpret_cast<uintptr_t>(outs[d]) & 15) == 0;
    }
    gp.out_feats = rows; gp.red = red; gp.ntok = tokens; gp.ld_out = ld_out;
    gp.out_token_major = out_token_major;
    gp.out_staged = vec ? 1 : 0;
    gp.out_tm_vec = (out_token_major && n_outs == 1 && (ld_out * osz) % 16 == 0 && (reinterpret_cast<uintptr_t>(outs[0]) & 15) == 0 &&
                     (!epi.residual || ((epi.ld_res * osz) % 16 == 0 && (reinterpret_cast<uintptr_t>(epi.residual) & 15) == 0)))
                        ? 1 : 0;
    gp.out_tma = (vec && n_outs == 1 && !mc_out) ? 1 : 0;
    if (gp.out_tma) {
        const uint32_t box_cols = dtype == NMG_F32 ? 16 : 64;
        if ((rc = encode_tmap_2d(&maps.out, dtype, outs[0], (uint64_t)tokens, (uint64_t)rows, (uint64_t)ld_out, box_cols, 32, dtype == NMG_F32 ? 2 : 1))) return rc;
    } else {
        maps.out = maps.a;  // never used; keeps the parameter defined
    }
    gp.mc_out = (vec && mc_out && (reinterpret_cast<uintptr_t>(mc_out) & 15) == 0) ? mc_out : nullptr;
    gp.tiles = tiles;
    gp.band = pair ? TC_BAND_PAIR : TC_BAND;
    // many waves over a long reduction: keep the producers in step (see the kernel); the counter is zeroed in stream order.
    // Operands that stay in L2 beside the output need no step keeping: 4096 x 4096, 4096 tokens 108.6 -> 107.4 us without.
    if ((int64_t)tiles.count() >= 3 * units && red >= 4096 && (row_ext + col_ext) * red * 2 * planes > (96ll << 20)) {
        if ((rc = get_wave_counter(&gp.wave_ctr))) return rc;
        NMG_CUDA(cudaMemsetAsync(gp.wave_ctr, 0, sizeof(unsigned), st));
    }
    gp.status = status;
    gp.act = epi.act; gp.residual = epi.residual; gp.ld_res = epi.ld_res;
    gp.res_vec = (epi.residual && (epi.ld_res * osz) % 16 == 0 && (reinterpret_cast<uintptr_t>(epi.residual) & 15) == 0) ? 1 : 0;
    if (source && (rc = tc_dense_expand(source->geo, dtype, source->transposed, source->val, source->idx, const_cast<char *>(dense), st))) return rc;
    if (dtype == NMG_F32) return gemm_launch<float, true>(gp, maps, st);
    if (dtype == NMG_F16) return pair ? gemm_launch<__half, true>(gp, maps, st) : gemm_launch<__half, false>(gp, maps, st);
    return pair ? gemm_launch<__nv_bfloat16, true>(gp, maps, st) : gemm_launch<__nv_bfloat16, false>(gp, maps, st);
}

// Two passes: expansion into `ws`, then the matmul on the expanded weight.  fp32: the activation's planes come first in `ws`.
int tc_dense_matmul(const Geo &geo, int dtype, bool transposed, const void *val, const int16_t *idx, const void *act, int64_t ld_act, bool act_k_major,
                    int64_t tokens, const void *bias, void *const *outs, int n_outs, void *mc_out, int64_t ld_out, int out_token_major,
                    void *ws, size_t ws_bytes, cudaStream_t st, const Epilogue &epi) {
    const int64_t rows = transposed ? geo.K : geo.M, red = transposed ? geo.M : geo.K;
    const size_t act_need = dtype == NMG_F32 ? tc_split_act_bytes(tokens, red) : 0, need = act_need + tc_dense_workspace_bytes(geo, dtype, transposed);
    if (!ws || ws_bytes < need) NMG_FAIL(NMG_ERR_WORKSPACE, "workspace of %zu bytes required for the expanded weight, got %zu", need, ws_bytes);
    char *act_buf = reinterpret_cast<char *>(((uintptr_t)ws + 255) & ~(uintptr_t)255);
    char *dense = reinterpret_cast<char *>(((uintptr_t)ws + act_need + 255) & ~(uintptr_t)255);
    DenseAct planes{act, ld_act, nullptr};
    int rc;
    if (dtype == NMG_F32 && (rc = tc_split_act(act, ld_act, act_k_major, tokens, red, act_buf, &planes, st))) return rc;
    const DenseSource source{geo, transposed, val, idx};
    return tc_dense_gemm(rows, red, dtype, dense, planes, tokens, bias, outs, n_outs, mc_out, ld_out, out_token_major, st, epi, &source);
}

}  // namespace nmg
