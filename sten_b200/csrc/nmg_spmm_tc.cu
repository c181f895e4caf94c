// Fused tensor-core matmul of grouped n:m weights: tcgen05.mma with the expanded weight and the accumulators in TMEM.
//
// In the format's orientation the n:m blocks run along the OUTPUT-feature axis of y = x W^T, so no operand of the
// forward product is structured-sparse along the reduction axis and tcgen05.mma.sp does not apply.  What the
// format does give is a weight that is smaller than its dense form in HBM and L2.  This kernel reads the column-ordered copy
// (bytes per dense element, 16-bit / fp32: values 2 n/m / 4 n/m; a pattern byte per column of a row-block, 1/m; row masks, n/8;
// for fp32 three bf16 planes of the values, 6 n/m.  2:4: 1.5 against 2 dense, fp32 5.5 against 4: the fp32 copy is larger than
// the dense weight, of which the forward product reads masks and planes, 3.25, and the transposed one values and patterns, 2.25).
// Dedicated warps expand it tile by tile into the tensor core's A operand in TMEM, and it is multiplied at dense tensor-core rate
// against activation tiles that arrive by TMA.  The same kernel computes the transposed product dX = dY W: only
// the expansion routine differs (the tile is W^T, the reduction runs over weight rows).
//
// CTA = 15 warps.  Warps 0..11 form three groups that expand the weight tile (128 output features x 64 reduction elements) of
// every third k-block each, from shared memory through registers into TMEM.  Warp 12 loads activation tiles (up to 256 tokens x 64
// reduction elements), warp 14 compressed weight tiles, both by TMA; warp 13 allocates TMEM and issues the MMAs (128 x tokens x 16,
// fp32 accumulate in TMEM).  fp32 weights: a k-block's three bf16 planes are expanded once and multiplied six times (the split
// products).  Warps 0..11 then run the epilogue (tcgen05.ld -> bias -> activation -> residual -> store).
//
// What bounds it with few tokens is latency, not bandwidth: at 4096 x 4096 and 16 tokens the 25 MB of compressed weight are
// 4 us of HBM time.  So the reduction axis is cut over a cluster of CTAs that fills the chip, and the partial tiles meet in
// distributed shared memory -- a second kernel that reads partial tiles from memory cost 4 .. 9 us for 7 .. 14 us of matmul
// (4096 x 1024, 384 tokens: 14.0 + 9.4 us) -- the tile is as wide as the batch needs, and the first tile's loads leave
// before the set-up barrier.  All waits are bounded; a wait that runs out sets the status word and the CTA drains to the
// common exit where TMEM is released.
#include <type_traits>

#include "nmg_spmm_simt.cuh"
#include "nmg_tc_common.cuh"

namespace nmg {


constexpr int FX_A_COLS = TC_BK / 2;  // TMEM columns of one A plane: 64 reduction elements, two per 32-bit column

struct TcParams {
    const void *bias;     // [out_feats] or NULL
    const void *residual; // added after the activation, same orientation as the output, or NULL
    int64_t ld_res;
    int act;              // NMG_EPI_NONE / NMG_EPI_GELU applied to (product + bias)
    void *out;
    const char *masks;    // forward: row masks [k-block][mask_rows][8 n bytes]
    int64_t mask_rows, nb;
    int64_t out_feats;    // M (forward) or K (transposed)
    int64_t red;          // reduction length: K (forward) or M (transposed)
    int64_t ntok, ld_out;
    int out_token_major;  // 1: out[token][feature], 0: out[feature][token]
    int out_vec;          // token-major 16-bit: rows are 4-byte aligned and hold an even count; feature-major: rows are 16-byte aligned
    const float *act_factors;  // fp32: of the activation's rows (DenseAct)
    int act_rows;         // fp32: rows of an activation plane
    int tiles_f, tiles_t; // output tiles along features / tokens
    int bn;               // tokens per tile: a multiple of 32, at most 256 (128 for fp32)
    int stages, slots;    // ring depths, from fx_plan
    int announce;         // tell the next kernel of the stream to start, see tc_matmul
    int groups;           // expansion groups at work: 3, or 2 with two stages
    int ksplit;           // CTAs per tile = cluster size: each takes one range of the reduction axis
    int exch_off;         // exchange area of the partial tiles: offset in shared memory; 0 = on top of the rings
    int misc_off;         // selector table and barriers
    uint32_t tmem_cols;
    int *status;
};
struct FxMaps {
    CUtensorMap x;     // activation (fp32: its planes below one another), box 64 x bn, 128-byte swizzle
    CUtensorMap val;   // forward: 16-bit values [planes * nb][Kpn * n], box 64 x 128/m row-blocks, 128-byte swizzle; transposed: [nb][Kpn * n], box 128 columns x 64/m
    CUtensorMap pat;   // transposed: pattern bytes [nb][Kpn], box 128 columns x 64/m row-blocks
};

// ---- weight-tile expansion ------------------------------------------------------------------------------
// The A operand lives in TMEM (lane = tile row, 32-bit column = two neighbouring reduction elements), so a tile is expanded
// in registers and never passes through shared memory: with the tile in swizzled shared memory its stores, the tensor core's
// reads of it and the table look-ups took 576 of the SM's 128-byte shared-memory cycles per 64 reduction elements of a 2:4
// weight.  One thread owns one tile row.
//
// Forward: the row is a weight row.  Its row masks say for every column whether the row holds the column's first (second)
// kept value; the values are shared by the m rows of the block and arrive as broadcast reads.  An output word (two columns) is
// the OR over the slots of (pair of values AND mask), and PRMT's sign mode spreads two mask bits over the halves of a word:
// two (n = 1) or four (n = 2) instructions per word on the half-rate integer pipe, which is what bounds the expansion, and
// the shift that brings a mask bit to the top of its byte runs on the multiply-add pipe.  Bit 8 j + q of a 32-column mask
// word is column 4 q + j.
// prmt with selector nibbles 8 + i: byte i's sign bit in all eight bits (__byte_perm knows no such selectors)
__device__ __forceinline__ uint32_t spread_signs(uint32_t w, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "r"(sel));
    return r;
}
// mask of columns 4 q + 2 i, 4 q + 2 i + 1 of a 32-column mask word: all ones in the half of every column whose bit is set
__device__ __forceinline__ uint32_t pair_mask(uint32_t word, int q, int i) { return spread_signs(word << (7 - q), i ? 0xbbaau : 0x9988u); }

// Offsets of the eight 16-byte pieces of this row-block's 128 bytes in a box of values (128-byte swizzle: piece ^ row-block)
template <int M_> __device__ __forceinline__ void piece_offsets(int row, uint32_t (&off)[8]) {
    const uint32_t rb = (uint32_t)(row / M_);
#pragma unroll
    for (int i = 0; i < 8; i++) off[i] = rb * 128u + (((uint32_t)i ^ rb) & 7u) * 16u;
}

// vals: PLANES planes of 16-bit values
template <int N_, int M_, int PLANES>
__device__ __forceinline__ void expand_forward(const char *vals, const char *masks, uint32_t a_tmem, int row, const uint32_t (&off)[8]) {
    constexpr int BOX = (TC_BM / M_) * 128, PLANE = BOX * N_;
    uint32_t mask[N_][2];  // 32 columns per word
    if constexpr (N_ == 2) {
        const uint4 k = *reinterpret_cast<const uint4 *>(masks + row * 16);
        mask[0][0] = k.x; mask[0][1] = k.y; mask[N_ - 1][0] = k.z; mask[N_ - 1][1] = k.w;
    } else {
        const uint2 k = *reinterpret_cast<const uint2 *>(masks + row * 8);
        mask[0][0] = k.x; mask[0][1] = k.y;
    }
    auto piece = [&](int pl, int box, int i) { return *reinterpret_cast<const uint4 *>(vals + pl * PLANE + box * BOX + off[i]); };
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t w[PLANES][16];
        if constexpr (N_ == 1) {  // eight columns per piece
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t m0 = pair_mask(mask[0][h], 2 * i, 0), m1 = pair_mask(mask[0][h], 2 * i, 1);
                const uint32_t m2 = pair_mask(mask[0][h], 2 * i + 1, 0), m3 = pair_mask(mask[0][h], 2 * i + 1, 1);
#pragma unroll
                for (int pl = 0; pl < PLANES; pl++) {
                    const uint4 v = piece(pl, 0, h * 4 + i);
                    w[pl][4 * i] = v.x & m0;
                    w[pl][4 * i + 1] = v.y & m1;
                    w[pl][4 * i + 2] = v.z & m2;
                    w[pl][4 * i + 3] = v.w & m3;
                }
            }
        } else {  // four columns: first values, second values of a pair, twice
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const uint32_t a0 = pair_mask(mask[0][h], q, 0), a1 = pair_mask(mask[N_ - 1][h], q, 0);
                const uint32_t b0 = pair_mask(mask[0][h], q, 1), b1 = pair_mask(mask[N_ - 1][h], q, 1);
#pragma unroll
                for (int pl = 0; pl < PLANES; pl++) {
                    const uint4 v = piece(pl, h, q);
                    w[pl][2 * q] = (v.x & a0) | (v.y & a1);
                    w[pl][2 * q + 1] = (v.z & b0) | (v.w & b1);
                }
            }
        }
#pragma unroll
        for (int pl = 0; pl < PLANES; pl++) tmem_st16(a_tmem + (uint32_t)(pl * FX_A_COLS + h * 16), w[pl]);
    }
}

// Transposed: the row is a weight column, the reduction runs over 64 weight rows = 64/m row-blocks.  A column of a row-block
// is n values plus a pattern; its m rows (n of them non-zero) are a byte permutation of the packed values and zero.  The
// permutation selectors of rows (2q, 2q+1) of every pattern are tabulated in shared memory, m/4 words per pattern, and the
// pattern byte of the column-ordered copy is the offset of its entry.
constexpr int FX_TABLE_BYTES = 256;
template <int W> struct Words { uint32_t w[W]; };
template <int W> __device__ __forceinline__ Words<W> lds_words(const char *p) {
    Words<W> r;
    if constexpr (W == 1) r.w[0] = *reinterpret_cast<const uint32_t *>(p);
    else if constexpr (W == 2) { const uint2 v = *reinterpret_cast<const uint2 *>(p); r.w[0] = v.x; r.w[1] = v.y; }
    else { const uint4 v = *reinterpret_cast<const uint4 *>(p); r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w; }
    return r;
}
template <int N_, int M_> __device__ __forceinline__ void build_table(char *table, int tid, int nthreads) {
    constexpr Order<N_, M_> ORD{};
    constexpr int C = Order<N_, M_>::C;
    for (int e = tid; e < C * (M_ / 4); e += nthreads) {  // word e: rows 4q .. 4q+3 of pattern p
        const int p = e / (M_ / 4), q = e - p * (M_ / 4);
        uint32_t word = 0;
        for (int r = 0; r < 4; r++) {
            uint32_t nib = 0x44;  // byte 4 of (values, 0): zero
            for (int sl = 0; sl < N_; sl++)
                if (ORD.v[p * Order<N_, M_>::LD + sl] == 4 * q + r) nib = sl == 0 ? 0x10 : 0x32;
            word |= nib << (8 * r);
        }
        reinterpret_cast<uint32_t *>(table)[e] = word;
    }
}

template <int N_, int M_, typename T, int PLANES>
__device__ __forceinline__ void expand_transposed(const char *vals, const char *pats, const char *table, uint32_t a_tmem, int row) {
    constexpr int W = M_ / 4, J = 32 / M_;  // row-blocks per 32 reduction elements
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t w[PLANES][16];
#pragma unroll
        for (int jj = 0; jj < J; jj++) {
            const int j = h * J + jj;
            const Words<W> sw = lds_words<W>(table + *reinterpret_cast<const uint8_t *>(pats + j * TC_BM + row));
            uint32_t v[PLANES];
            if constexpr (N_ == 1) {
                const char *src = vals + (j * TC_BM + row) * (int)sizeof(T);
                if constexpr (PLANES == 1) v[0] = *reinterpret_cast<const uint16_t *>(src);
                else split3_pair(*reinterpret_cast<const float *>(src), 0.f, v[0], v[1], v[2]);
            } else {  // two columns' first values, then their second values
                const char *src = vals + (j * TC_BM + (row & ~1)) * 2 * (int)sizeof(T);
                if constexpr (PLANES == 1) {
                    const uint2 a = *reinterpret_cast<const uint2 *>(src);
                    v[0] = __byte_perm(a.x, a.y, (row & 1) ? 0x7632 : 0x5410);
                } else {
                    const float *f = reinterpret_cast<const float *>(src) + (row & 1);
                    split3_pair(f[0], f[2], v[0], v[1], v[2]);
                }
            }
#pragma unroll
            for (int pl = 0; pl < PLANES; pl++)
#pragma unroll
                for (int q = 0; q < M_ / 2; q++) w[pl][jj * (M_ / 2) + q] = __byte_perm(v[pl], 0u, (q & 1) ? (sw.w[q >> 1] >> 16) : sw.w[q >> 1]);
        }
#pragma unroll
        for (int pl = 0; pl < PLANES; pl++) tmem_st16(a_tmem + (uint32_t)(pl * FX_A_COLS + h * 16), w[pl]);
    }
}

// ---- the kernel -------------------------------------------------------------------------------------------
// Shared memory of one CTA: a ring of activation stages, a ring of slots for compressed weight tiles, the exchange area of the
// partial tiles (on top of the rings when it does not fit beside them), the selector table and the barriers.
constexpr int FX_GROUPS = 3;                       // expansion groups of four warps: warps 0 .. 11
constexpr int FX_WARP_X = 12, FX_WARP_MMA = 13, FX_WARP_W = 14;  // activation loads, MMA issue (and TMEM), weight loads
constexpr int FX_THREADS = 32 * 15;
constexpr int FX_MAX_STAGES = 8, FX_MAX_SLOTS = 12;
constexpr int FX_SMEM_LIMIT = 224 * 1024;
constexpr int FX_MISC_BYTES = 512 + FX_TABLE_BYTES;
struct FxPlan { int stages, slots, groups, exch_off; uint32_t tmem_cols; size_t total; };
__host__ __device__ constexpr int fx_val_bytes(int n, int m, int es, bool transposed) {  // forward fp32: three 16-bit planes
    return 128 * TC_BK / m * n * (es == 4 && !transposed ? 6 : es);
}
__host__ __device__ constexpr int fx_slot_bytes(int n, int m, int es, bool transposed) {  // values, then masks (forward) or pattern bytes
    return fx_val_bytes(n, m, es, transposed) + (transposed ? 128 * TC_BK / m : 128 * 8 * n);
}
// columns per CTA of a cluster in the exchange, a multiple of four.  The area is [source][4 columns][128 features][4]: a warp's
// push is 512 consecutive bytes (16-byte pieces scattered over feature rows moved 16 bytes per clock), and so is its read.
__host__ __device__ inline int fx_cols_per_owner(int bn, int ks) { return ((bn + ks - 1) / ks + 3) & ~3; }
static FxPlan fx_plan(int planes, int bn, int ks, int slot_bytes) {
    FxPlan p;
    const int x_bytes = planes * bn * TC_BK * 2;
    const int acc = planes > 1 ? 2 * bn : bn;  // fp32: accumulator and running tile
    const int exch = ks > 1 ? ks * 128 * fx_cols_per_owner(bn, ks) * 4 : 0;
    const int budget = FX_SMEM_LIMIT - FX_MISC_BYTES - 1024;
    // A slot always serves the same group (slots are a multiple of the groups) and there are at least as many stages as groups:
    // no barrier is waited on two phases ahead, which a parity wait could not tell apart.
    const int tmem_stages = (512 - acc) / (planes * FX_A_COLS);
    p.groups = tmem_stages < FX_GROUPS ? tmem_stages : FX_GROUPS;
    const int min_rings = p.groups * (x_bytes + slot_bytes);
    const int room = exch + min_rings <= budget ? budget - exch : budget;
    p.slots = 2 * p.groups;
    while (p.slots > p.groups && p.groups * x_bytes + p.slots * slot_bytes > room) p.slots -= p.groups;
    p.stages = (room - p.slots * slot_bytes) / x_bytes;
    if (p.stages > tmem_stages) p.stages = tmem_stages;
    if (p.stages > FX_MAX_STAGES) p.stages = FX_MAX_STAGES;
    while (p.slots + p.groups <= FX_MAX_SLOTS && p.stages * x_bytes + (p.slots + p.groups) * slot_bytes <= room) p.slots += p.groups;
    const int rings = p.stages * x_bytes + p.slots * slot_bytes;
    p.exch_off = (ks > 1 && room < budget) ? (rings + 1023) & ~1023 : 0;
    const int used = p.exch_off ? p.exch_off + exch : (rings > exch ? rings : exch);
    p.total = (size_t)((used + 255) & ~255) + FX_MISC_BYTES + 1024;
    p.tmem_cols = 32;
    while ((int)p.tmem_cols < acc + p.stages * planes * FX_A_COLS) p.tmem_cols *= 2;
    return p;
}

// 16 bytes into a CTA of the cluster, counted by the mbarrier at `bar` in that CTA
__device__ __forceinline__ void dsmem_push_v4(uint32_t cluster_addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];"
                 ::"r"(cluster_addr), "r"(bar), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Epilogue of COLS neighbouring tokens of one feature per lane (a warp: 32 neighbouring features): bias, activation, residual,
// conversion, store.  nt of the tokens exist.  All lanes of the warp call this.
template <typename T, int COLS>
__device__ __forceinline__ void finish_store(const TcParams &prm, uint32_t (&r)[COLS], int64_t feat, bool feat_ok, int64_t tokc, int nt, float b) {
    T *out = static_cast<T *>(prm.out);
    const T *res = static_cast<const T *>(prm.residual);
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < COLS; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + b);
    if (prm.act == NMG_EPI_GELU) {
#pragma unroll
        for (int j = 0; j < COLS; j++) r[j] = __float_as_uint(gelu_erf(__uint_as_float(r[j])));
    }
    if (res && feat_ok) {
        const int64_t step = prm.out_token_major ? prm.ld_res : 1;
        const T *src = prm.out_token_major ? res + tokc * prm.ld_res + feat : res + feat * prm.ld_res + tokc;
#pragma unroll
        for (int j = 0; j < COLS; j++)
            if (j < nt) r[j] = __float_as_uint(__uint_as_float(r[j]) + DT<T>::to_f32(src[j * step]));
    }
    if (!prm.out_token_major) {
        if (!feat_ok) return;
        T *dst = out + feat * prm.ld_out + tokc;
        if (nt >= COLS && prm.out_vec) {  // whole 8- or 16-byte stores
            if constexpr (sizeof(T) == 4) {
#pragma unroll
                for (int v = 0; v < COLS / 4; v++) reinterpret_cast<uint4 *>(dst)[v] = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
            } else {
#pragma unroll
                for (int v = 0; v < COLS / 4; v++)
                    reinterpret_cast<uint2 *>(dst)[v] = make_uint2(pack2<T>(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1])),
                                                                  pack2<T>(__uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3])));
            }
        } else {
#pragma unroll
            for (int j = 0; j < COLS; j++)
                if (j < nt) dst[j] = DT<T>::from_f32(__uint_as_float(r[j]));
        }
        return;
    }
    if (sizeof(T) == 2 && prm.out_vec) {
        // neighbouring lanes exchange one value so that each stores two neighbouring features of one token
        const int odd = lane & 1;
        T *dst = out + (tokc + odd) * prm.ld_out + (feat - odd);
        const bool pair_ok = feat - odd < prm.out_feats;
#pragma unroll
        for (int j = 0; j < COLS; j += 2, dst += 2 * prm.ld_out) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? r[j] : r[j + 1], 1);
            const uint32_t w = odd ? pack2<T>(__uint_as_float(got), __uint_as_float(r[j + 1])) : pack2<T>(__uint_as_float(r[j]), __uint_as_float(got));
            if (j + odd < nt && pair_ok) *reinterpret_cast<uint32_t *>(dst) = w;
        }
        return;
    }
    if (feat_ok) {
        T *dst = out + tokc * prm.ld_out + feat;
#pragma unroll
        for (int j = 0; j < COLS; j++, dst += prm.ld_out)
            if (j < nt) *dst = DT<T>::from_f32(__uint_as_float(r[j]));
    }
}

// One CTA computes 128 features x bn tokens over its range of the reduction axis; the `ksplit` CTAs of a cluster share the
// tile and add their partial tiles through distributed shared memory, in the order of the ranges.
//
// FINE (fp32 forward): the accumulator restarts at every k-block and a k-block's products are added smallest first, so that most
// roundings are those of a small sum.  For a handful of K-major columns, which the gather kernels otherwise serve with fp32 FMAs:
// the error is below theirs at every size, K = 256 / 1024 / 16384, 2:4 0.7 / 0.9 / 1.4e-7 against 2.0 / 4.0 / 16.6e-7, 1:16 0.6 /
// 0.8 / 1.3e-7 against 0.8 / 1.5 / 5.8e-7 (without FINE 11 / 11 / 35e-7 and 7 / 7 / 21e-7).  It costs 8 of 29 us at 4096 x 4096,
// nothing at 1024 x 1024.
template <int N_, int M_, typename T, bool TRANSPOSED, bool FINE>
__global__ void __launch_bounds__(FX_THREADS, 1) spmm_tc_kernel(const TcParams prm, const __grid_constant__ FxMaps maps) {
    constexpr bool SPLIT = sizeof(T) == 4;
    constexpr int PLANES = SPLIT ? SPLIT_PLANES : 1, TERMS = SPLIT ? SPLIT_TERMS : 1;
    using E = typename TcMode<T>::elem;  // element type the tensor cores see
    static_assert(TC_BM % M_ == 0 && 32 % M_ == 0 && M_ % 4 == 0 && N_ <= 2, "tile must hold whole row-blocks; a column's values fit one word");
    static_assert(Order<N_, M_>::C * M_ <= FX_TABLE_BYTES, "a pattern byte is an offset into the selector table");
    constexpr int SLOT_BYTES = fx_slot_bytes(N_, M_, (int)sizeof(T), TRANSPOSED), VAL_BYTES = fx_val_bytes(N_, M_, (int)sizeof(T), TRANSPOSED);
    static_assert(TRANSPOSED || (SLOT_BYTES % 1024 == 0 && VAL_BYTES % 1024 == 0), "swizzled boxes start on 1024-byte boundaries");

    extern __shared__ char smem_raw[];
    char *smem = reinterpret_cast<char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bn = prm.bn, stages = prm.stages, slots = prm.slots;
    const int b_bytes = bn * TC_BK * 2;
    const int x_bytes = PLANES * b_bytes;
    char *slot0 = smem + stages * x_bytes;  // 1024-byte aligned
    char *table = smem + prm.misc_off;
    char *misc = table + FX_TABLE_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(misc);  // activation loads and the expansion group's four warps -> MMA
    uint64_t *empty = full + FX_MAX_STAGES;
    uint64_t *full_w = empty + FX_MAX_STAGES;      // weight loads -> expansion group
    uint64_t *empty_w = full_w + FX_MAX_SLOTS;     // expansion group -> weight loads
    uint64_t *chunk_done = empty_w + FX_MAX_SLOTS; // MMA -> promotion: the accumulator holds a finished chunk (fp32)
    uint64_t *promoted = chunk_done + 1;           // promotion -> MMA: the accumulator may be overwritten
    uint64_t *all_done = promoted + 1;             // MMA -> everyone: the tile is complete
    uint64_t *exchanged = all_done + 1;            // partial tiles of this CTA's columns have arrived
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 496);
    static_assert((2 * FX_MAX_STAGES + 2 * FX_MAX_SLOTS + 4) * 8 <= 496, "barriers overlap the TMEM slot");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ks = prm.ksplit;
    const int split = ks > 1 ? (int)cluster_ctarank() : 0;
    int tile_f, tile_t;
    tile_of_cta((int)blockIdx.x / ks, prm.tiles_f, prm.tiles_t, tile_f, tile_t);
    const int64_t tok0 = (int64_t)tile_t * bn;
    const int64_t feat0 = (int64_t)tile_f * TC_BM;
    // 32-bit loop arithmetic throughout: the single MMA-issuing thread must stay ahead of the tensor core, and a
    // 64-bit division per iteration on that thread is enough to make issue the bottleneck.
    const int nkb_all = (int)((prm.red + TC_BK - 1) / TC_BK);
    const int kb_per = (nkb_all + ks - 1) / ks;
    const int kb_base = split * kb_per;  // this CTA's first k-block
    const int nkb = (nkb_all < kb_base + kb_per ? nkb_all : kb_base + kb_per) - kb_base;  // >= 1 by the host's choice of ksplit
    // k-blocks per accumulation chunk.  fp32: 4, and two chunks at least, so that at most 76 of the additions to an accumulator find a sum of
    // full size there.  A promotion costs 0.5 us at 64 tokens and 1.2 at 256, so up to four k-blocks make one chunk where their stages are
    // there together: the largest product of the first `hold` waits for the small ones of all of them, which leaves four such additions per
    // k-block (three k-blocks in two stages: 32).  Relative error 0.8 .. 1.4e-7 then, else at most 1.3e-6.
    const bool at_once = nkb <= 3 || (nkb == 4 && prm.stages >= 4);
    const int chunk_kb = SPLIT ? (FINE ? 1 : at_once ? nkb : nkb < 8 ? (nkb + 1) / 2 : 4) : nkb;
    const int hold = SPLIT && !FINE && at_once ? min(nkb, prm.stages) : 1;
    const int nchunks = (nkb + chunk_kb - 1) / chunk_kb;
    const uint32_t tmem_cols = prm.tmem_cols;
    const int cols_live = (int)(prm.ntok - tok0 < bn ? prm.ntok - tok0 : bn);  // token columns of this tile that exist
    const int cpo = fx_cols_per_owner(bn, ks);                                    // columns each CTA of the cluster finishes
    const bool exch_apart = ks > 1 && prm.exch_off != 0;

    // ---- loads, by the two producer warps
    auto load_x = [&](int kb, int s) {
        mbar_expect_tx(&full[s], (uint32_t)x_bytes);
#pragma unroll
        for (int pl = 0; pl < PLANES; pl++)
            tma_load_2d(smem + s * x_bytes + pl * b_bytes, &maps.x, (kb_base + kb) * TC_BK, (SPLIT ? pl * prm.act_rows : 0) + (int)tok0, &full[s]);
    };
    auto load_w = [&](int kb, int s) {
        mbar_expect_tx(&full_w[s], (uint32_t)SLOT_BYTES);
        char *w = slot0 + s * SLOT_BYTES;
        if constexpr (TRANSPOSED) {
            const int y = (kb_base + kb) * (TC_BK / M_);
            tma_load_2d(w, &maps.val, (int)feat0 * N_, y, &full_w[s]);
            tma_load_2d(w + VAL_BYTES, &maps.pat, (int)feat0, y, &full_w[s]);
        } else {
#pragma unroll
            for (int bx = 0; bx < PLANES * N_; bx++)  // 64 values per box; the planes lie below one another
                tma_load_2d(w + bx * (TC_BM / M_) * 128, &maps.val, ((kb_base + kb) * N_ + bx % N_) * TC_BK, bx / N_ * (int)prm.nb + (int)(feat0 / M_), &full_w[s]);
            bulk_load(w + VAL_BYTES, prm.masks + ((int64_t)(kb_base + kb) * prm.mask_rows + feat0) * (8 * N_), 128 * 8 * N_, &full_w[s]);
        }
    };
    const int groups = prm.groups;
    const int lead_x = nkb < 2 ? nkb : 2, lead_w = nkb < groups ? nkb : groups;  // loads issued before the set-up barrier

    // ---- set-up.  The producers initialise their own barriers and issue every group's first loads before the CTA-wide barrier,
    // so that their latency runs beside the TMEM allocation.
    if (warp == FX_WARP_W) {
        if (lane == 0) {
            for (int s = 0; s < slots; s++) {
                mbar_init(&full_w[s], 1);
                mbar_init(&empty_w[s], 4);
            }
            mbar_fence_init();
        }
        __syncwarp();
        dependents_wait();  // from here on other kernels' results may be read
        if (elect_one())
            for (int kb = 0; kb < lead_w; kb++) load_w(kb, kb);
        __syncwarp();
    } else if (warp == FX_WARP_X) {
        if (lane == 0) {
            for (int s = 0; s < stages; s++) {
                mbar_init(&full[s], 5);
                mbar_init(&empty[s], 1);
            }
            mbar_init(chunk_done, 1);
            mbar_init(promoted, 4 * FX_GROUPS);
            mbar_init(all_done, 1);
            mbar_init(exchanged, 1);
            mbar_fence_init();
            if (ks > 1) {  // bytes this CTA will receive: 16 per feature, source and four live columns
                int mine = cols_live - split * cpo;
                mine = mine < 0 ? 0 : (mine < cpo ? mine : cpo);
                mbar_expect_tx(exchanged, (uint32_t)(ks * 128 * 16 * ((mine + 3) / 4)));
            }
        }
        __syncwarp();
        dependents_wait();
        if (elect_one())
            for (int kb = 0; kb < lead_x; kb++) load_x(kb, kb);
        __syncwarp();
    } else {
        if (warp == FX_WARP_MMA) tmem_alloc(tmem_slot, tmem_cols);
        if (TRANSPOSED && warp < FX_WARP_X) build_table<N_, M_>(table, tid, FX_WARP_X * 32);
        dependents_wait();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t a_base = tmem_base + (uint32_t)(SPLIT ? 2 * bn : bn);  // A stages follow the accumulator (and the running tile)
    // A partial tile is pushed into the other CTAs' shared memory: they must have started (waited for before the push).
    __syncwarp();
    if (exch_apart) cluster_arrive();

    // fp32 mode: a finished chunk of the accumulator is added to the running tile (columns bn .. 2 bn) with round-to-nearest
    // adds.  The MMAs wait for it, so all twelve warps take part: each its quarter of the lanes of every third slice.
    auto promote_chunk = [&](int c) -> bool {
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(chunk_done, (uint32_t)(c & 1), prm.status, 15))) return false;
        tc_fence_after();
        for (int sl = warp >> 2; sl < bn / 32; sl += FX_GROUPS) {
            uint32_t r[32];
            tmem_ld32(lane_base + (uint32_t)(sl * 32), r);
            if (c > 0) {
                uint32_t run[32];
                tmem_ld32(lane_base + (uint32_t)(bn + sl * 32), run);
#pragma unroll
                for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__fadd_rn(__uint_as_float(run[j]), __uint_as_float(r[j])));
            }
            tmem_st32(lane_base + (uint32_t)(bn + sl * 32), r);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(promoted);
        return true;
    };

    bool ok = true;
    if (warp == FX_WARP_X || warp == FX_WARP_W) {
        // ------------------------------------------------------------------ activation and compressed weight loads
        const bool is_x = warp == FX_WARP_X;
        const int ring = is_x ? stages : slots;
        uint64_t *freed = is_x ? empty : empty_w;
        int s = is_x ? lead_x : lead_w;
        uint32_t ph = 1;
        if (s >= ring) { s -= ring; ph ^= 1; }
        for (int kb = is_x ? lead_x : lead_w; kb < nkb; kb++) {
            ok = mbar_wait_bounded(&freed[s], ph, prm.status, is_x ? 11 : 18);
            if (!__all_sync(0xffffffffu, ok)) break;
            if (elect_one()) {
                if (is_x) load_x(kb, s);
                else load_w(kb, s);
            }
            __syncwarp();
            if (++s == ring) { s = 0; ph ^= 1; }
        }
    } else if (warp == FX_WARP_MMA) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = make_idesc<E>(bn);
        const uint32_t d_tmem = __shfl_sync(0xffffffffu, tmem_base, 0), at_base = __shfl_sync(0xffffffffu, a_base, 0);
        const uint64_t bdesc0 = make_sw128_desc(smem_u32(smem));
        int s = 0, chunk = 0, in_chunk = 0;
        uint32_t ph = 0;
        for (int kb = 0; kb < nkb; kb++) {
            const bool first = in_chunk == 0;
            if (first && chunk > 0) ok = mbar_wait_bounded(promoted, (uint32_t)((chunk - 1) & 1), prm.status, 16);
            ok = ok && mbar_wait_bounded(&full[s], ph, prm.status, 12);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const bool chunk_end = in_chunk + 1 == chunk_kb && kb + 1 < nkb;
            if (elect_one()) {
                auto product = [&](int stage, int t, bool restart) {
                    const uint32_t at = at_base + (uint32_t)((stage * PLANES + (SPLIT ? split_w(t) : 0)) * FX_A_COLS);
                    const uint64_t bt = bdesc0 + (uint64_t)(uint32_t)(stage * (x_bytes >> 4) + (SPLIT ? split_x(t) : 0) * (b_bytes >> 4));
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; k++)  // 16 elements = 8 TMEM columns of A, 32 bytes = 2 descriptor units of B
                        tc_mma_f16_ta(d_tmem, at + 8 * k, bt + 2 * k, idesc, (restart && k == 0) ? 0u : 1u);
                };
#pragma unroll
                for (int t = 0; t < TERMS - 1; t++) product(s, t, first && t == 0);
                if (kb >= hold - 1) {
                    for (int held = 0; SPLIT && kb == hold - 1 && held < kb; held++) {  // k-block = stage
                        product(held, TERMS - 1, false);
                        tc_commit(&empty[held]);
                    }
                    product(s, TERMS - 1, first && TERMS == 1);
                    tc_commit(&empty[s]);  // arrives when the MMAs above have read the stage
                }
                if (chunk_end) tc_commit(chunk_done);
            }
            __syncwarp();
            in_chunk++;
            if (chunk_end) {
                in_chunk = 0;
                chunk++;
            }
            if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (elect_one()) tc_commit(all_done);  // also on the error path: the others fall through their bounded waits sooner
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ expansion groups
        const int group = warp >> 2, gtid = tid & 127;
        int drained = 0;  // fp32: accumulation chunks already promoted
        int s = group, w = group;
        uint32_t ph = 0, phw = 0;
        const uint32_t a_lane = a_base + ((uint32_t)((warp & 3) * 32) << 16);
        uint32_t off[8];
        if constexpr (!TRANSPOSED) piece_offsets<M_>(gtid, off);
        for (int kb = group; group < groups && kb < nkb; kb += groups) {
            if constexpr (SPLIT) {
                // Before feeding a later chunk, promote the finished ones: the MMAs of a chunk depend only on tiles that are
                // already published, so this wait cannot deadlock, and the MMA issuer needs the promotion before it may
                // restart the accumulator.
                while (ok && drained < kb / chunk_kb) {
                    ok = promote_chunk(drained);
                    drained++;
                }
            }
            ok = ok && mbar_wait_bounded(&full_w[w], phw, prm.status, 19) && mbar_wait_bounded(&empty[s], ph ^ 1, prm.status, 14);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();  // the MMAs that read this stage are done
            const char *vals = slot0 + w * SLOT_BYTES;
            const uint32_t a_tmem = a_lane + (uint32_t)(s * PLANES * FX_A_COLS);
            if constexpr (TRANSPOSED) expand_transposed<N_, M_, T, PLANES>(vals, vals + VAL_BYTES, table, a_tmem, gtid);
            else expand_forward<N_, M_, PLANES>(vals, vals + VAL_BYTES, a_tmem, gtid, off);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_w[w]);  // the slot has been read
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
            if ((s += groups) >= stages) { s -= stages; ph ^= 1; }
            if ((w += groups) >= slots) { w -= slots; phw ^= 1; }
        }
        if constexpr (SPLIT)
            while (ok && drained < nchunks - 1) {  // the chunks behind the last tile this group published (all of them for an idle group)
                ok = promote_chunk(drained);
                drained++;
            }
        ok = mbar_wait_bounded(all_done, 0, prm.status, 17) && ok;
    }
    if (prm.announce) dependents_launch();  // the first warps are here when the last loads have been issued
    __syncwarp();
    tc_fence_before();
    if (exch_apart) cluster_wait();          // the other CTAs have started
    else if (ks > 1) cluster_sync_all();     // every CTA's MMAs are done: shared memory of all of them is free for the exchange
    if (SPLIT && nchunks > 1) __syncthreads();  // group 0's promotions, before everybody's reads of the running tile
    tc_fence_after();

    // ---- epilogue: warps 0 .. 11, each a quarter of the TMEM lanes and every third slice of 32 token columns
    const int fl = tid & 127;                     // this thread's feature row of the tile (warps 0 .. 11)
    const int64_t feat = feat0 + fl;
    const bool feat_ok = warp < FX_WARP_X && feat < prm.out_feats;
    const float bias = (prm.bias && feat_ok) ? DT<T>::to_f32(static_cast<const T *>(prm.bias)[feat]) : 0.f;
    if (warp < FX_WARP_X) {
        const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t exch = smem_u32(smem + prm.exch_off) + (uint32_t)(split * cpo * 128 * 4 + fl * 16), bar = smem_u32(exchanged);
        const uint32_t inv_cpo = 65536u / (uint32_t)cpo + 1u;
        for (int sl = warp >> 2; sl * 32 < cols_live; sl += FX_GROUPS) {
            uint32_t r[32];
            __syncwarp();
            tmem_ld32(lane_base + (uint32_t)(sl * 32), r);
            if (SPLIT && nchunks > 1) {
                uint32_t run[32];
                tmem_ld32(lane_base + (uint32_t)(bn + sl * 32), run);
#pragma unroll
                for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__fadd_rn(__uint_as_float(run[j]), __uint_as_float(r[j])));
            }
            if constexpr (SPLIT) {  // tokens with a tiny row
                const float f = sl * 32 + lane < cols_live && prm.act_factors[tok0 + sl * 32 + lane] == TINY_FACTOR ? TINY_FACTOR : 1.f;
                if (__any_sync(0xffffffffu, f != 1.f)) {
#pragma unroll
                    for (int j = 0; j < 32; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * __shfl_sync(0xffffffffu, f, j));
                }
            }
            if (ks > 1) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {  // cpo is a multiple of four: four columns have one owner
                    const uint32_t col = (uint32_t)(sl * 32 + j), owner = (col * inv_cpo) >> 16;
                    if ((int)col < cols_live)
                        dsmem_push_v4(map_to_rank(exch + (col - owner * (uint32_t)cpo) * 512u, owner), map_to_rank(bar, owner), r[j], r[j + 1], r[j + 2], r[j + 3]);
                }
            } else {
                finish_store<T, 32>(prm, r, feat, feat_ok, tok0 + sl * 32, cols_live - sl * 32, bias);
            }
        }
    }
    if (ks > 1 && warp < FX_WARP_X) {
        const int c0 = split * cpo;
        const int ncols = cols_live - c0 < cpo ? cols_live - c0 : cpo;  // may be <= 0
        ok = mbar_wait_cluster_bounded(exchanged, 0, prm.status, 20);
        if (__all_sync(0xffffffffu, ok)) {
            const char *src = smem + prm.exch_off + fl * 16;
            for (int c = (warp >> 2) * 4; c < ncols; c += 4 * FX_GROUPS) {
                float4 acc = *reinterpret_cast<const float4 *>(src + c * 512);
                for (int s = 1; s < ks; s++) {  // in the order of the ranges
                    const float4 v = *reinterpret_cast<const float4 *>(src + (s * cpo + c) * 512);
                    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                }
                uint32_t r[4] = {__float_as_uint(acc.x), __float_as_uint(acc.y), __float_as_uint(acc.z), __float_as_uint(acc.w)};
                finish_store<T, 4>(prm, r, feat, feat_ok, tok0 + c0 + c, ncols - c, bias);
            }
        }
    }
    // A CTA whose wait for the others' partial tiles ran out must not give up shared memory that they may still write to: it stays
    // until every CTA of the cluster has ended (exited threads count as arrived, and all waits of the others are bounded).
    if (__syncthreads_or(ks > 1 && warp < FX_WARP_X && !ok)) cluster_sync_all();
    if (warp == FX_WARP_MMA) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
}

// ------------------------------------------------------------------------------------------------------ host side
bool tc_supported(const Geo &geo, int dtype) {
    if (dtype != NMG_F16 && dtype != NMG_BF16 && dtype != NMG_F32) return false;
    return (geo.n == 1 && geo.m == 4) || (geo.n == 2 && geo.m == 4) || (geo.n == 1 && geo.m == 8) || (geo.n == 2 && geo.m == 8) ||
           (geo.n == 1 && geo.m == 16);
}

// Tile width and cluster size: the pair with the smallest estimate of a CTA's time, from what the parts of the kernel measure
// on a B200 (timestamps inside the kernel, 2:4 weights, ns):
//   per k-block of 64: 300, the expansion and the issue of its MMAs (three planes in fp32: 900); above 192 tokens the MMAs
//     themselves (2 clocks per token)
//   per 32-column slice a warp finishes: 450
//   exchange between ks CTAs: 900 for its barriers, 17 per column for the distributed-shared-memory traffic, 27 per column
//     finished (bn / ks of them)
// The token axis is cut into equal tiles, so that a batch just above a multiple does not pay for a nearly empty one.
// A grid that does not fit the chip at once runs in waves; kFxClusters is what fits (cudaOccupancyMaxActiveClusters: the GPCs
// are not all alike, 24 clusters of 6 do not fit although 144 < 148).
constexpr int kFxClusters[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
struct FxChoice { int bn, tiles_f, tiles_t, ksplit; int64_t ns; };
static FxChoice fx_choose(int64_t feats, int64_t red, int64_t tokens, int dtype) {
    const int max_bn = dtype == NMG_F32 ? 128 : 256;  // fp32: the accumulator, the running tile and two stages of three A planes share TMEM
    const int64_t tiles_f = (feats + TC_BM - 1) / TC_BM, nkb = (red + TC_BK - 1) / TC_BK;
    FxChoice best{};
    int64_t best_ns = -1;
    for (int64_t cap = 32; cap <= max_bn; cap += 32) {
        const int64_t parts = (tokens + cap - 1) / cap;
        const int bn = (int)round_up((tokens + parts - 1) / parts, 32);
        if (bn != cap) continue;
        const int64_t tiles_t = (tokens + bn - 1) / bn, tiles = tiles_f * tiles_t;
        for (int want = 1; want <= 8; want++) {  // 8: the portable cluster size
            if (want > 1 && want > nkb / 2) break;
            const int64_t per = (nkb + want - 1) / want;
            const int ks = (int)((nkb + per - 1) / per);  // every range non-empty
            const int64_t waves = (tiles + kFxClusters[ks] - 1) / kFxClusters[ks];
            int64_t ns = 3000 + per * (dtype == NMG_F32 ? 900 : bn > 192 ? 300 + (bn - 192) : 300);
            if (ks > 1) ns += 900 + bn * 17 + bn * 27 / ks;
            else ns += (bn / 32 + 2) / 3 * 450;
            ns *= waves;
            if (best_ns < 0 || ns < best_ns) {
                best_ns = ns;
                best = FxChoice{bn, (int)tiles_f, (int)tiles_t, ks, ns};
            }
        }
    }
    return best;
}

size_t tc_split_workspace_bytes(const Geo &geo, int dtype, bool transposed, int64_t tokens) {
    return dtype == NMG_F32 ? tc_split_act_bytes(tokens, transposed ? geo.M : geo.K) : 0;
}

template <int N_, int M_, typename T, bool TR, bool FINE = false>
static int tc_launch_one(const TcParams &p0, const FxMaps &maps, cudaStream_t st) {
    const FxPlan plan = fx_plan(sizeof(T) == 4 ? SPLIT_PLANES : 1, p0.bn, p0.ksplit, fx_slot_bytes(N_, M_, (int)sizeof(T), TR));
    TcParams p = p0;
    p.stages = plan.stages;
    p.slots = plan.slots;
    p.groups = plan.groups;
    p.exch_off = plan.exch_off;
    p.tmem_cols = plan.tmem_cols;
    p.misc_off = (int)(plan.total - 1024 - FX_MISC_BYTES);
    const int64_t ctas = (int64_t)p.tiles_f * p.tiles_t * p.ksplit;
    if (ctas > 0x7fffffff) NMG_FAIL(NMG_ERR_UNSUPPORTED, "too many output tiles for one launch");
    NMG_ALLOW_SMEM(plan.total, spmm_tc_kernel<N_, M_, T, TR, FINE>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(FX_THREADS);
    cfg.dynamicSmemBytes = plan.total;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the set-up overlaps the preceding kernel's end
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.ksplit;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.ksplit > 1 ? 2 : 1;
    NMG_CUDA(cudaLaunchKernelEx(&cfg, spmm_tc_kernel<N_, M_, T, TR, FINE>, p, maps));
    return NMG_OK;
}

template <int N_, int M_>
static int tc_launch_nm(int dtype, bool transposed, bool fine, const TcParams &p, const FxMaps &maps, cudaStream_t st) {
    if (dtype == NMG_F16) return transposed ? tc_launch_one<N_, M_, __half, true>(p, maps, st) : tc_launch_one<N_, M_, __half, false>(p, maps, st);
    if (dtype == NMG_F32)
        return transposed ? tc_launch_one<N_, M_, float, true>(p, maps, st) : fine ? tc_launch_one<N_, M_, float, false, true>(p, maps, st) : tc_launch_one<N_, M_, float, false>(p, maps, st);
    return transposed ? tc_launch_one<N_, M_, __nv_bfloat16, true>(p, maps, st) : tc_launch_one<N_, M_, __nv_bfloat16, false>(p, maps, st);
}

// Policy of the two tensor-core variants.  The fused kernel reads the column-ordered copy; without one (have_packed) a call
// would build it first and throw it away.  Measured, us, 2:4: fused with a kept copy / fused after building one / two passes
//   fp32   tokens    1024 x 1024       4096 x 1024       1024 x 4096       4096 x 4096
//              64    10 /  23 / 21     13 /  33 / 27    17 / 35 / 61      26 /  81 /  98
//             256    13 /  26 / 23     22 /  43 / 30    27 / 46 / 62      58 / 114 / 104
//             512    18 /  31 / 25     31 /  51 / 35    36 / 55 / 65     100 / 156 / 119
//             768    20 /   - / 27     54 /   - / 44    55 /  - / 67     171 /   - / 139
//            1024    24 /   - / 28     58 /   - / 53    61 /  - / 71     197 /   - / 166
//   bf16     1024     9 /  24 / 17     12 /  30 /  21    20 / 37 / 31      27 /  65 /  42
//            1280    10 /  24 / 17     19 /  37 /  25    21 / 37 / 32      49 /  86 /  60
//            1500    10 /  24 / 17     20 /  39 /  25    23 / 40 / 33      50 /  88 /  61
//            3072    11 /  26 / 17     32 /  51 /  30    26 / 44 / 33      87 / 130 /  89
// fp32 with a copy: above 512 tokens the fused kernel wins while all its tiles are resident, and loses in its second wave.  Without one,
// up to 512 tokens the shape decides, not the count; the fused kernel takes them, with the same results as with a copy.  The transposed
// product of a 16-bit weight has the structured-sparse kernel in place of the second variant (from 1280 tokens).
bool tc_use_dense(const Geo &geo, int dtype, bool transposed, int64_t tokens, bool have_packed) {
    const bool fused = tc_supported(geo, dtype), dense = tc_dense_supported(geo, dtype);
    if (!dense) return false;
    if (!fused) return true;
    if (!have_packed) return tokens >= (dtype == NMG_F32 ? 513 : 1280);
    if (dtype == NMG_F32) return tokens > 1024 || (tokens > 512 && ((transposed ? geo.K : geo.M) + TC_BM - 1) / TC_BM * ((tokens + 127) / 128) > kFxClusters[1]);
    return tokens >= (transposed ? 1280 : 1536);
}

// act: [tokens][ld_act] with the reduction axis contiguous (X for the forward, dY for the transposed product).
int tc_matmul(const Geo &geo, int dtype, bool transposed, bool dense, const void *val, const int16_t *idx, const void *pat,
              const void *nval, const void *act, int64_t ld_act, bool act_k_major, int64_t tokens, const void *bias, void *const *outs, int n_outs,
              void *mc_out, int64_t ld_out, int out_token_major, void *ws, size_t ws_bytes, cudaStream_t st, const Epilogue &epi, bool alone) {
    if (n_outs < 1 || (n_outs > 1 && !dense)) NMG_FAIL(NMG_ERR_UNSUPPORTED, "several output buffers need the two-pass tensor-core variant");
    void *out = outs[0];
    int rc;
    if (dense) {
        const ProfileEvents pe = take_profile_events();
        if (pe.start) NMG_CUDA(cudaEventRecord(pe.start, st));
        rc = tc_dense_matmul(geo, dtype, transposed, val, idx, act, ld_act, act_k_major, tokens, bias, outs, n_outs, mc_out, ld_out, out_token_major, ws, ws_bytes, st, epi);
        if (rc == NMG_OK && pe.stop) NMG_CUDA(cudaEventRecord(pe.stop, st));
        return rc;
    }
    const int64_t red = transposed ? geo.M : geo.K;
    const int64_t feats = transposed ? geo.K : geo.M;
    const bool fine = dtype == NMG_F32 && act_k_major && tokens < 64;
    const FxChoice fx = fx_choose(feats, red, tokens, dtype);
    DenseAct x{act, ld_act, nullptr};
    if (dtype == NMG_F32) {
        const size_t need = tc_split_act_bytes(tokens, red);
        if (!ws || ws_bytes < need) NMG_FAIL(NMG_ERR_WORKSPACE, "workspace of %zu bytes required for the split activation, got %zu", need, ws_bytes);
        if ((rc = tc_split_act(act, ld_act, act_k_major, tokens, red, reinterpret_cast<char *>(((uintptr_t)ws + 255) & ~(uintptr_t)255), &x, st))) return rc;
    }
    int *status = nullptr;
    if ((rc = get_status_word(&status))) return rc;
    const size_t es = dtype_size(dtype);
    FxMaps maps;
    const int edt = dtype == NMG_F32 ? NMG_BF16 : dtype, planes = dtype == NMG_F32 ? SPLIT_PLANES : 1;
    if ((rc = encode_tmap_2d(&maps.x, edt, x.base, (uint64_t)red, (uint64_t)tokens * planes, (uint64_t)x.ld, TC_BK, (uint32_t)fx.bn, 1))) return rc;
    const int64_t Kpn = natural_width(geo);
    const NaturalLayout lay = natural_layout(geo, dtype);
    const char *masks = static_cast<const char *>(nval) + lay.val_bytes;
    const uint64_t row_elems = (uint64_t)(Kpn * geo.n);
    if (transposed) {
        if ((rc = encode_tmap_2d_bytes(&maps.pat, pat, (uint64_t)Kpn, (uint64_t)geo.nb, (uint64_t)Kpn, TC_BM, (uint32_t)(TC_BK / geo.m)))) return rc;
        if ((rc = encode_tmap_2d(&maps.val, dtype, nval, row_elems, (uint64_t)geo.nb, row_elems, (uint32_t)(TC_BM * geo.n), (uint32_t)(TC_BK / geo.m), 0))) return rc;
    } else {
        const char *vals = dtype != NMG_F32 ? static_cast<const char *>(nval) : masks + lay.mask_bytes;
        if ((rc = encode_tmap_2d(&maps.val, edt, vals, row_elems, (uint64_t)(geo.nb * planes), row_elems, TC_BK, (uint32_t)(TC_BM / geo.m), 1))) return rc;
        maps.pat = maps.val;  // never used; keeps the parameter defined
    }
    TcParams p{};
    p.bias = bias; p.out = out; p.out_feats = feats; p.red = red; p.ntok = tokens; p.ld_out = ld_out;
    p.residual = epi.residual; p.ld_res = epi.ld_res; p.act = epi.act;
    p.out_token_major = out_token_major;
    p.out_vec = out_token_major ? (ld_out % 2 == 0 && feats % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & 3) == 0)
                                : (ld_out * es % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0);
    p.tiles_f = fx.tiles_f; p.tiles_t = fx.tiles_t; p.bn = fx.bn; p.ksplit = fx.ksplit;
    // The set-up of the next kernel beside this one's end saves 0.3 .. 0.9 us where kernels of this sort follow one another (f16 2:4, 384 x 1984,
    // 11 tokens 6.5 -> 5.6; 4096 x 4096, 16 tokens 10.1 -> 9.7).  A pass over the activation that settles on the SMs left free then is the slower
    // for it (mm bf16 2240 x 9216, 64 columns 14.1 -> 15.2), and so are some long ones (5440 x 10944 1:16, 128 tokens 23.8 -> 24.5).
    p.announce = alone && dtype != NMG_F32 && fx.ns < 14000;
    p.act_factors = x.factors; p.act_rows = (int)tokens;
    p.masks = masks; p.mask_rows = natural_mask_rows(geo); p.nb = geo.nb;
    p.status = status;
    const ProfileEvents pe = take_profile_events();
    if (pe.start) NMG_CUDA(cudaEventRecord(pe.start, st));
    rc = NMG_ERR_UNSUPPORTED;
#define NMG_TC_CASE(N_, M_)                                                                         \
    if (geo.n == N_ && geo.m == M_)                                                                \
        rc = tc_launch_nm<N_, M_>(dtype, transposed, fine, p, maps, st);
    NMG_TC_CASE(1, 4)
    NMG_TC_CASE(2, 4)
    NMG_TC_CASE(1, 8)
    NMG_TC_CASE(2, 8)
    NMG_TC_CASE(1, 16)
#undef NMG_TC_CASE
    if (rc == NMG_ERR_UNSUPPORTED) set_error("no tensor-core kernel for %d:%d", geo.n, geo.m);
    if (rc == NMG_OK && pe.stop) NMG_CUDA(cudaEventRecord(pe.stop, st));
    return rc;
}

// ---- activation / residual after kernels that do not fuse them --------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) epilogue_kernel(T *out, int64_t rows, int64_t cols, int64_t ld_out, int act, const T *res, int64_t ld_res) {
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y)
        for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += (int64_t)gridDim.x * blockDim.x) {
            float v = DT<T>::to_f32(out[r * ld_out + c]);
            if (act == NMG_EPI_GELU) v = 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
            if (res) v += DT<T>::to_f32(res[r * ld_res + c]);
            out[r * ld_out + c] = DT<T>::from_f32(v);
        }
}

int launch_epilogue(int dtype, void *out, int64_t rows, int64_t cols, int64_t ld_out, const Epilogue &epi, cudaStream_t st) {
    if (!epi.any() || rows < 1 || cols < 1) return NMG_OK;
    dim3 grid((unsigned)((cols + 255) / 256 < 64 ? (cols + 255) / 256 : 64), (unsigned)(rows < 65535 ? rows : 65535));
    NMG_DISPATCH_DTYPE(dtype, T, {
        epilogue_kernel<T><<<grid, 256, 0, st>>>(static_cast<T *>(out), rows, cols, ld_out, epi.act, static_cast<const T *>(epi.residual), epi.ld_res);
    });
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

}  // namespace nmg
