// SIMT transposed matmul  dX = dY * W  (the backward of y = x W^T with respect to x) for a grouped n:m weight.
//
// The reduction runs over the rows of W, which is the axis the n:m blocks live on, so the operand a thread
// must select dynamically is a row of dY (one of the m rows of a row-block), while the output column is
// fixed.  The kernel therefore works on a column-ordered copy of the weight (built once per call in the
// workspace by build_natural_kernel): for every row-block mb and column k it stores the column's pattern and
// its n kept values.  A warp owns KW consecutive columns; its lanes are tokens.  For every row-block the
// warp pulls the m x TT slice of dY^T from shared memory into registers once and re-uses it for all KW
// columns; the pattern of each column selects, through a warp-uniform switch over the compile-time pattern
// table, which n of those registers are multiplied.  Accumulators stay in registers over all row-blocks.
#include <type_traits>

#include "nmg_spmm_simt.cuh"
#include "nmg_tc_common.cuh"

namespace nmg {

// ------------------------------------------------------------------------------------------ column-ordered copy
struct NaturalParams {
    const void *val; const int16_t *idx; void *pat; void *nval;
    __nv_bfloat16 *planes;  // fp32 weights the tensor-core kernel serves: three bf16 planes, else NULL
    int64_t nb, nc, Kp;
    int n, m, g, cc;
    int wide;    // 16-bit pattern ids
    int planar;  // n = 2: neighbouring columns' first values, then their second values
};
// One thread per stored column slot.  SMALL: fewer than 2^31 slots, 32-bit index arithmetic.
template <typename T, bool SMALL>
__global__ void build_natural_kernel(const NaturalParams prm) {
    using I = typename std::conditional<SMALL, uint32_t, uint64_t>::type;
    const I total = (I)(prm.nb * prm.nc * prm.cc), nb = (I)prm.nb;
    const T *val = static_cast<const T *>(prm.val);
    T *nval = static_cast<T *>(prm.nval);
    for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
        const I tile = e / (uint32_t)prm.cc, kc = tile / nb;
        const int slot = (int)(e - tile * (uint32_t)prm.cc);
        const int64_t mb = (int64_t)(tile - kc * nb);
        const int c = prm.idx[e];
        if (c < 0 || c >= prm.cc) continue;  // malformed index: leave the column empty
        const int64_t o = mb * prm.Kp + (int64_t)kc * prm.cc + c;
        if (prm.wide) static_cast<uint16_t *>(prm.pat)[o] = (uint16_t)(slot / prm.g);
        else static_cast<uint8_t *>(prm.pat)[o] = (uint8_t)(slot / prm.g * prm.m);
        for (int s = 0; s < prm.n; s++) {
            const int64_t d = prm.planar ? (o & ~(int64_t)1) * 2 + s * 2 + (o & 1) : o * prm.n + s;
            const T v = val[(int64_t)e * prm.n + s];
            nval[d] = v;
            if (sizeof(T) == 4 && prm.planes) {  // exact three-way split
                const int64_t plane = prm.nb * prm.Kp * prm.n;
                __nv_bfloat16 w[3];
                split3(DT<T>::to_f32(v), w);
                for (int t = 0; t < 3; t++) prm.planes[t * plane + d] = w[t];
            }
        }
    }
}

// The same for n <= 2, byte patterns and chunks of whole 16-byte pieces.  HBM-bound work that one scattered store per slot and
// a memset before it did slowly (with the row masks, 4096 x 4096: 74 us bf16 2:4, 128 fp32; now 56 and 75): an item is R row-blocks x Q chunks, about 512
// columns, one piece of eight slots per thread; slots are scattered in shared memory and leave as whole rows, zeros included.
constexpr int NATURAL_THREADS = 256;
struct NaturalRows { int R, Q, groups, spans; };
template <typename T, int N_>
__global__ void __launch_bounds__(NATURAL_THREADS) build_natural_rows_kernel(const NaturalParams prm, const NaturalRows it) {
    extern __shared__ __align__(16) char smem[];
    constexpr int V = 16 / (int)sizeof(T), VL = N_ * 8 / V;  // values per 16 bytes, 16-byte loads of values per piece
    const int R = it.R, Q = it.Q, cc = prm.cc, cols = Q * cc, tid = (int)threadIdx.x;
    T *vals = reinterpret_cast<T *>(smem);                               // [R][cols * N_]
    uint8_t *pats = reinterpret_cast<uint8_t *>(vals + R * cols * N_);  // [R][cols]
    for (int i = tid; i < R * cols * N_ / V; i += NATURAL_THREADS) reinterpret_cast<uint4 *>(vals)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < R * cols / 8; i += NATURAL_THREADS) reinterpret_cast<uint2 *>(pats)[i] = make_uint2(0, 0);
    const int per_chunk = R * cc / 8, q = tid / per_chunk, e8 = (tid - q * per_chunk) * 8, j = e8 / cc, slot0 = e8 - j * cc;
    const bool has = tid < Q * per_chunk;
    const T *val = static_cast<const T *>(prm.val);
    T *nval = static_cast<T *>(prm.nval);
    const int64_t plane = prm.nb * prm.Kp * N_;
    for (int64_t item = blockIdx.x; item < (int64_t)it.groups * it.spans; item += gridDim.x) {
        const int span = (int)(item / it.groups), grp = (int)(item - (int64_t)span * it.groups);
        __syncthreads();  // the buffers are zeros
        const int64_t mb0 = (int64_t)grp * R;
        if (has && span * Q + q < prm.nc && mb0 + j < prm.nb) {
            const int64_t e = ((int64_t)(span * Q + q) * prm.nb + mb0 + j) * cc + slot0;
            const uint4 iv = __ldg(reinterpret_cast<const uint4 *>(prm.idx + e));
            uint4 vv[VL];
#pragma unroll
            for (int i = 0; i < VL; i++) vv[i] = __ldg(reinterpret_cast<const uint4 *>(val + e * N_) + i);
            const int16_t *ci = reinterpret_cast<const int16_t *>(&iv);
            const T *v = reinterpret_cast<const T *>(vv);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int c = ci[k];
                if ((unsigned)c >= (unsigned)cc) continue;  // malformed index: leave the column empty
                const int o = j * cols + q * cc + c;
                pats[o] = (uint8_t)((slot0 + k) / prm.g * prm.m);
                if (N_ == 1) {
                    vals[o] = v[k];
                } else {  // pairs of columns, planar
                    T *d = vals + (o & ~1) * 2 + (o & 1);
                    d[0] = v[k * N_];
                    d[2] = v[k * N_ + (N_ - 1)];
                }
            }
        }
        __syncthreads();
        const int64_t c0 = (int64_t)span * cols;
        const int rows = (int)(prm.nb - mb0 < R ? prm.nb - mb0 : R), lim = (int)(prm.Kp - c0 < cols ? prm.Kp - c0 : cols);
        for (int i = tid; i < R * cols / 8; i += NATURAL_THREADS) {
            const int l = i / (cols / 8), c = (i - l * (cols / 8)) * 8;
            if (l < rows && c < lim) {
                const int64_t o = (mb0 + l) * prm.Kp + c0 + c;
                *reinterpret_cast<uint2 *>(static_cast<uint8_t *>(prm.pat) + o) = *reinterpret_cast<const uint2 *>(pats + i * 8);
#pragma unroll
                for (int u = 0; u < VL; u++) reinterpret_cast<uint4 *>(nval + o * N_)[u] = reinterpret_cast<const uint4 *>(vals + i * 8 * N_)[u];
                if (sizeof(T) == 4 && prm.planes) {  // exact three-way split
#pragma unroll
                    for (int u = 0; u < N_; u++) {
                        __align__(16) uint32_t w[3][4];
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            split3_pair(DT<T>::to_f32(vals[(i * N_ + u) * 8 + 2 * k]), DT<T>::to_f32(vals[(i * N_ + u) * 8 + 2 * k + 1]), w[0][k], w[1][k], w[2][k]);
#pragma unroll
                        for (int t = 0; t < 3; t++) *reinterpret_cast<uint4 *>(prm.planes + t * plane + o * N_ + u * 8) = *reinterpret_cast<const uint4 *>(w[t]);
                    }
                }
            }
            *reinterpret_cast<uint2 *>(pats + i * 8) = make_uint2(0, 0);
#pragma unroll
            for (int u = 0; u < VL; u++) reinterpret_cast<uint4 *>(vals + i * 8 * N_)[u] = make_uint4(0, 0, 0, 0);
        }
    }
}

// Row masks of the forward tensor-core kernel, [k-block of 64 columns][row][8 n bytes]: per slot two words of "the row holds
// the column's value of this slot"; bit 8 j + q of a word is column 4 q + j of its 32.
__global__ void __launch_bounds__(256) build_masks_kernel(const uint8_t *__restrict__ pat, const int8_t *__restrict__ slot_of_row, uint32_t *__restrict__ masks, int64_t M,
                                                          int64_t Kp, int64_t rows, int n, int m, int patterns) {
    __shared__ int8_t table[31 * 16];  // row -> slot of every pattern; at most 28 patterns of up to 16 rows
    for (int i = threadIdx.x; i < patterns * m; i += blockDim.x) table[i] = slot_of_row[i];
    __syncthreads();
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= rows) return;
    for (int64_t kb = blockIdx.y; kb < Kp / 64; kb += gridDim.y) {
        uint32_t mask[2][2] = {{0, 0}, {0, 0}};
        if (row < M) {
            const int64_t mb = row / m;
            const int r = (int)(row - mb * m);
            const uint4 *src = reinterpret_cast<const uint4 *>(pat + mb * Kp + kb * 64);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 v = __ldg(src + i);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    const int col = i * 16 + c, bit = 8 * (col & 3) + ((col & 31) >> 2);
                    // the byte is pattern * m: where the pattern's row table starts
                    const int s = table[((w[c >> 2] >> (8 * (c & 3))) & 0xffu) + r];
                    if (s == 0) mask[0][col >> 5] |= 1u << bit;
                    if (s == 1) mask[1][col >> 5] |= 1u << bit;
                }
            }
        }
        uint32_t *dst = masks + (kb * rows + row) * 2 * n;
        dst[0] = mask[0][0];
        dst[1] = mask[0][1];
        if (n == 2) { dst[2] = mask[1][0]; dst[3] = mask[1][1]; }
    }
}

static bool bwd_specialised(int n, int m) {
    return (n == 1 && m == 4) || (n == 2 && m == 4) || (n == 1 && m == 8) || (n == 2 && m == 8) || (n == 1 && m == 16) ||
           (n == 3 && m == 6);
}

// Width of the column-ordered copy: the padded weight width rounded up to the 128-column CTA tile, so every
// row segment a CTA stages is full-size and 16-byte aligned.
int64_t natural_width(const Geo &geo) { return round_up(geo.nc * geo.cc, 128); }

// Sections of the copy: one pattern entry per column, the values in the weight's dtype and, where the tensor-core kernel
// serves the pattern, the row masks and an fp32 weight's values split into three bf16 planes (split in the kernel, every one
// of a block's m rows would repeat the conversions: 4096 x 4096 2:4, 256 tokens 132 us).  The patterns with specialised
// kernels (at most 28) store one byte, pattern id times m: the offset of the pattern's row selectors in the expansion table of
// the tensor-core kernel; with n = 2 their values are stored pair-wise planar.  All others store 16-bit ids.
NaturalLayout natural_layout(const Geo &geo, int dtype) {
    const size_t entries = (size_t)geo.nb * (size_t)natural_width(geo);
    NaturalLayout l;
    l.pat_bytes = (entries * (bwd_specialised(geo.n, geo.m) ? 1 : 2) + 255) & ~(size_t)255;
    l.val_bytes = (entries * geo.n * dtype_size(dtype) + 255) & ~(size_t)255;
    l.mask_bytes = tc_supported(geo, dtype) ? (size_t)(natural_width(geo) / 64) * (size_t)natural_mask_rows(geo) * 8 * geo.n : 0;
    l.plane_bytes = (dtype == NMG_F32 && tc_supported(geo, dtype)) ? (3 * entries * geo.n * 2 + 255) & ~(size_t)255 : 0;
    l.total = l.pat_bytes + l.val_bytes + l.mask_bytes + l.plane_bytes;
    return l;
}
int64_t natural_mask_rows(const Geo &geo) { return round_up(geo.M, 128); }

size_t natural_bytes(const Geo &geo, int dtype, size_t *pat_bytes_out) {
    const NaturalLayout l = natural_layout(geo, dtype);
    if (pat_bytes_out) *pat_bytes_out = l.pat_bytes;
    return l.total;
}

int launch_build_natural(const Geo &geo, int dtype, const void *val, const int16_t *idx, void *pat, void *nval, cudaStream_t st) {
    const NaturalLayout lay = natural_layout(geo, dtype);
    NaturalParams p{val, idx, pat, nval, nullptr, geo.nb, geo.nc, natural_width(geo), geo.n, geo.m, geo.g, geo.cc, bwd_specialised(geo.n, geo.m) ? 0 : 1,
                    bwd_specialised(geo.n, geo.m) && geo.n == 2 ? 1 : 0};
    const int64_t total = geo.nb * geo.nc * geo.cc;
    int64_t blocks = (total + 255) / 256;
    if (blocks > 148 * 64) blocks = 148 * 64;
    const bool rows_kernel = bwd_specialised(geo.n, geo.m) && geo.n <= 2 && geo.cc % 8 == 0 && geo.cc <= 8 * NATURAL_THREADS &&
                             ((reinterpret_cast<uintptr_t>(val) | reinterpret_cast<uintptr_t>(idx)) & 15) == 0;
    if (lay.plane_bytes) p.planes = reinterpret_cast<__nv_bfloat16 *>(static_cast<char *>(nval) + lay.val_bytes + lay.mask_bytes);
    if (rows_kernel) {
        NaturalRows it;
        it.Q = 512 / geo.cc < 1 ? 1 : 512 / geo.cc;
        it.R = NATURAL_THREADS * 8 / (it.Q * geo.cc);  // one piece per thread
        it.groups = (int)((geo.nb + it.R - 1) / it.R);
        it.spans = (int)((p.Kp + it.Q * geo.cc - 1) / (it.Q * geo.cc));  // up to the padded width: the padding becomes zeros too
        int sms = 148, rc;
        if ((rc = device_sms(&sms))) return rc;
        const int64_t items = (int64_t)it.groups * it.spans, cap = (int64_t)sms * 8;
        const size_t smem = (size_t)it.R * it.Q * geo.cc * (geo.n * dtype_size(dtype) + 1);
        NMG_DISPATCH_DTYPE(dtype, T, {
            if (geo.n == 1) build_natural_rows_kernel<T, 1><<<(unsigned)(items < cap ? items : cap), NATURAL_THREADS, smem, st>>>(p, it);
            else build_natural_rows_kernel<T, 2><<<(unsigned)(items < cap ? items : cap), NATURAL_THREADS, smem, st>>>(p, it);
        });
    } else {
    // every (mb, k) of the chunks is written exactly once because idx is a permutation per tile; clear first so that the
    // columns between the last chunk and the padded width, and what a malformed idx leaves out, are zeros
    NMG_CUDA(cudaMemsetAsync(pat, 0, lay.pat_bytes + lay.val_bytes, st));  // the values follow the patterns
    if (lay.plane_bytes) NMG_CUDA(cudaMemsetAsync(p.planes, 0, lay.plane_bytes, st));
    if (total < 0x40000000ll) {
        NMG_DISPATCH_DTYPE(dtype, T, (build_natural_kernel<T, true><<<(unsigned)blocks, 256, 0, st>>>(p)));
    } else {
        NMG_DISPATCH_DTYPE(dtype, T, (build_natural_kernel<T, false><<<(unsigned)blocks, 256, 0, st>>>(p)));
    }
    }
    if (lay.mask_bytes) {
        PatternTable tab;
        int rc = get_pattern_table(geo.n, geo.m, &tab);
        if (rc) return rc;
        const int64_t rows = natural_mask_rows(geo), kbs = natural_width(geo) / 64;
        build_masks_kernel<<<dim3((unsigned)((rows + 255) / 256), (unsigned)(kbs < 65535 ? kbs : 65535)), 256, 0, st>>>(
            static_cast<const uint8_t *>(pat), tab.slot_of_row, reinterpret_cast<uint32_t *>(static_cast<char *>(nval) + lay.val_bytes), geo.M, natural_width(geo), rows, geo.n, geo.m, geo.C);
    }
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

// ------------------------------------------------------------------------------------------ generic kernel
struct GenBwdParams {
    const uint16_t *pat; const void *nval; const void *dy; void *dx; const int8_t *order;
    int64_t M, K, Kp, ntok, ld_dy, ld_dx, nb;
    int n, m;
};
template <typename T>
__global__ void spmm_bwd_generic_kernel(const GenBwdParams prm) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // lanes along columns: coalesced dX stores
    const int64_t tok = blockIdx.y;
    if (k >= prm.K) return;
    const T *dy = static_cast<const T *>(prm.dy) + tok * prm.ld_dy;
    const T *nval = static_cast<const T *>(prm.nval);
    float acc = 0.f;
    for (int64_t mb = 0; mb < prm.nb; mb++) {
        const int p = prm.pat[mb * prm.Kp + k];
        for (int s = 0; s < prm.n; s++) {
            const int64_t row = mb * prm.m + prm.order[p * prm.n + s];
            if (row < prm.M) acc = fmaf(DT<T>::to_f32(nval[(mb * prm.Kp + k) * prm.n + s]), DT<T>::to_f32(dy[row]), acc);
        }
    }
    static_cast<T *>(prm.dx)[tok * prm.ld_dx + k] = DT<T>::from_f32(acc);
}

// ------------------------------------------------------------------------------------------ host side
static int bwd_rb_stage(int m) {  // rows per stage <= 64 keeps one TMA box (256-row limit) and ~32 KB of dY^T
    int rs = 64 / m;
    return rs > 0 ? rs : 1;
}

size_t simt_bwd_workspace_bytes(const Geo &geo, int64_t tokens, int dtype) {
    (void)dtype;
    return bwd_specialised(geo.n, geo.m) ? (size_t)geo.M * (size_t)round_up(tokens, 128) * 4 + 256 : 0;
}

int simt_bwd(const Geo &geo, int dtype, const void *pat, const void *nval, const void *dy, int64_t ld_dy,
             int64_t tokens, void *dx, int64_t ld_dx, void *ws, size_t ws_bytes, cudaStream_t st) {
    const size_t need = simt_bwd_workspace_bytes(geo, tokens, dtype);
    if (need && (!ws || ws_bytes < need)) NMG_FAIL(NMG_ERR_WORKSPACE, "workspace of %zu bytes required, got %zu", need, ws_bytes);
    char *base = reinterpret_cast<char *>(((uintptr_t)ws + 255) & ~(uintptr_t)255);
    int rc = NMG_OK;
    const int64_t Kp = natural_width(geo);

    if (!bwd_specialised(geo.n, geo.m)) {
        PatternTable tab;
        if ((rc = get_pattern_table(geo.n, geo.m, &tab))) return rc;
        if (tokens > 65535) NMG_FAIL(NMG_ERR_UNSUPPORTED, "generic transposed kernel handles at most 65535 tokens per call");
        GenBwdParams p{static_cast<const uint16_t *>(pat), nval, dy, dx, tab.order, geo.M, geo.K, Kp, tokens, ld_dy, ld_dx, geo.nb, geo.n, geo.m};
        dim3 grid((unsigned)((geo.K + 127) / 128), (unsigned)tokens);
        const ProfileEvents pe = take_profile_events();
        if (pe.start) NMG_CUDA(cudaEventRecord(pe.start, st));
        NMG_DISPATCH_DTYPE(dtype, T, (spmm_bwd_generic_kernel<T><<<grid, 128, 0, st>>>(p)));
        NMG_CUDA(cudaGetLastError());
        if (pe.stop) NMG_CUDA(cudaEventRecord(pe.stop, st));
        return NMG_OK;
    }

    float *yt = reinterpret_cast<float *>(base);
    const int64_t ld_yt = round_up(tokens, 128);
    if ((rc = launch_transpose_to_f32(dy, dtype, tokens, geo.M, ld_dy, yt, ld_yt, st))) return rc;
    const int rs = bwd_rb_stage(geo.m);
    CUtensorMap tm;
    if ((rc = encode_tmap_2d(&tm, NMG_F32, yt, (uint64_t)ld_yt, (uint64_t)geo.M, (uint64_t)ld_yt, (uint32_t)kBwdTok, (uint32_t)(rs * geo.m), 0)))
        return rc;
    int *status = nullptr;
    if ((rc = get_status_word(&status))) return rc;
    BwdParams p{static_cast<const uint8_t *>(pat), nval, dx, geo.M, geo.K, Kp, tokens, ld_dx, geo.nb, rs, status};
    const ProfileEvents pe = take_profile_events();
    if (pe.start) NMG_CUDA(cudaEventRecord(pe.start, st));
#define NMG_BWD_LAUNCH(N_, M_)                                                \
    if (geo.n == N_ && geo.m == M_) {                                         \
        rc = simt_bwd_launch<N_, M_>(dtype, p, tm, tokens, st);               \
        if (rc == NMG_OK && pe.stop) NMG_CUDA(cudaEventRecord(pe.stop, st));  \
        return rc;                                                            \
    }
    NMG_BWD_LAUNCH(1, 4)
    NMG_BWD_LAUNCH(2, 4)
    NMG_BWD_LAUNCH(1, 8)
    NMG_BWD_LAUNCH(2, 8)
    NMG_BWD_LAUNCH(1, 16)
    NMG_BWD_LAUNCH(3, 6)
#undef NMG_BWD_LAUNCH
    NMG_FAIL(NMG_ERR_UNSUPPORTED, "no specialised transposed kernel for %d:%d", geo.n, geo.m);
}

}  // namespace nmg
