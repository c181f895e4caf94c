// Format conversion kernels: dense -> nmg magnitude sparsifier (bit-exact with the sequential definition of the
// format) and nmg -> dense.  Both are one pass over the weight; the weight is read / written in place in its
// [batch][M][K] layout, so no padded, permuted or zero-filled temporaries exist.
#include "nmg_common.cuh"

namespace nmg {

// =====================================================================================================
// Sparsifier.
//
// Definition of the result (the reference's CPU implementation): for every tile, score each (column c, pattern p)
// with the fp32 sum of |w| over the rows of p (summed in slot order), sort all (score, c, p) triples
// descending (ties: larger c, then larger p) and walk the list once, accepting a triple when its column is
// still free and its pattern holds fewer than g columns.
//
// That walk is a greedy matching of columns (capacity 1) to patterns (capacity g) by descending weight under a strict
// total order of the pairs.  Such a matching is the unique stable one: the heaviest pair must be matched in any stable
// matching (otherwise it blocks), remove it and repeat.  Deferred acceptance reaches the same matching in a few parallel
// rounds instead of C*g sequential steps: every free column proposes to the best pattern it can still enter, every
// pattern keeps its g best proposers (sorted by (score, c) descending) and releases the rest, released columns propose
// again.  A pattern's final list in descending order is exactly the order in which the sequential walk accepted its
// columns, so val / idx come out bit for bit identical -- without the C^2*g-element sort, without a sequential chain of
// C*g dependent reductions, and without scratch memory in HBM.
//
// One warp per tile.  Lanes own columns (c = lane, lane + 32, ...) when columns propose, and patterns (p = lane,
// lane + 32, ...) when patterns merge their proposers.  The tile is read with 16-byte loads where alignment allows.
// =====================================================================================================

// (row-block, column chunk, batch entry) of a tile; 32-bit division whenever the tile count allows it (a 64-bit division
// costs about as much as scoring a column).
__device__ __forceinline__ void tile_coords(int64_t tile, int64_t nb, int64_t nc, int64_t tiles, int64_t &mb, int64_t &kc, int64_t &b) {
    if (tiles < 0x7fffffffll) {
        const unsigned t = (unsigned)tile, unb = (unsigned)nb, unc = (unsigned)nc;
        const unsigned q = t / unb;
        mb = t - q * unb;
        const unsigned q2 = q / unc;
        kc = q - q2 * unc;
        b = q2;
    } else {
        mb = tile % nb;
        kc = (tile / nb) % nc;
        b = tile / (nb * nc);
    }
}

static int sm_count() {
    int sms = 148;
    return device_sms(&sms) == NMG_OK ? sms : 148;
}

struct SparsifyParams {
    const void *dense;
    void *val;
    int16_t *idx;
    const int8_t *order;  // [C][n] device
    int64_t M, K, ld, batch_stride;
    int64_t nb, nc, tiles;
    int n, m, g, C, cc;
    int slab_bytes;  // shared memory per warp
};

// A proposal / list entry: fp32 score bits (non-negative, so unsigned order = float order) above the column index.
// Comparing entries of one pattern as integers is the format's order (score, then larger column first).
__device__ __forceinline__ uint64_t sp_key(uint32_t score_bits, int c) { return ((uint64_t)score_bits << 16) | (uint32_t)c; }

// Shared memory of one warp (host and device agree through this function).
struct SparsifySlab { size_t list, inbox, x, park, state, prop_p, prop_i, cnt, total; };
__host__ __device__ inline SparsifySlab sparsify_slab(int m, int cc, int C, size_t es) {
    SparsifySlab l;
    size_t o = 0;
    l.list = o;   o += (size_t)cc * 8;                                   // [C][g] kept proposers of every pattern, descending
    l.inbox = o;  o += (size_t)cc * 8;                                   // [cc] this round's proposals, grouped by pattern
    l.x = o;      o += (((size_t)m * cc * es) + 15) & ~(size_t)15;       // [m][cc] the tile
    l.park = o;   o += (size_t)cc * 4;                                   // [cc] score of the column's proposal
    l.state = o;  o += (size_t)cc * 2;                                   // [cc] pattern the column is held by, -1 = free
    l.prop_p = o; o += (size_t)cc * 2;                                   // [cc] pattern proposed to this round
    l.prop_i = o; o += (size_t)cc * 2;                                   // [cc] position inside that pattern's inbox segment
    o = (o + 3) & ~(size_t)3;
    l.cnt = o;    o += (size_t)C * 4 * 3;                                // [C] list lengths, proposals this round, segment starts
    l.total = (o + 15) & ~(size_t)15;
    return l;
}


// Zero phase of the selection.  Triples whose score is 0 come last in the format's order, sorted by larger column, then
// larger pattern; when the walk reaches them every pattern in which a still-free column scores above zero is full.  So
// the free columns, taken from the largest index down, each fill the largest pattern that has room left: a closed form,
// no rounds.  (Zero-padded columns of a last chunk and all-zero columns of a pruned weight end up here; letting them
// run through the rounds would cost one round per pattern with hundreds of tied proposals each.)
// On entry cnt[p] holds the list lengths; rem / cum are scratch of C ints each.  All lanes of the warp call this.
__device__ __forceinline__ void sparsify_zero_phase(int lane, int cc, int C, int g, uint64_t *list, int16_t *state, int *cnt, int *rem, int *cum) {
    // cum[p] = free places in patterns with a larger index (suffix sum), rem[p] = free places of p
    const int pchunk = (C + 31) / 32;
    const int p0 = lane * pchunk, p1 = min(C, p0 + pchunk);
    int local = 0;
    for (int p = p0; p < p1; p++) { rem[p] = g - cnt[p]; local += g - cnt[p]; }
    int incl = local;  // inclusive suffix sum over lanes
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_down_sync(0xffffffffu, incl, d);
        if (lane + d < 32) incl += t;
    }
    int run = incl - local;  // free places in the chunks of higher lanes
    for (int p = p1 - 1; p >= p0; p--) { cum[p] = run; run += g - cnt[p]; }
    __syncwarp();
    int above = 0;  // free columns in higher rows of the column-to-lane layout (larger indices), warp-uniform
    for (int k = (cc - 1) / 32; k >= 0; k--) {
        const int c = k * 32 + lane;
        const bool is_free = c < cc && state[c] < 0;
        const uint32_t mask = __ballot_sync(0xffffffffu, is_free);
        if (is_free) {
            const int i = above + __popc(lane == 31 ? 0u : (mask >> (lane + 1)));  // free columns with a larger index
            int lo = 0, hi = C - 1;  // largest p with cum[p] <= i (cum decreases with p, cum[C - 1] = 0)
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (cum[mid] <= i) hi = mid; else lo = mid + 1;
            }
            // patterns without room share their cum with the next smaller pattern that has some: step down to it
            int p = lo;
            while (p > 0 && i - cum[p] >= rem[p]) p--;
            list[p * g + cnt[p] + (i - cum[p])] = (uint64_t)(uint32_t)c;  // score 0
            state[c] = (int16_t)p;
        }
        above += __popc(mask);
    }
    __syncwarp();
}

template <typename T>
__global__ void __launch_bounds__(256) sparsify_kernel(SparsifyParams prm) {
    extern __shared__ __align__(16) char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int n = prm.n, m = prm.m, g = prm.g, C = prm.C, cc = prm.cc;
    constexpr int V = 16 / (int)sizeof(T);  // elements per 16-byte access

    // CTA-wide copy of the pattern table, then one slab per warp.
    int8_t *ord = reinterpret_cast<int8_t *>(smem);
    const int ord_bytes = (C * n + 15) & ~15;
    for (int i = threadIdx.x; i < C * n; i += blockDim.x) ord[i] = prm.order[i];
    __syncthreads();

    char *slab = smem + ord_bytes + (size_t)warp * prm.slab_bytes;
    const SparsifySlab lay = sparsify_slab(m, cc, C, sizeof(T));
    uint64_t *list = reinterpret_cast<uint64_t *>(slab + lay.list);
    uint64_t *inbox = reinterpret_cast<uint64_t *>(slab + lay.inbox);
    T *x = reinterpret_cast<T *>(slab + lay.x);
    uint32_t *park = reinterpret_cast<uint32_t *>(slab + lay.park);
    int16_t *state = reinterpret_cast<int16_t *>(slab + lay.state);
    int16_t *prop_p = reinterpret_cast<int16_t *>(slab + lay.prop_p);
    int16_t *prop_i = reinterpret_cast<int16_t *>(slab + lay.prop_i);
    int *cnt = reinterpret_cast<int *>(slab + lay.cnt);
    int *icnt = cnt + C;
    int *ioff = icnt + C;

    const T *dense = static_cast<const T *>(prm.dense);
    T *val = static_cast<T *>(prm.val);
    const int pchunk = (C + 31) / 32;  // patterns per lane in the prefix sum

    for (int64_t tile = (int64_t)blockIdx.x * nwarps + warp; tile < prm.tiles; tile += (int64_t)gridDim.x * nwarps) {
        int64_t mb, kc, b;
        tile_coords(tile, prm.nb, prm.nc, prm.tiles, mb, kc, b);
        const int64_t row0 = mb * m, col0 = kc * cc;
        const T *src = dense + b * prm.batch_stride;
        // ---- load the tile (rows beyond M and columns beyond K read as zero)
        const bool full_cols = col0 + cc <= prm.K;
        for (int r = 0; r < m; r++) {
            const bool row_ok = row0 + r < prm.M;
            const T *srow = src + (row0 + r) * prm.ld + col0;
            T *xr = x + r * cc;
            if (row_ok && full_cols && (cc % V) == 0 && (reinterpret_cast<uintptr_t>(srow) & 15) == 0) {
                for (int c = lane * V; c < cc; c += 32 * V)
                    *reinterpret_cast<uint4 *>(xr + c) = __ldg(reinterpret_cast<const uint4 *>(srow + c));
            } else {
                for (int c = lane; c < cc; c += 32) xr[c] = (row_ok && col0 + c < prm.K) ? srow[c] : DT<T>::from_f32(0.f);
            }
        }
        for (int c = lane; c < cc; c += 32) state[c] = -1;
        for (int p = lane; p < C; p += 32) cnt[p] = 0;
        __syncwarp();

        // ---- deferred acceptance.  Every round with a free column makes at least one proposal (column, pattern) that was
        // never made before, so cc * C rounds cannot be exceeded; real weights settle in a handful.
        for (int round = 0; round < cc * C + 2; round++) {
            for (int p = lane; p < C; p += 32) icnt[p] = 0;
            __syncwarp();
            // columns propose: the best pattern (larger p on equal score) among those the column can still enter
            bool proposed = false;
            for (int c = lane; c < cc; c += 32) {
                prop_p[c] = -1;
                if (state[c] >= 0) continue;
                uint32_t best_s = 0;
                int best_p = -1;
                for (int p = 0; p < C; p++) {
                    float s = 0.f;
                    for (int i = 0; i < n; i++) s = __fadd_rn(s, fabsf(DT<T>::to_f32(x[(int)ord[p * n + i] * cc + c])));
                    const uint32_t sb = __float_as_uint(s);
                    if (sb == 0) continue;  // zero scores are placed by the closed form after the rounds
                    if (cnt[p] >= g && sp_key(sb, c) <= list[p * g + g - 1]) continue;  // full, and every kept proposer ranks higher
                    if (best_p < 0 || sb >= best_s) { best_s = sb; best_p = p; }
                }
                if (best_p < 0) continue;  // nothing above zero is open to this column: it waits for the zero phase
                proposed = true;
                prop_p[c] = (int16_t)best_p;
                prop_i[c] = (int16_t)atomicAdd(&icnt[best_p], 1);
                park[c] = best_s;
            }
            if (!__any_sync(0xffffffffu, proposed)) break;
            __syncwarp();
            // exclusive prefix sum of the proposal counts -> start of every pattern's inbox segment
            {
                const int p0 = lane * pchunk, p1 = min(C, p0 + pchunk);
                int local = 0;
                for (int p = p0; p < p1; p++) local += icnt[p];
                int incl = local;
                for (int d = 1; d < 32; d <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += t;
                }
                int run = incl - local;
                for (int p = p0; p < p1; p++) { ioff[p] = run; run += icnt[p]; }
            }
            __syncwarp();
            for (int c = lane; c < cc; c += 32)
                if (prop_p[c] >= 0) inbox[ioff[prop_p[c]] + prop_i[c]] = sp_key(park[c], c);
            __syncwarp();
            // patterns merge their proposers into their sorted lists; what does not fit is released
            for (int p = lane; p < C; p += 32) {
                uint64_t *lp = list + p * g;
                int L = cnt[p];
                const int e0 = ioff[p], e1 = e0 + icnt[p];
                for (int e = e0; e < e1; e++) {
                    const uint64_t key = inbox[e];
                    if (L == g) {
                        if (key <= lp[g - 1]) continue;            // stays free (state is still -1)
                        state[(int)(lp[g - 1] & 0xffffu)] = -1;     // the weakest kept proposer is released
                        L = g - 1;
                    }
                    int j = L;
                    while (j > 0 && lp[j - 1] < key) { lp[j] = lp[j - 1]; j--; }
                    lp[j] = key;
                    L++;
                    state[(int)(key & 0xffffu)] = (int16_t)p;
                }
                cnt[p] = L;
            }
            __syncwarp();
        }
        __syncwarp();
        sparsify_zero_phase(lane, cc, C, g, list, state, cnt, icnt, ioff);

        // ---- write the tile: idx = the lists' columns, val = the kept rows of those columns
        int16_t *idx_out = prm.idx + tile * cc;
        T *val_out = val + tile * (int64_t)cc * n;
        for (int s0 = lane; s0 < cc; s0 += 32) idx_out[s0] = (int16_t)(list[s0] & 0xffffu);
        for (int e = lane; e < cc * n; e += 32) {
            const int s0 = e / n, t = e - s0 * n;
            const int c = (int)(list[s0] & 0xffffu), p = s0 / g;
            val_out[e] = x[(int)ord[p * n + t] * cc + c];
        }
        __syncwarp();
    }
}

// Shared memory of one warp in the (n, m)-specialised kernel: no copy of the tile (its values are re-read through L1),
// lists as separate score / column arrays, proposals as column indices.  8.3 KB for a 448-column tile, so that about
// twenty-seven warps are resident per SM: the selection is a chain of dependent shared-memory accesses, and residency is what hides it.
struct SparsifyLean { size_t lscore, park, lcol, inbox, state, prop_p, freel, cnt, total; };
__host__ __device__ inline SparsifyLean sparsify_lean(int cc, int C) {
    SparsifyLean l;
    size_t o = 0;
    l.lscore = o; o += (size_t)cc * 4;   // [C][g] score bits of the kept proposers, descending by (score, column)
    l.park = o;   o += (size_t)cc * 4;   // [cc] score of the column's current proposal / match
    l.lcol = o;   o += (size_t)cc * 2;   // [C][g] their columns
    l.inbox = o;  o += (size_t)cc * 2;   // [cc] this round's proposing columns, grouped by pattern
    l.state = o;  o += (size_t)cc * 2;   // [cc] pattern the column is held by, -1 = free
    l.prop_p = o; o += (size_t)cc * 2;   // [cc] pattern proposed to this round, -1 = none
    l.freel = o;  o += (size_t)cc * 2;   // columns that propose in the next round (rejected or released in this one)
    o = (o + 3) & ~(size_t)3;
    l.cnt = o;    o += (size_t)C * 4 * 3 + 4;  // cnt, icnt, ioff per pattern + the length of freel
    l.total = (o + 15) & ~(size_t)15;
    return l;
}

// Specialisation on (n, m): the pattern table is a compile-time constant, so a column's |w| values sit in registers and
// all C scores are straight-line adds; which patterns are full is one bit mask (C <= 32), so the first round -- where
// nothing is full -- touches no shared state at all.  The first round's proposals are placed by rank (every proposal
// counts the larger proposals of its own pattern, all lanes busy) instead of by one lane per pattern inserting in turn.
template <int N_, int M_, typename T>
__global__ void __launch_bounds__(256, 4) sparsify_nm_kernel(SparsifyParams prm) {
    extern __shared__ __align__(16) char smem[];
    constexpr Order<N_, M_> ORD{};
    constexpr int C = Order<N_, M_>::C;
    static_assert(C <= 32, "the full-pattern mask is one word");
    constexpr int V = 16 / (int)sizeof(T);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int g = prm.g, cc = prm.cc;

    int8_t *ord = reinterpret_cast<int8_t *>(smem);  // run-time copy of the table for the output stage
    constexpr int ord_bytes = (C * N_ + 15) & ~15;
    for (int i = threadIdx.x; i < C * N_; i += blockDim.x) ord[i] = (int8_t)ORD.v[(i / N_) * Order<N_, M_>::LD + (i % N_)];
    __syncthreads();

    char *slab = smem + ord_bytes + (size_t)warp * prm.slab_bytes;
    const SparsifyLean lay = sparsify_lean(cc, C);
    uint32_t *lscore = reinterpret_cast<uint32_t *>(slab + lay.lscore);
    uint32_t *park = reinterpret_cast<uint32_t *>(slab + lay.park);
    int16_t *lcol = reinterpret_cast<int16_t *>(slab + lay.lcol);
    int16_t *inbox = reinterpret_cast<int16_t *>(slab + lay.inbox);
    int16_t *state = reinterpret_cast<int16_t *>(slab + lay.state);
    int16_t *prop_p = reinterpret_cast<int16_t *>(slab + lay.prop_p);
    int16_t *freel = reinterpret_cast<int16_t *>(slab + lay.freel);
    int *cnt = reinterpret_cast<int *>(slab + lay.cnt);
    int *icnt = cnt + C;
    int *ioff = icnt + C;
    int *nfree = ioff + C;

    const T *dense = static_cast<const T *>(prm.dense);
    T *val = static_cast<T *>(prm.val);
    const bool g_pow2 = (g & (g - 1)) == 0;
    const int g_shift = 31 - __clz(g);
    // (score, column) order of the format: larger score first, on equal scores the larger column
    auto above = [](uint32_t s1, int c1, uint32_t s2, int c2) { return s1 > s2 || (s1 == s2 && c1 > c2); };

    for (int64_t tile = (int64_t)blockIdx.x * nwarps + warp; tile < prm.tiles; tile += (int64_t)gridDim.x * nwarps) {
        int64_t mb, kc, b;
        tile_coords(tile, prm.nb, prm.nc, prm.tiles, mb, kc, b);
        const int64_t row0 = mb * M_, col0 = kc * cc;
        const T *src = dense + b * prm.batch_stride + row0 * prm.ld + col0;  // element (r, c) of the tile at src[r * ld + c]
        const int rows_ok = (int)(prm.M - row0 < M_ ? prm.M - row0 : M_);    // rows beyond M and columns beyond K read as zero
        const int cols_ok = (int)(prm.K - col0 < cc ? prm.K - col0 : cc);
        auto tile_at = [&](int r, int c) -> T { return (r < rows_ok && c < cols_ok) ? __ldg(src + (int64_t)r * prm.ld + c) : DT<T>::from_f32(0.f); };

        for (int c = lane; c < cc; c += 32) state[c] = -1;
        if (lane < C) cnt[lane] = 0;
        uint32_t full_mask = 0;  // bit p: pattern p holds g columns (warp-uniform)
        __syncwarp();

        // Deferred acceptance.  Every round with a proposal makes at least one (column, pattern) proposal that was never
        // made before, so cc * C rounds cannot be exceeded; real weights settle in a handful.
        // After the first round only the columns that were rejected or released propose again: they are kept as a list, so
        // that a late round with a handful of free columns costs a handful of iterations, not a sweep over the tile.
        for (int round = 0; round < cc * C + 2; round++) {
            const int F = round == 0 ? cc : *nfree;  // proposers of this round: every column, then the list
            if (lane < C) icnt[lane] = 0;
            __syncwarp();
            if (lane == 0) *nfree = 0;
            bool proposed = false;
            for (int e = lane; e < F; e += 32) {
                const int c = round == 0 ? e : (int)freel[e];
                prop_p[c] = -1;
                float a[M_];
#pragma unroll
                for (int r = 0; r < M_; r++) a[r] = fabsf(DT<T>::to_f32(tile_at(r, c)));
                uint32_t best_s = 0;  // a score of zero never wins: zero scores are placed by the closed form after the rounds
                int best_p = -1;
                if (full_mask == 0) {  // first round(s): every pattern is open, nothing but registers
                    // the sum starts from the first value (0 + x = x exactly for x >= 0) and zero scores are sorted out once,
                    // after the scan: a zero maximum means that every score of the column is zero
#pragma unroll
                    for (int p = 0; p < C; p++) {
                        float sc = a[ORD.row(p, 0)];
#pragma unroll
                        for (int i = 1; i < N_; i++) sc = __fadd_rn(sc, a[ORD.row(p, i)]);
                        const uint32_t sb = __float_as_uint(sc);
                        if (sb >= best_s) { best_s = sb; best_p = p; }
                    }
                    if (best_s == 0) best_p = -1;
                } else {
#pragma unroll
                    for (int p = 0; p < C; p++) {
                        float sc = a[ORD.row(p, 0)];
#pragma unroll
                        for (int i = 1; i < N_; i++) sc = __fadd_rn(sc, a[ORD.row(p, i)]);
                        const uint32_t sb = __float_as_uint(sc);
                        bool open = sb != 0 && sb >= best_s;
                        // full pattern: only a proposer that ranks above its weakest kept one gets in
                        if (open && ((full_mask >> p) & 1u)) open = above(sb, c, lscore[p * g + g - 1], lcol[p * g + g - 1]);
                        if (open) { best_s = sb; best_p = p; }
                    }
                }
                if (best_p < 0) continue;  // nothing above zero is open to this column: it waits for the zero phase
                proposed = true;
                prop_p[c] = (int16_t)best_p;
                park[c] = best_s;
                atomicAdd(&icnt[best_p], 1);
            }
            if (!__any_sync(0xffffffffu, proposed)) break;
            __syncwarp();
            int total;
            {   // exclusive prefix sum over the patterns (one per lane) -> start of every pattern's inbox segment
                const int mine = lane < C ? icnt[lane] : 0;
                int incl = mine;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += t;
                }
                if (lane < C) { ioff[lane] = incl - mine; icnt[lane] = 0; }  // icnt becomes the fill cursor of the segment
                total = __shfl_sync(0xffffffffu, incl, 31);
            }
            __syncwarp();
            for (int e = lane; e < F; e += 32) {
                const int c = round == 0 ? e : (int)freel[e];
                const int p = prop_p[c];
                if (p >= 0) inbox[ioff[p] + atomicAdd(&icnt[p], 1)] = (int16_t)c;
            }
            __syncwarp();  // the list has been read: the steps below refill it
            if (round == 0) {
                // all lists are empty: a proposal's place is its rank among the proposals of its pattern
                for (int e = lane; e < total; e += 32) {
                    const int c = inbox[e], p = prop_p[c];
                    const uint32_t sc = park[c];
                    const int e0 = ioff[p], e1 = e0 + icnt[p];
                    int rank = 0;
                    for (int j = e0; j < e1; j++) {
                        const int c2 = inbox[j];
                        rank += above(park[c2], c2, sc, c) ? 1 : 0;
                    }
                    if (rank < g) { lscore[p * g + rank] = sc; lcol[p * g + rank] = (int16_t)c; state[c] = (int16_t)p; }
                    else freel[atomicAdd(nfree, 1)] = (int16_t)c;
                }
                if (lane < C) cnt[lane] = min(icnt[lane], g);
            } else if (lane < C) {
                const int p = lane;
                uint32_t *ls = lscore + p * g;
                int16_t *lc = lcol + p * g;
                int L = cnt[p];
                const int e0 = ioff[p], e1 = e0 + icnt[p];
                for (int e = e0; e < e1; e++) {
                    const int c = inbox[e];
                    const uint32_t sc = park[c];
                    if (L == g) {
                        if (!above(sc, c, ls[g - 1], lc[g - 1])) {  // stays free
                            freel[atomicAdd(nfree, 1)] = (int16_t)c;
                            continue;
                        }
                        state[lc[g - 1]] = -1;                          // the weakest kept proposer is released
                        freel[atomicAdd(nfree, 1)] = lc[g - 1];
                        L = g - 1;
                    }
                    int j = L;
                    while (j > 0 && above(sc, c, ls[j - 1], lc[j - 1])) { ls[j] = ls[j - 1]; lc[j] = lc[j - 1]; j--; }
                    ls[j] = sc;
                    lc[j] = (int16_t)c;
                    L++;
                    state[c] = (int16_t)p;
                }
                cnt[p] = L;
            }
            __syncwarp();
            full_mask = __ballot_sync(0xffffffffu, lane < C && cnt[lane] == g);
        }
        __syncwarp();
        // zero phase on the split lists: same closed form as sparsify_zero_phase, columns only
        {
            const int mine = lane < C ? g - cnt[lane] : 0;  // free places of pattern `lane`
            int incl = mine;                                 // inclusive suffix sum over lanes
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_down_sync(0xffffffffu, incl, d);
                if (lane + d < 32) incl += t;
            }
            if (lane < C) { icnt[lane] = mine; ioff[lane] = incl - mine; }  // rem[p], cum[p] = free places in larger patterns
            __syncwarp();
            int above_cnt = 0;
            for (int k = (cc - 1) / 32; k >= 0; k--) {
                const int c = k * 32 + lane;
                const bool is_free = c < cc && state[c] < 0;
                const uint32_t mask = __ballot_sync(0xffffffffu, is_free);
                if (is_free) {
                    const int i = above_cnt + __popc(lane == 31 ? 0u : (mask >> (lane + 1)));  // free columns with a larger index
                    int p = C - 1;
                    while (p > 0 && ioff[p] + icnt[p] <= i) p--;  // largest pattern whose range of places contains i
                    lcol[p * g + cnt[p] + (i - ioff[p])] = (int16_t)c;
                    state[c] = (int16_t)p;
                }
                above_cnt += __popc(mask);
            }
            __syncwarp();
        }

        int16_t *idx_out = prm.idx + tile * cc;
        T *val_out = val + tile * (int64_t)cc * N_;
        if ((cc & 7) == 0 && (reinterpret_cast<uintptr_t>(idx_out) & 15) == 0) {
            for (int s0 = lane * 8; s0 < cc; s0 += 256) *reinterpret_cast<uint4 *>(idx_out + s0) = *reinterpret_cast<const uint4 *>(lcol + s0);
        } else {
            for (int s0 = lane; s0 < cc; s0 += 32) idx_out[s0] = lcol[s0];
        }
        const int nvals = cc * N_;
        if ((nvals % V) == 0 && (reinterpret_cast<uintptr_t>(val_out) & 15) == 0) {
            for (int v = lane * V; v < nvals; v += 32 * V) {
                __align__(16) T out[V];
#pragma unroll
                for (int u = 0; u < V; u++) {
                    const int e = v + u, s0 = e / N_, t = e % N_;
                    const int c = lcol[s0], p = g_pow2 ? (s0 >> g_shift) : s0 / g;
                    out[u] = tile_at((int)ord[p * N_ + t], c);
                }
                *reinterpret_cast<uint4 *>(val_out + v) = *reinterpret_cast<const uint4 *>(out);
            }
        } else {
            for (int e = lane; e < nvals; e += 32) {
                const int s0 = e / N_, t = e % N_;
                const int c = lcol[s0], p = s0 / g;
                val_out[e] = tile_at((int)ord[p * N_ + t], c);
            }
        }
        __syncwarp();
    }
}

// ---- several tiles per warp: few patterns ----------------------------------------------------------------------------
// L lanes per tile, 32 / L tiles per warp.  The selection is bound by instructions and by the latency of its dependent steps;
// with a warp per tile most lanes idle after the first round, where a few displaced columns are left (counted on random
// weights, 2:4, g = 16: 12 more proposals per 96-column tile).
//   round 0   every column's best pattern from registers, four columns per lane and step; the proposals are grouped by
//             pattern, and a proposal's place in its pattern's sorted list is its rank among them.
//   rounds    the first L columns of the tile's queue of displaced columns propose, each to the best pattern that would keep
//             it (a pattern's threshold is the score of its weakest kept entry); the lanes that own the patterns insert what
//             they were sent, at the same time, and queue the entry that falls out.
//   zeros     scores of zero are placed by the closed form of sparsify_zero_phase.
// Entries are 64-bit keys, score above column + 1: one comparison is the format's order.  The tile is staged in shared memory
// (16-byte asynchronous copies where the alignment allows).  A tile's slab is 32 bytes more than a multiple of 128, so that
// the tiles of a warp use different banks.  TWICE: the ranks of round 0 use the tile's own place and it is staged again (from
// L2) for what follows; more warps are then resident, which pays where the grouped proposals are not small beside the tile.
// 4096 x 4096, before (a warp per tile) and now: 2:4 fp32 187 -> 104 us, bf16 184 -> 89, 1:4 fp32 173 -> 84, 1:8 fp32 93 -> 68
// (there all 32 lanes), 1:8 g = 4 fp16 195 -> 68.  Tried and slower: sorting a pattern per lane by a network (139 where this
// took 121), the tile left in global memory for more resident warps (129).
struct SparsifyLanes { int xs, x, in, list, prop, thr, sent, cnt, off, queue, qmask, zmask, words, total; };
__host__ __device__ inline SparsifyLanes sparsify_lanes(int m, int cc, int C, int lanes, int es, bool twice) {
    SparsifyLanes l;
    const int quads = (cc + 3) / 4;
    int o = 0;
    l.words = ((quads + lanes - 1) / lanes * 4 + 31) / 32;  // one bit per column of a lane
    l.xs = quads * 4;                                       // row stride of the staged tile
    const int x_bytes = (m * l.xs * es + 15) & ~15, in_bytes = (cc + 2 * C) * 8;
    l.x = o;                                                // [m][xs] the tile
    l.in = twice ? o : o + x_bytes;                         // round 0: proposals grouped by pattern, every group padded to 2
    o += twice ? (x_bytes > in_bytes ? x_bytes : in_bytes) : x_bytes + in_bytes;
    l.list = o = (o + 15) & ~15; o += l.xs * 8;             // [C][g] kept entries, descending (round 0: by column)
    l.prop = o;   o += lanes * 8;                           // later rounds: the proposal of every lane
    l.thr = o = (o + 15) & ~15; o += C * 4;                 // smallest score that a pattern may still keep
    l.sent = o;   o += C * 4;                               // lanes that propose to the pattern
    l.cnt = o;    o += C * 4;
    l.off = o;    o += C * 4;
    l.zmask = o;  o += lanes * l.words * 4;                 // columns with no open pattern above zero
    l.qmask = 1;
    while (l.qmask < cc) l.qmask <<= 1;
    l.queue = o;  o += l.qmask * 2 + 4;                     // ring of displaced columns, its write position
    l.qmask--;
    l.total = ((o + 127) & ~127) + 32;
    return l;
}

template <typename T> __device__ __forceinline__ void load_quad(const T *p, float *a) {  // magnitudes of four staged neighbours
    if constexpr (sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        a[0] = fabsf(v.x); a[1] = fabsf(v.y); a[2] = fabsf(v.z); a[3] = fabsf(v.w);
    } else {
        __align__(8) T v[4];
        *reinterpret_cast<uint2 *>(v) = *reinterpret_cast<const uint2 *>(p);
#pragma unroll
        for (int u = 0; u < 4; u++) a[u] = fabsf(DT<T>::to_f32(v[u]));
    }
}

template <int N_, int M_, int L, bool TWICE, typename T>
__global__ void __launch_bounds__(128, 5) sparsify_lanes_kernel(SparsifyParams prm) {
    extern __shared__ __align__(16) char smem[];
    constexpr Order<N_, M_> ORD{};
    constexpr int C = Order<N_, M_>::C, TILES = 32 / L;
    static_assert(C <= 31, "pattern 31 marks a column without a proposal");
    constexpr int V = 16 / (int)sizeof(T);
    constexpr uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int sub = lane / L, sl = lane % L;  // tile of the warp, lane of the tile
    const int g = prm.g, cc = prm.cc;
    int8_t *ord = reinterpret_cast<int8_t *>(smem);  // run-time copy of the table for the output stage
    constexpr int ORD_BYTES = (C * N_ + 15) & ~15;
    for (int i = threadIdx.x; i < C * N_; i += blockDim.x) ord[i] = (int8_t)ORD.v[(i / N_) * Order<N_, M_>::LD + (i % N_)];
    __syncthreads();

    const SparsifyLanes lay = sparsify_lanes(M_, cc, C, L, (int)sizeof(T), TWICE);
    char *slab = smem + ORD_BYTES + (warp * TILES + sub) * lay.total;
    T *x = reinterpret_cast<T *>(slab + lay.x);
    uint64_t *in = reinterpret_cast<uint64_t *>(slab + lay.in), *list = reinterpret_cast<uint64_t *>(slab + lay.list);
    uint64_t *prop = reinterpret_cast<uint64_t *>(slab + lay.prop);
    uint32_t *thr = reinterpret_cast<uint32_t *>(slab + lay.thr), *sent = reinterpret_cast<uint32_t *>(slab + lay.sent);
    int *cnt = reinterpret_cast<int *>(slab + lay.cnt), *off = reinterpret_cast<int *>(slab + lay.off);
    uint16_t *queue = reinterpret_cast<uint16_t *>(slab + lay.queue);
    const int words = lay.words, xs = lay.xs, quads = xs >> 2, qmask = lay.qmask;
    uint32_t *tail = reinterpret_cast<uint32_t *>(queue + qmask + 1);
    uint32_t *zmask = reinterpret_cast<uint32_t *>(slab + lay.zmask), *my_z = zmask + sl * words;
    const bool g_pow2 = (g & (g - 1)) == 0;
    const int g_shift = 31 - __clz(g);
    const T *dense = static_cast<const T *>(prm.dense);
    T *val = static_cast<T *>(prm.val);
    auto displace = [&](int c) { queue[atomicAdd(tail, 1u) & qmask] = (uint16_t)c; };  // a column is in the queue at most once
    auto col_of = [](uint64_t key) { return (int)(uint32_t)key - 1; };

    const int64_t stride = (int64_t)gridDim.x * nwarps * TILES;
    for (int64_t tile0 = ((int64_t)blockIdx.x * nwarps + warp) * TILES; tile0 < prm.tiles; tile0 += stride) {
        const int64_t tile = tile0 + sub;
        const bool live = tile < prm.tiles;
        int64_t mb, kc, b;
        tile_coords(live ? tile : tile0, prm.nb, prm.nc, prm.tiles, mb, kc, b);
        const int64_t row0 = mb * M_, col0 = kc * cc;
        const T *src = dense + b * prm.batch_stride + row0 * prm.ld + col0;  // element (r, c) of the tile at src[r * ld + c]
        const int rows_ok = (int)(prm.M - row0 < M_ ? prm.M - row0 : M_);    // rows beyond M and columns beyond K read as zero
        const int cols_ok = (int)(prm.K - col0 < cc ? prm.K - col0 : cc);
        auto global_at = [&](int r, int c) -> T { return (r < rows_ok && c < cols_ok) ? __ldg(src + r * prm.ld + c) : DT<T>::from_f32(0.f); };
        // ---- the tile
        auto stage = [&]() {
            if (rows_ok == M_ && cols_ok == cc && (cc % V) == 0 && (prm.ld % V) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
                for (int r = 0; r < M_; r++)
                    for (int v = sl * V; v < cc; v += L * V) cp_async_16(x + r * xs + v, src + r * prm.ld + v);
                cp_async_commit();
            } else {
                for (int r = 0; r < M_; r++)
                    for (int c = sl; c < xs; c += L) x[r * xs + c] = global_at(r, c);
            }
        };
        stage();
        for (int p = sl; p < C; p += L) cnt[p] = 0;
        for (int w = 0; w < words; w++) my_z[w] = 0;
        if (sl == 0) *tail = 0;
        cp_async_wait<0>();
        __syncwarp();

        // ---- round 0: proposals.  By column: score, number within the pattern (in no order), pattern (31: none)
        for (int q = sl, bit = 0; q < quads; q += L, bit += 4) {
            float a[M_][4];
#pragma unroll
            for (int r = 0; r < M_; r++) load_quad(x + r * xs + q * 4, a[r]);
            uint32_t best_s[4] = {0, 0, 0, 0};
            int best_p[4] = {0, 0, 0, 0};
            // the sum starts from the first value (0 + x = x exactly for x >= 0); a zero maximum means that every score is zero
#pragma unroll
            for (int p = 0; p < C; p++)
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    float sc = a[ORD.row(p, 0)][u];
#pragma unroll
                    for (int i = 1; i < N_; i++) sc = __fadd_rn(sc, a[ORD.row(p, i)][u]);
                    const uint32_t sb = __float_as_uint(sc);
                    if (sb >= best_s[u]) { best_s[u] = sb; best_p[u] = p; }
                }
            uint32_t zero = 0, w[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                w[u] = 31;
                if (best_s[u] != 0) w[u] = (uint32_t)best_p[u] | ((uint32_t)atomicAdd(&cnt[best_p[u]], 1) << 5);
                else if (q * 4 + u < cc) zero |= 1u << u;
            }
            if (zero) my_z[bit >> 5] |= zero << (bit & 31);
            uint4 *by_col = reinterpret_cast<uint4 *>(list + q * 4);
            by_col[0] = make_uint4(w[0], best_s[0], w[1], best_s[1]);
            by_col[1] = make_uint4(w[2], best_s[2], w[3], best_s[3]);
        }
        __syncwarp();
        for (int p = sl; p < C; p += L) {
            int o = 0;
            for (int r = 0; r < p; r++) o += (cnt[r] + 1) & ~1;
            off[p] = o;
            if (cnt[p] & 1) in[o + cnt[p]] = 0;
        }
        __syncwarp();
        for (int c = sl; c < cc; c += L) {
            const uint64_t e = list[c];
            const int p = (int)(e & 31);
            if (p < 31) in[off[p] + ((uint32_t)e >> 5)] = (e & 0xffffffff00000000ull) | (uint32_t)((c + 1) | (p << 16));
        }
        __syncwarp();
        // a lane ranks two neighbours at a time: groups are padded to two, so they share a pattern
        const int slots = off[C - 1] + cnt[C - 1];
        for (int e = 2 * sl; e < slots; e += 2 * L) {
            const ulonglong2 key = *reinterpret_cast<const ulonglong2 *>(in + e);
            const int p = (int)((uint32_t)key.x >> 16);
            const ulonglong2 *from = reinterpret_cast<const ulonglong2 *>(in + off[p]);
            const int pairs = (cnt[p] + 1) >> 1;
            int rank0 = 0, rank1 = 0;
#pragma unroll 2
            for (int j = 0; j < pairs; j++) {
                const ulonglong2 v = from[j];
                rank0 += v.x > key.x ? 1 : 0;
                rank1 += v.x > key.y ? 1 : 0;
                rank0 += v.y > key.x ? 1 : 0;
                rank1 += v.y > key.y ? 1 : 0;
            }
            auto place = [&](uint64_t k, int rank) {
                const int c1 = (int)(k & 0xffff);
                if (rank < g) list[p * g + rank] = (k & 0xffffffff00000000ull) | (uint32_t)c1;
                else displace(c1 - 1);
            };
            place(key.x, rank0);
            if (key.y != 0) place(key.y, rank1);  // zero: padding
        }
        __syncwarp();
        if (TWICE) stage();
        for (int p = sl; p < C; p += L) {
            const int n = min(cnt[p], g);
            cnt[p] = n;
            thr[p] = n == g ? (uint32_t)(list[p * g + g - 1] >> 32) : 1u;
            sent[p] = 0;
        }
        if (TWICE) cp_async_wait<0>();
        __syncwarp();

        // ---- later rounds.  Every round with a proposal makes at least one (column, pattern) proposal that was never made
        // before, so cc * C rounds cannot be exceeded.
        uint32_t head = 0;
        for (int round = 0; round < cc * C; round++) {
            const int queued = (int)(*tail - head);
            const bool active = sl < queued;
            if (!__any_sync(FULL, active)) break;
            if (active) {
                const int c = queue[(head + sl) & qmask];
                float a[M_];
#pragma unroll
                for (int r = 0; r < M_; r++) a[r] = fabsf(DT<T>::to_f32(x[r * xs + c]));
                uint32_t best_s = 0;
                int best_p = -1;
                bool tie = false;
#pragma unroll
                for (int p = 0; p < C; p++) {
                    float sc = a[ORD.row(p, 0)];
#pragma unroll
                    for (int i = 1; i < N_; i++) sc = __fadd_rn(sc, a[ORD.row(p, i)]);
                    const uint32_t sb = __float_as_uint(sc), t = thr[p];
                    tie |= sb == t;
                    if (sb >= best_s && sb >= t) { best_s = sb; best_p = p; }
                }
                if (tie) {  // a score like some pattern's weakest: if it is full, only the larger column gets in
                    best_s = 0;
                    best_p = -1;
                    for (int p = 0; p < C; p++) {
                        float sc = fabsf(DT<T>::to_f32(x[(int)ord[p * N_] * xs + c]));
#pragma unroll
                        for (int i = 1; i < N_; i++) sc = __fadd_rn(sc, fabsf(DT<T>::to_f32(x[(int)ord[p * N_ + i] * xs + c])));
                        const uint32_t sb = __float_as_uint(sc), t = thr[p];
                        if (sb < best_s || sb < t || (sb == t && cnt[p] == g && c < col_of(list[p * g + g - 1]))) continue;
                        best_s = sb;
                        best_p = p;
                    }
                }
                if (best_p >= 0) {
                    prop[sl] = ((uint64_t)best_s << 32) | (uint32_t)(c + 1);
                    atomicOr(&sent[best_p], 1u << sl);
                } else {
                    // nothing above zero is open: placed by the zero phase.  Column c is bit (c / 4) / L * 4 + c % 4 of lane (c / 4) % L
                    const int q = c >> 2, bit = (q / L) * 4 + (c & 3);
                    atomicOr(&zmask[(q % L) * words + (bit >> 5)], 1u << (bit & 31));
                }
            }
            head += (uint32_t)min(queued, L);
            __syncwarp();
            for (int p = sl; p < C; p += L) {
                uint32_t from = sent[p];
                if (from == 0) continue;
                sent[p] = 0;
                uint64_t *lp = list + p * g;
                int n = cnt[p];
                for (; from; from &= from - 1) {
                    const uint64_t key = prop[__ffs(from) - 1];
                    int j = n;
                    if (n == g) {
                        const uint64_t last = lp[--j];
                        displace(col_of(key < last ? key : last));  // the weakest falls out, a kept entry or the proposal
                        if (key < last) continue;
                    } else {
                        n++;
                    }
                    for (; j > 0; j--) {
                        const uint64_t prev = lp[j - 1];
                        if (prev > key) break;
                        lp[j] = prev;
                    }
                    lp[j] = key;
                }
                cnt[p] = n;
                if (n == g) thr[p] = (uint32_t)(lp[g - 1] >> 32);
            }
            __syncwarp();
        }

        // ---- zero phase (padded columns, pruned weights): see sparsify_zero_phase
        uint32_t zeros = 0;
        for (int w = 0; w < words; w++) zeros |= my_z[w];
        if (__any_sync(FULL, zeros != 0)) {
            for (int p = sl; p < C; p += L) {
                int o = 0;
                for (int q = p + 1; q < C; q++) o += g - cnt[q];
                off[p] = o;  // free places in larger patterns
            }
            __syncwarp();
            constexpr uint32_t TILE_LANES = L == 32 ? FULL : (1u << (L & 31)) - 1u;
            int above = 0;  // free columns with larger indices
            for (int k = (quads - 1) / L; k >= 0; k--) {
                const uint32_t nib = (my_z[k >> 3] >> ((k & 7) * 4)) & 15u;
                int later = 0, all = 0;  // free columns of larger lanes, of all lanes
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t mask = (__ballot_sync(FULL, (nib >> u) & 1u) >> (sub * L)) & TILE_LANES;
                    all += __popc(mask);
                    later += __popc(sl == 31 ? 0u : mask >> (sl + 1));
                }
                for (int u = 3; u >= 0; u--) {
                    if (((nib >> u) & 1u) == 0) continue;
                    const int i = above + later++;
                    int p = C - 1;
                    while (p > 0 && off[p] + (g - cnt[p]) <= i) p--;  // largest pattern whose range of places contains i
                    list[p * g + cnt[p] + (i - off[p])] = (uint32_t)((k * L + sl) * 4 + u + 1);
                }
                above += all;
            }
        }
        __syncwarp();

        // ---- output
        if (live) {
            uint16_t *idx_out = reinterpret_cast<uint16_t *>(prm.idx) + tile * cc;
            T *val_out = val + tile * (int64_t)cc * N_;
            if ((cc & 3) == 0 && (reinterpret_cast<uintptr_t>(idx_out) & 7) == 0) {
                for (int s0 = sl * 4; s0 < cc; s0 += L * 4) {
                    const ulonglong2 e0 = *reinterpret_cast<const ulonglong2 *>(list + s0), e1 = *reinterpret_cast<const ulonglong2 *>(list + s0 + 2);
                    const uint32_t lo = (uint32_t)(col_of(e0.x) | (col_of(e0.y) << 16)), hi = (uint32_t)(col_of(e1.x) | (col_of(e1.y) << 16));
                    *reinterpret_cast<uint2 *>(idx_out + s0) = make_uint2(lo, hi);
                }
            } else {
                for (int s0 = sl; s0 < cc; s0 += L) idx_out[s0] = (uint16_t)col_of(list[s0]);
            }
            const int nvals = cc * N_;
            if ((nvals % V) == 0 && (reinterpret_cast<uintptr_t>(val_out) & 15) == 0) {
                for (int v = sl * V; v < nvals; v += L * V) {
                    __align__(16) T out[V];
#pragma unroll
                    for (int u = 0; u < V; u++) {
                        const int e = v + u, s0 = e / N_, t = e % N_;
                        const int p = g_pow2 ? (s0 >> g_shift) : s0 / g;
                        out[u] = x[(int)ord[p * N_ + t] * xs + col_of(list[s0])];
                    }
                    *reinterpret_cast<uint4 *>(val_out + v) = *reinterpret_cast<const uint4 *>(out);
                }
            } else {
                for (int e = sl; e < nvals; e += L) {
                    const int s0 = e / N_, t = e % N_;
                    val_out[e] = x[(int)ord[(s0 / g) * N_ + t] * xs + col_of(list[s0])];
                }
            }
        }
        __syncwarp();
    }
}

// Launch with L lanes per tile; *served = false when fewer than `min_warps` warps would be resident per SM.
template <int N_, int M_, int L, bool TWICE> static int sparsify_lanes_launch(int dtype, const SparsifyParams &p, int min_warps, bool *served, cudaStream_t st) {
    const int es = (int)dtype_size(dtype);
    constexpr int C = Order<N_, M_>::C, ORD_BYTES = (C * N_ + 15) & ~15, TILES = 32 / L;
    const size_t per_warp = (size_t)TILES * sparsify_lanes(M_, p.cc, C, L, es, TWICE).total;
    int warps = 0, resident = 0;  // whatever keeps the most warps resident; on a tie the smaller CTA
    for (int w = 1; w <= 4; w++) {
        const size_t cta = ORD_BYTES + w * per_warp;
        if (cta > 226 * 1024) break;
        int per_sm = (int)((size_t)227 * 1024 / (cta + 1024));
        if (per_sm > 24) per_sm = 24;
        if (per_sm * w > resident) { resident = per_sm * w; warps = w; }
    }
    *served = resident >= min_warps;
    if (!*served) return NMG_OK;
    const size_t smem = ORD_BYTES + warps * per_warp;
    const int64_t ctas = (p.tiles + warps * TILES - 1) / (warps * TILES), cap = (int64_t)sm_count() * 64;
    NMG_DISPATCH_DTYPE(dtype, T, {
        NMG_ALLOW_SMEM(smem, sparsify_lanes_kernel<N_, M_, L, TWICE, T>);
        sparsify_lanes_kernel<N_, M_, L, TWICE, T><<<(unsigned)(ctas < cap ? ctas : cap), warps * 32, smem, st>>>(p);
    });
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

// =====================================================================================================
// Densifier: one CTA per tile.  The tile's idx is inverted in shared memory (column -> slot), val is staged,
// and the m x cc block is written row by row with coalesced stores; zeros are produced by the same stores, so
// the output needs no separate clearing pass.
// =====================================================================================================
struct DensifyParams {
    const void *val;
    const int16_t *idx;
    void *dense;
    const int8_t *slot_of_row;  // [C][m] device
    int64_t M, K, ld, batch_stride;
    int64_t nb, nc, tiles;
    int n, m, g, C, cc;
};

template <typename T>
__global__ void __launch_bounds__(128) densify_kernel(DensifyParams prm) {
    extern __shared__ __align__(16) char smem[];
    const int n = prm.n, m = prm.m, g = prm.g, C = prm.C, cc = prm.cc;
    T *sval = reinterpret_cast<T *>(smem);                                             // [cc][n]
    int16_t *pos = reinterpret_cast<int16_t *>(smem + (((size_t)cc * n * sizeof(T) + 15) & ~(size_t)15));  // [cc]
    int8_t *sor = reinterpret_cast<int8_t *>(pos + cc);                                // [C][m]
    for (int i = threadIdx.x; i < C * m; i += blockDim.x) sor[i] = prm.slot_of_row[i];

    const T *val = static_cast<const T *>(prm.val);
    T *dense = static_cast<T *>(prm.dense);
    for (int64_t tile = blockIdx.x; tile < prm.tiles; tile += gridDim.x) {
        int64_t mb, kc, b;
        tile_coords(tile, prm.nb, prm.nc, prm.tiles, mb, kc, b);
        __syncthreads();
        for (int c = threadIdx.x; c < cc; c += blockDim.x) pos[c] = -1;
        constexpr int V = 16 / (int)sizeof(T);  // elements per 16-byte access
        const T *vsrc = val + tile * (int64_t)cc * n;
        if (((cc * n) % V) == 0 && (reinterpret_cast<uintptr_t>(vsrc) & 15) == 0) {
            for (int e = threadIdx.x * V; e < cc * n; e += blockDim.x * V)
                *reinterpret_cast<uint4 *>(sval + e) = __ldg(reinterpret_cast<const uint4 *>(vsrc + e));
        } else {
            for (int e = threadIdx.x; e < cc * n; e += blockDim.x) sval[e] = vsrc[e];
        }
        __syncthreads();
        const int16_t *isrc = prm.idx + tile * cc;
        if ((cc & 7) == 0 && (reinterpret_cast<uintptr_t>(isrc) & 15) == 0) {
            for (int s8 = threadIdx.x * 8; s8 < cc; s8 += blockDim.x * 8) {
                const uint4 iv = __ldg(reinterpret_cast<const uint4 *>(isrc + s8));
                const int16_t *ci = reinterpret_cast<const int16_t *>(&iv);
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (ci[u] >= 0 && ci[u] < cc) pos[ci[u]] = (int16_t)(s8 + u);  // a malformed index is ignored, never dereferenced
            }
        } else {
            for (int s = threadIdx.x; s < cc; s += blockDim.x) {
                const int c = isrc[s];
                if (c >= 0 && c < cc) pos[c] = (int16_t)s;
            }
        }
        __syncthreads();
        T *dst = dense + b * prm.batch_stride;
        const int64_t col0 = kc * cc;
        // 16-byte stores where the row piece allows it: every thread assembles V consecutive columns of one row
        const bool vec = (cc % V) == 0 && col0 + cc <= prm.K && (prm.ld % V) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
        if (vec) {
            const int per_row = cc / V;
            for (int v = threadIdx.x; v < m * per_row; v += blockDim.x) {
                const int r = v / per_row, c0 = (v - r * per_row) * V;
                const int64_t row = mb * m + r;
                if (row >= prm.M) continue;
                __align__(16) T out[V];
#pragma unroll
                for (int u = 0; u < V; u++) {
                    const int sl = pos[c0 + u];
                    T val_u = DT<T>::from_f32(0.f);
                    if (sl >= 0) {
                        const int t = sor[(sl / g) * m + r];
                        if (t >= 0) val_u = sval[sl * n + t];
                    }
                    out[u] = val_u;
                }
                *reinterpret_cast<uint4 *>(dst + row * prm.ld + col0 + c0) = *reinterpret_cast<const uint4 *>(out);
            }
            continue;
        }
        for (int r = 0; r < m; r++) {
            const int64_t row = mb * m + r;
            if (row >= prm.M) break;
            T *drow = dst + row * prm.ld + kc * cc;
            for (int c = threadIdx.x; c < cc; c += blockDim.x) {
                if (kc * cc + c >= prm.K) break;
                const int s = pos[c];
                T v = DT<T>::from_f32(0.f);
                if (s >= 0) {
                    const int t = sor[(s / g) * m + r];
                    if (t >= 0) v = sval[s * n + t];
                }
                drow[c] = v;
            }
        }
    }
}

// =====================================================================================================
// Layout gather: the values of a dense tensor at the positions an existing (idx) layout keeps.  One warp per tile; the
// tile's rows are short contiguous spans, so the indexed reads hit L1 / L2.
// =====================================================================================================
struct GatherParams {
    const void *dense;
    const int16_t *idx;
    void *val;
    const int8_t *order;  // [C][n] device
    int64_t M, K, ld, batch_stride;
    int64_t nb, nc, tiles;
    int n, m, g, C, cc;
};

template <typename T>
__global__ void __launch_bounds__(256) gather_layout_kernel(GatherParams prm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int n = prm.n, m = prm.m, g = prm.g, cc = prm.cc;
    const T *dense = static_cast<const T *>(prm.dense);
    T *val = static_cast<T *>(prm.val);
    for (int64_t tile = (int64_t)blockIdx.x * nwarps + warp; tile < prm.tiles; tile += (int64_t)gridDim.x * nwarps) {
        int64_t mb, kc, b;
        tile_coords(tile, prm.nb, prm.nc, prm.tiles, mb, kc, b);
        const T *src = dense + b * prm.batch_stride;
        const int16_t *isrc = prm.idx + tile * cc;
        T *vdst = val + tile * (int64_t)cc * n;
        for (int s = lane; s < cc; s += 32) {
            const int c = isrc[s];
            const int8_t *o = prm.order + (s / g) * n;
            const int64_t col = kc * cc + c;
            const bool col_ok = c >= 0 && c < cc && col < prm.K;  // a malformed index reads as zero, never dereferenced
            for (int t = 0; t < n; t++) {
                const int64_t row = mb * m + o[t];
                vdst[s * n + t] = (col_ok && row < prm.M) ? src[row * prm.ld + col] : DT<T>::from_f32(0.f);
            }
        }
    }
}

static int check_dtype(int dtype) {
    if (dtype != NMG_F32 && dtype != NMG_F16 && dtype != NMG_BF16)
        NMG_FAIL(NMG_ERR_INVALID, "dtype must be NMG_F32, NMG_F16 or NMG_BF16, got %d", dtype);
    return NMG_OK;
}

}  // namespace nmg

using namespace nmg;

extern "C" int nmg_sparsify(const void *dense, int64_t batch, int64_t M, int64_t K, int64_t ld_dense,
                            int64_t batch_stride, int n, int m, int g, int dtype, void *val, int16_t *idx,
                            void *stream) {
    Geo geo;
    int rc = make_geo(M, K, n, m, g, &geo);
    if (rc) return rc;
    if ((rc = check_dtype(dtype))) return rc;
    if (!dense || !val || !idx) NMG_FAIL(NMG_ERR_INVALID, "dense, val and idx must be non-NULL");
    if (n < 1) NMG_FAIL(NMG_ERR_INVALID, "the sparsifier needs n >= 1");
    if (batch < 1 || ld_dense < K || (batch > 1 && batch_stride < M * ld_dense))
        NMG_FAIL(NMG_ERR_INVALID, "bad batch / leading dimension (batch=%lld ld=%lld)", (long long)batch, (long long)ld_dense);
    PatternTable tab;
    if ((rc = get_pattern_table(n, m, &tab))) return rc;

    SparsifyParams p{};
    p.dense = dense; p.val = val; p.idx = idx; p.order = tab.order;
    p.M = M; p.K = K; p.ld = ld_dense; p.batch_stride = batch_stride;
    p.nb = geo.nb; p.nc = geo.nc; p.tiles = batch * geo.nb * geo.nc;
    p.n = n; p.m = m; p.g = g; p.C = geo.C; p.cc = geo.cc;
    cudaStream_t st = (cudaStream_t)stream;
    // whole: tiles are staged by 16-byte copies, cheap enough to be made twice
    const int V = 16 / (int)dtype_size(dtype);
    const bool whole = geo.cc % V == 0 && ld_dense % V == 0 && (batch == 1 || batch_stride % V == 0) && (reinterpret_cast<uintptr_t>(dense) & 15) == 0;
    // Few patterns: several tiles per warp.  Eight lanes per tile when that leaves at least twelve resident warps to hide the
    // latency of the shared memory, else a warp per tile down to four; larger tiles, and 16 or 28 patterns (whose later rounds
    // keep 32 lanes busy: 1:16 68 us against 74 to 102, 2:8 152 against 158), go to the kernel that does not stage the tile.
#define NMG_SPARSIFY_CASE(N_, M_)                                                                     \
    if (n == N_ && m == M_) {                                                                         \
        bool served = false;                                                                          \
        if (M_ == 4 && whole && ((rc = sparsify_lanes_launch<N_, M_, 8, M_ == 4>(dtype, p, 12, &served, st)) || served)) return rc; \
        if ((rc = sparsify_lanes_launch<N_, M_, 8, false>(dtype, p, 12, &served, st)) || served) return rc;  \
        if ((rc = sparsify_lanes_launch<N_, M_, 32, false>(dtype, p, 4, &served, st)) || served) return rc;  \
    }
    NMG_SPARSIFY_CASE(1, 4)
    NMG_SPARSIFY_CASE(2, 4)
    NMG_SPARSIFY_CASE(1, 8)
#undef NMG_SPARSIFY_CASE
    const bool specialised = (n == 1 && (m == 4 || m == 8 || m == 16)) || (n == 2 && (m == 4 || m == 8));
    const size_t slab = specialised ? sparsify_lean(geo.cc, geo.C).total : sparsify_slab(m, geo.cc, geo.C, dtype_size(dtype)).total;
    const size_t ord_bytes = ((size_t)geo.C * n + 15) & ~(size_t)15;
    const size_t budget = 200 * 1024;
    if (ord_bytes + slab > budget)
        NMG_FAIL(NMG_ERR_UNSUPPORTED, "tile of m=%d x %d columns needs %zu bytes of shared memory (limit %zu)", m, geo.cc,
                 ord_bytes + slab, budget);
    // warps per CTA: whatever keeps the most warps resident per SM (227 KB of shared memory, at most 8 warps per CTA); on a
    // tie the smaller CTA, for a finer tail
    int warps = 1, best_resident = 0;
    for (int w = 1; w <= 8; w++) {
        const size_t per_cta = ord_bytes + (size_t)w * slab + 1024;  // + the per-CTA reservation of the driver
        if (per_cta > 227 * 1024) break;
        int per_sm = (int)((size_t)227 * 1024 / per_cta);
        if (per_sm > 32) per_sm = 32;
        if (per_sm * w > 64) per_sm = 64 / w;
        if (per_sm * w > best_resident) { best_resident = per_sm * w; warps = w; }
    }
    p.slab_bytes = (int)slab;
    const size_t smem = ord_bytes + warps * slab;
    int64_t ctas = (p.tiles + warps - 1) / warps;
    const int64_t max_ctas = (int64_t)sm_count() * 16;
    if (ctas > max_ctas) ctas = max_ctas;
    bool launched = false;
#define NMG_SPARSIFY_CASE(N_, M_)                                                                                     \
    if (!launched && n == N_ && m == M_) {                                                                            \
        NMG_DISPATCH_DTYPE(dtype, T, {                                                                                \
            NMG_ALLOW_SMEM(smem, sparsify_nm_kernel<N_, M_, T>); \
            sparsify_nm_kernel<N_, M_, T><<<(unsigned)ctas, warps * 32, smem, st>>>(p);                               \
        });                                                                                                           \
        launched = true;                                                                                              \
    }
    NMG_SPARSIFY_CASE(1, 4)
    NMG_SPARSIFY_CASE(2, 4)
    NMG_SPARSIFY_CASE(1, 8)
    NMG_SPARSIFY_CASE(2, 8)
    NMG_SPARSIFY_CASE(1, 16)
#undef NMG_SPARSIFY_CASE
    if (!launched) {
        NMG_DISPATCH_DTYPE(dtype, T, {
            NMG_ALLOW_SMEM(smem, sparsify_kernel<T>);
            sparsify_kernel<T><<<(unsigned)ctas, warps * 32, smem, st>>>(p);
        });
    }
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

extern "C" int nmg_densify(const void *val, const int16_t *idx, int64_t batch, int64_t M, int64_t K, int n, int m,
                           int g, int dtype, void *dense, int64_t ld_dense, int64_t batch_stride, void *stream) {
    Geo geo;
    int rc = make_geo(M, K, n, m, g, &geo);
    if (rc) return rc;
    if ((rc = check_dtype(dtype))) return rc;
    if (!dense || !val || !idx) NMG_FAIL(NMG_ERR_INVALID, "dense, val and idx must be non-NULL");
    if (batch < 1 || ld_dense < K || (batch > 1 && batch_stride < M * ld_dense))
        NMG_FAIL(NMG_ERR_INVALID, "bad batch / leading dimension (batch=%lld ld=%lld)", (long long)batch, (long long)ld_dense);
    cudaStream_t st = (cudaStream_t)stream;
    // The weight-expansion pass of the matmul path (tiles scattered in shared memory, stores that also write the zeros) takes
    // what its items can hold; the kernel below serves the rest.
    const size_t es0 = dtype_size(dtype);
    const int64_t tiles1 = geo.nb * geo.nc;
    const bool parts_aligned = batch == 1 || (batch_stride % 8 == 0 && tiles1 * geo.cc % 8 == 0);  // every batch entry like the first
    if (parts_aligned && tc_expand_plain_supported(geo, dtype, val, idx, dense, ld_dense)) {
        for (int64_t b = 0; b < batch; b++) {
            const char *vb = static_cast<const char *>(val) + (size_t)b * tiles1 * geo.cc * n * es0;
            if ((rc = tc_expand_plain(geo, dtype, vb, idx + b * tiles1 * geo.cc, static_cast<char *>(dense) + (size_t)b * batch_stride * es0, ld_dense, st)))
                return rc;
        }
        return NMG_OK;
    }
    PatternTable tab;
    if ((rc = get_pattern_table(n, m, &tab))) return rc;

    DensifyParams p{};
    p.val = val; p.idx = idx; p.dense = dense; p.slot_of_row = tab.slot_of_row;
    p.M = M; p.K = K; p.ld = ld_dense; p.batch_stride = batch_stride;
    p.nb = geo.nb; p.nc = geo.nc; p.tiles = batch * geo.nb * geo.nc;
    p.n = n; p.m = m; p.g = g; p.C = geo.C; p.cc = geo.cc;
    const size_t es = dtype_size(dtype);
    const size_t smem = (((size_t)geo.cc * n * es + 15) & ~(size_t)15) + (size_t)geo.cc * 2 + (size_t)geo.C * m;
    if (smem > 200 * 1024)
        NMG_FAIL(NMG_ERR_UNSUPPORTED, "tile of %d columns needs %zu bytes of shared memory (limit %d)", geo.cc, smem, 200 * 1024);
    int64_t ctas = p.tiles;
    const int64_t max_ctas = (int64_t)sm_count() * 32;
    if (ctas > max_ctas) ctas = max_ctas;
    NMG_DISPATCH_DTYPE(dtype, T, {
        NMG_ALLOW_SMEM(smem, densify_kernel<T>);
        densify_kernel<T><<<(unsigned)ctas, 128, smem, st>>>(p);
    });
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

// The same for n <= 2 and chunks of whole 16-byte pieces.  Element by element from global memory 4096 x 4096 bf16 2:4 took 29 us, now 18
// (59 MB: 9 us at the copy rate).  An item is R row-blocks x Q chunks, about 512 columns; its rows come in whole lines, and a
// thread gathers one piece of eight slots from shared memory and stores it in 16-byte pieces.  VEC: 16-byte aligned rows.
constexpr int GATHER_THREADS = 256;
struct GatherRows { int R, Q, groups, spans; };
template <typename T, int N_, bool VEC>
__global__ void __launch_bounds__(GATHER_THREADS) gather_rows_kernel(const GatherParams prm, const GatherRows it) {
    extern __shared__ __align__(16) char smem[];
    constexpr int V = 16 / (int)sizeof(T);
    const int m = prm.m, cc = prm.cc, R = it.R, Q = it.Q, cols = Q * cc, rows = R * m, tid = (int)threadIdx.x;
    T *tile = reinterpret_cast<T *>(smem);                                 // [rows][cols]
    int8_t *ord = reinterpret_cast<int8_t *>(tile + (size_t)rows * cols);  // [C][N_]
    for (int i = tid; i < prm.C * N_; i += GATHER_THREADS) ord[i] = prm.order[i];
    const int per_chunk = R * cc / 8, q = tid / per_chunk, e8 = (tid - q * per_chunk) * 8, j = e8 / cc, slot0 = e8 - j * cc;
    const bool has = tid < Q * per_chunk;
    const T *dense = static_cast<const T *>(prm.dense);
    T *val = static_cast<T *>(prm.val);
    const int64_t per_batch = (int64_t)it.groups * it.spans, items = prm.tiles / (prm.nb * prm.nc) * per_batch;
    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const int64_t b = item / per_batch;
        const int in_batch = (int)(item - b * per_batch), span = in_batch / it.groups, grp = in_batch - span * it.groups;
        const int64_t mb0 = (int64_t)grp * R, r0 = mb0 * m, c0 = (int64_t)span * cols;
        const bool mine = has && span * Q + q < prm.nc && mb0 + j < prm.nb;
        const int64_t slot = ((b * prm.nc + span * Q + q) * prm.nb + mb0 + j) * cc + slot0;
        uint4 iv = make_uint4(0, 0, 0, 0);
        if (mine) iv = __ldg(reinterpret_cast<const uint4 *>(prm.idx + slot));
        const T *src = dense + b * prm.batch_stride + r0 * prm.ld + c0;
        const int row_lim = (int)(prm.M - r0 < rows ? prm.M - r0 : rows), col_lim = (int)(prm.K - c0 < cols ? prm.K - c0 : cols);
        __syncthreads();  // the previous item has been gathered
        if constexpr (VEC) {
            const int vpl = cols / V;
            for (int i = tid; i < rows * vpl; i += GATHER_THREADS) {
                const int l = i / vpl, c = (i - l * vpl) * V;
                if (l < row_lim && c + V <= col_lim) {
                    cp_async_16(tile + i * V, src + l * prm.ld + c);
                } else {  // the weight's edge
#pragma unroll
                    for (int u = 0; u < V; u++) tile[i * V + u] = (l < row_lim && c + u < col_lim) ? __ldg(src + l * prm.ld + c + u) : DT<T>::from_f32(0.f);
                }
            }
            cp_async_commit();
            cp_async_wait<0>();
        } else {
            for (int i = tid; i < rows * cols; i += GATHER_THREADS) {
                const int l = i / cols, c = i - l * cols;
                tile[i] = (l < row_lim && c < col_lim) ? __ldg(src + l * prm.ld + c) : DT<T>::from_f32(0.f);
            }
        }
        __syncthreads();
        if (mine) {
            const int16_t *ci = reinterpret_cast<const int16_t *>(&iv);
            __align__(16) T out[8 * N_];
            const T *base = tile + j * m * cols + q * cc;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int c = ci[k];
                const int8_t *o = ord + (slot0 + k) / prm.g * N_;
#pragma unroll
                for (int t = 0; t < N_; t++) out[k * N_ + t] = (unsigned)c < (unsigned)cc ? base[(int)o[t] * cols + c] : DT<T>::from_f32(0.f);  // a malformed index reads as zero
            }
            uint4 *dst = reinterpret_cast<uint4 *>(val + slot * N_);
#pragma unroll
            for (int i = 0; i < 8 * N_ / V; i++) dst[i] = reinterpret_cast<const uint4 *>(out)[i];
        }
    }
}

extern "C" int nmg_gather(const void *dense, const int16_t *idx, int64_t batch, int64_t M, int64_t K, int64_t ld_dense,
                          int64_t batch_stride, int n, int m, int g, int dtype, void *val, void *stream) {
    Geo geo;
    int rc = make_geo(M, K, n, m, g, &geo);
    if (rc) return rc;
    if ((rc = check_dtype(dtype))) return rc;
    if (!dense || !val || !idx) NMG_FAIL(NMG_ERR_INVALID, "dense, val and idx must be non-NULL");
    if (n < 1) NMG_FAIL(NMG_ERR_INVALID, "n must be >= 1");
    if (batch < 1 || ld_dense < K || (batch > 1 && batch_stride < M * ld_dense))
        NMG_FAIL(NMG_ERR_INVALID, "bad batch / leading dimension (batch=%lld ld=%lld)", (long long)batch, (long long)ld_dense);
    PatternTable tab;
    if ((rc = get_pattern_table(n, m, &tab))) return rc;
    GatherParams p{};
    p.dense = dense; p.idx = idx; p.val = val; p.order = tab.order;
    p.M = M; p.K = K; p.ld = ld_dense; p.batch_stride = batch_stride;
    p.nb = geo.nb; p.nc = geo.nc; p.tiles = batch * geo.nb * geo.nc;
    p.n = n; p.m = m; p.g = g; p.C = geo.C; p.cc = geo.cc;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t es = dtype_size(dtype);
    GatherRows it;
    it.Q = 512 / geo.cc < 1 ? 1 : 512 / geo.cc;
    if (it.Q > geo.nc) it.Q = (int)geo.nc;
    it.R = GATHER_THREADS * 8 / (it.Q * geo.cc);
    const int fit = (int)(32 * 1024 / ((size_t)m * it.Q * geo.cc * es));
    if (it.R > fit) it.R = fit;
    if (it.R >= 1 && n <= 2 && geo.cc % 8 == 0 && ((reinterpret_cast<uintptr_t>(val) | reinterpret_cast<uintptr_t>(idx)) & 15) == 0 && geo.nb < 0x3fffffff &&
        geo.nc < 0x3fffffff) {
        it.groups = (int)((geo.nb + it.R - 1) / it.R);
        it.spans = (int)((geo.nc + it.Q - 1) / it.Q);
        const size_t smem = (size_t)it.R * m * it.Q * geo.cc * es + (size_t)geo.C * n + 16;  // at most 34 KB
        const int64_t items = batch * it.groups * it.spans, cap = (int64_t)sm_count() * 6;
        const unsigned grid = (unsigned)(items < cap ? items : cap);
        const bool vec = (ld_dense * es) % 16 == 0 && (batch == 1 || (batch_stride * es) % 16 == 0) && (reinterpret_cast<uintptr_t>(dense) & 15) == 0;
        NMG_DISPATCH_DTYPE(dtype, T, {
            if (n == 1) {
                if (vec) gather_rows_kernel<T, 1, true><<<grid, GATHER_THREADS, smem, st>>>(p, it);
                else gather_rows_kernel<T, 1, false><<<grid, GATHER_THREADS, smem, st>>>(p, it);
            } else {
                if (vec) gather_rows_kernel<T, 2, true><<<grid, GATHER_THREADS, smem, st>>>(p, it);
                else gather_rows_kernel<T, 2, false><<<grid, GATHER_THREADS, smem, st>>>(p, it);
            }
        });
        NMG_CUDA(cudaGetLastError());
        return NMG_OK;
    }
    int64_t ctas = (p.tiles + 7) / 8;
    const int64_t max_ctas = (int64_t)sm_count() * 16;
    if (ctas > max_ctas) ctas = max_ctas;
    NMG_DISPATCH_DTYPE(dtype, T, { gather_layout_kernel<T><<<(unsigned)ctas, 256, 0, st>>>(p); });
    NMG_CUDA(cudaGetLastError());
    return NMG_OK;
}

// =====================================================================================================
// Column sums (the bias gradient): out[c] = sum over rows of x[r][c], fp32 accumulation.
// HBM-bound.  A lane owns one 16-byte piece of columns, the warps of a CTA and the CTAs of a column group stride over the rows;
// partial sums meet in shared memory, then in the workspace, where a second kernel adds the row ranges in order.
// 4096 x 4096 bf16 (33.5 MB, 5.2 us at the copy rate): 12.5 + 2.8 us from HBM, torch's reduction 21.
// =====================================================================================================
constexpr int SUM_THREADS = 256;
// Sum of partial sums.  For fp32 results what each addition rounds off is summed beside it (Knuth's two-sum): those few additions
// are of the result's own size and made most of the error.  4096 rows of mean 0.3 and deviation 1: 5.6e-8 relative without,
// torch's reduction 5.2e-8.  In the lanes too it cost 14.4 us for 10.6 (4096 x 4096) and gave nothing more; those add four rows in pairs.
template <typename T> struct ColumnSum {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float v) {
        if constexpr (sizeof(T) == 4) {
            const float s = __fadd_rn(hi, v), t = __fsub_rn(s, hi);
            lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(v, t)));
            hi = s;
        } else {
            hi += v;
        }
    }
    __device__ __forceinline__ float value() const { return sizeof(T) == 4 && isfinite(hi) ? hi + lo : hi; }
};
template <typename T, int V>
__global__ void __launch_bounds__(SUM_THREADS) column_sum_kernel(const T *x, int64_t rows, int64_t cols, int64_t ld, int64_t rows_per_cta, float *partial) {
    __shared__ float red[SUM_THREADS / 32][32 * V];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int WARPS = SUM_THREADS / 32, AHEAD = 4;
    const int64_t c = ((int64_t)blockIdx.x * 32 + lane) * V, r0 = (int64_t)blockIdx.y * rows_per_cta;
    const int64_t r1 = r0 + rows_per_cta < rows ? r0 + rows_per_cta : rows;
    float acc[V];
#pragma unroll
    for (int u = 0; u < V; u++) acc[u] = 0.f;
    if (c < cols) {  // V > 1: cols is a multiple of V
        int64_t r = r0 + warp;
        for (; r + (AHEAD - 1) * WARPS < r1; r += AHEAD * WARPS) {
            __align__(16) T v[AHEAD][V];
#pragma unroll
            for (int a = 0; a < AHEAD; a++) {
                const T *src = x + (r + a * WARPS) * ld + c;
                if constexpr (V > 1) *reinterpret_cast<uint4 *>(v[a]) = __ldg(reinterpret_cast<const uint4 *>(src));
                else v[a][0] = __ldg(src);
            }
#pragma unroll
            for (int u = 0; u < V; u++)
                acc[u] += (DT<T>::to_f32(v[0][u]) + DT<T>::to_f32(v[1][u])) + (DT<T>::to_f32(v[2][u]) + DT<T>::to_f32(v[3][u]));
        }
        for (; r < r1; r += WARPS)
#pragma unroll
            for (int u = 0; u < V; u++) acc[u] += DT<T>::to_f32(__ldg(x + r * ld + c + u));
    }
#pragma unroll
    for (int u = 0; u < V; u++) red[warp][lane * V + u] = acc[u];
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = threadIdx.x; i < 32 * V; i += SUM_THREADS) {
        ColumnSum<T> sum;
#pragma unroll
        for (int w = 0; w < WARPS; w++) sum.add(red[w][i]);
        const int64_t col = (int64_t)blockIdx.x * 32 * V + i;
        if (col < cols) partial[(int64_t)blockIdx.y * cols + col] = sum.value();
    }
}
template <typename T>
__global__ void __launch_bounds__(SUM_THREADS) column_sum_finish_kernel(const float *partial, int ranges, int64_t cols, T *out) {
    __shared__ float red[SUM_THREADS / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t c = (int64_t)blockIdx.x * 32 + lane;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    ColumnSum<T> sum;
    if (c < cols) {
#pragma unroll 4
        for (int i = warp; i < ranges; i += SUM_THREADS / 32) sum.add(partial[i * cols + c]);
    }
    red[warp][lane] = sum.value();
    __syncthreads();
    if (warp != 0 || c >= cols) return;
    ColumnSum<T> all;
#pragma unroll
    for (int w = 0; w < SUM_THREADS / 32; w++) all.add(red[w][lane]);
    out[c] = DT<T>::from_f32(all.value());
}

// Row ranges: two waves of CTAs at most, at least 32 rows each
static int column_sum_ranges(int64_t rows, int64_t cols, int64_t per_cta) {
    const int64_t groups = (cols + per_cta - 1) / per_cta, want = (148 * 8 + groups - 1) / groups, most = (rows + 31) / 32;
    const int64_t r = want < most ? want : most;
    return (int)(r < 1 ? 1 : r > 256 ? 256 : r);
}

extern "C" size_t nmg_column_sum_workspace_bytes(int64_t rows, int64_t cols) {
    if (rows < 1 || cols < 1) return 0;
    return (size_t)column_sum_ranges(rows, cols, 256) * (size_t)cols * 4 + 256;  // the widest column groups have the most ranges
}

extern "C" int nmg_column_sum(const void *x, int64_t rows, int64_t cols, int64_t ld, int dtype, void *out, void *workspace, size_t workspace_bytes, void *stream) {
    int rc;
    if ((rc = check_dtype(dtype))) return rc;
    if (!x || !out) NMG_FAIL(NMG_ERR_INVALID, "x and out must be non-NULL");
    if (rows < 1 || cols < 1 || ld < cols) NMG_FAIL(NMG_ERR_INVALID, "bad shape (%lld x %lld, ld %lld)", (long long)rows, (long long)cols, (long long)ld);
    const size_t es = dtype_size(dtype);
    const int V = 16 / (int)es;
    const bool vec = cols % V == 0 && ld % V == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    const int64_t per_cta = vec ? 32 * V : 32, groups = (cols + per_cta - 1) / per_cta;
    const int ranges = column_sum_ranges(rows, cols, per_cta);
    if (!workspace || workspace_bytes < (size_t)ranges * cols * 4 + 256)
        NMG_FAIL(NMG_ERR_WORKSPACE, "workspace of %zu bytes required, got %zu", (size_t)ranges * cols * 4 + 256, workspace_bytes);
    float *partial = reinterpret_cast<float *>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    const int64_t rows_per_cta = (rows + ranges - 1) / ranges;
    cudaStream_t st = (cudaStream_t)stream;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((cols + 31) / 32));
    cfg.blockDim = dim3(SUM_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const dim3 grid((unsigned)groups, (unsigned)ranges);
    NMG_DISPATCH_DTYPE(dtype, T, {
        if (vec) column_sum_kernel<T, 16 / (int)sizeof(T)><<<grid, SUM_THREADS, 0, st>>>(static_cast<const T *>(x), rows, cols, ld, rows_per_cta, partial);
        else column_sum_kernel<T, 1><<<grid, SUM_THREADS, 0, st>>>(static_cast<const T *>(x), rows, cols, ld, rows_per_cta, partial);
        NMG_CUDA(cudaGetLastError());
        NMG_CUDA(cudaLaunchKernelEx(&cfg, column_sum_finish_kernel<T>, static_cast<const float *>(partial), ranges, cols, static_cast<T *>(out)));
    });
    return NMG_OK;
}
