// Widths of the output tiles of the two-pass product.  Plain C++ but for the accessors.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define NMG_BOTH __host__ __device__
#else
#define NMG_BOTH
#endif

namespace nmg {

constexpr int TILE_COLS = 256;  // columns of the widest tile

// The output's tiles: the first f_wide rows of tiles are bn columns wide, the f_narrow rows below them bn_tail.
struct GemmTiles {
    int f_wide, f_narrow;    // rows of tiles
    int t_wide, t_narrow;    // tiles per row
    int bn, bn_tail;         // columns of a tile
    NMG_BOTH int wide() const { return f_wide * t_wide; }
    NMG_BOTH int count() const { return f_wide * t_wide + f_narrow * t_narrow; }
};

// The choice whose slowest pair costs least.  A tile of bn columns costs what bn + 40 columns at full rate do (narrow
// tiles read more shared memory per product; fp32, 3072 <- 768, 4096 tokens: 28.6 us per wave at 256, 15.8 at 128, 10.8 at 64).
// Tiles of one width leave most pairs without work in a last wave that is not full, so some rows of tiles at the end of the
// order may be narrower: their tiles then fill the places that the wide ones leave.  Tile i goes to pair i % units.
// 4096 x 4096 bf16, 4096 tokens: 256 tiles, 3.46 waves of 74 pairs, 110.0 -> 106.7 us with three of sixteen rows in tiles of 192;
// 4096 x 1024 f16 pair, 12288 tokens: 212.0 -> 208.2.  From sixteen waves on the last one is too small a part.
// 16-bit: wide tiles have 256 columns, narrow ones 128 or 192 (whole staged groups for both halves of the drain warps).
//
// It runs on every call: no divisions inside, and no width that takes as many tiles per row as a narrower one.  Host time, fp32: 40000
// rows by 128 columns 11 -> 0.3 us, 4096 by 768 1.3 -> 0.8, at most 1.3.
inline GemmTiles gemm_tiles(int64_t tiles_f, int64_t cols, int64_t units, bool fp32, bool pair) {
    GemmTiles best{(int)tiles_f, 0, (int)((cols + TILE_COLS - 1) / TILE_COLS), 0, TILE_COLS, TILE_COLS};
    if (!pair) return best;
    const int step = fp32 ? 32 : 64, least = fp32 ? 64 : 128, widths = (TILE_COLS - least) / step + 1;
    int per_row[7];  // tiles per row at width least + i * step
    for (int i = 0; i < widths; i++) per_row[i] = (int)((cols + least + i * step - 1) / (least + i * step));
    auto wasteful = [&](int i) { return i > 0 && per_row[i] == per_row[i - 1]; };
    const int u = (int)units;
    int64_t best_cost = INT64_MAX;
    for (int i = widths - 1; i >= (fp32 ? 0 : widths - 1); i--) {
        if (fp32 && wasteful(i)) continue;
        const int bn = least + i * step, cost = bn + 40;
        const int64_t all = tiles_f * per_row[i], uniform = (all + u - 1) / u * cost;
        if (uniform < best_cost) {
            best = GemmTiles{(int)tiles_f, 0, per_row[i], 0, bn, bn};
            best_cost = uniform;
        }
        if (all > 16 * units) continue;  // a sixteenth of the last wave at most: not worth a second shape of tiles
        const int waves_row = per_row[i] / u, rest_row = per_row[i] - waves_row * u;
        for (int j = i - 1; j >= 0; j--) {
            if (wasteful(j)) continue;
            const int bn_tail = least + j * step, cost_tail = bn_tail + 40;
            int full = (int)(all / u), rest = (int)(all - (int64_t)full * u), tail = 0;  // waves of wide tiles, what is left of them, narrow tiles
            // more narrow tiles than two waves of them never help: a wide tile does the same columns in less time
            for (int f = 1; f < tiles_f && tail + per_row[j] <= 2 * u; f++) {
                tail += per_row[j];
                full -= waves_row;
                if ((rest -= rest_row) < 0) { rest += u; full--; }
                int64_t c = (int64_t)full * cost + (tail <= u ? 1 : 2) * cost_tail;  // a pair without a tile of the last wide wave
                if (rest > 0) {
                    const int over = tail - (u - rest);                               // narrow tiles left for the pairs with one
                    const int64_t with = (int64_t)(full + 1) * cost + (over <= 0 ? 0 : over <= u ? 1 : 2) * cost_tail;
                    if (with > c) c = with;
                }
                if (c < best_cost) {
                    best = GemmTiles{(int)tiles_f - f, f, per_row[i], per_row[j], bn, bn_tail};
                    best_cost = c;
                }
            }
        }
    }
    return best;
}

}  // namespace nmg
