// Which kernel takes the linear layers of a network in inference: by slabs (linear_batch.cu), by tiles (linear_tc.cu) or none.  Host code without CUDA.
#pragma once

namespace lineartc {

constexpr int kM = 128;                               // rows of a tile
constexpr int kSlice = 64;                            // depth of a stage
constexpr int kSlab = 192, kMostSlabDepth = 384;      // columns of W that a CTA keeps, and how deep they may be
constexpr int kMostSlabColumns = 1536;
constexpr int kTile = 256, kMostTileDepth = 1024;     // columns of a tile
constexpr long long kMostRows = 1LL << 24;            // tiles are counted in 32 bits

enum class Route { none, slabs, tiles };

inline bool slab_shape(long long rows, int K, int N) {
    return rows > 0 && rows <= kMostRows && K > 0 && K % kSlice == 0 && K <= kMostSlabDepth && N > 0 && N % kSlab == 0 && N <= kMostSlabColumns;
}
inline bool tile_shape(long long rows, int K, int N) {
    return rows > 0 && rows <= kMostRows && K > 0 && K % kSlice == 0 && K <= kMostTileDepth && N > 0 && N % kTile == 0 &&
           (rows + kM - 1) / kM * (N / kTile) <= (1LL << 28);
}
// sms: of the device, 0 where it cannot run the kernels.  A CTA holds one slab, and those of one row of tiles run together.
inline Route batch_route(int count, long long rows, int K, int N, int slab_sms, int tile_sms) {
    if (slab_shape(rows, K, N) && slab_sms >= N / kSlab * count) return Route::slabs;
    return tile_shape(rows, K, N) && tile_sms > 0 ? Route::tiles : Route::none;
}

// Whether a batch takes less of the GPU's time than the library's products, one by one, between the kernels of a network (behind a token shift and in
// front of a gate, captured; the library's chain over the one launch's).  By slabs three layers 1.40 at 12544 x 192, 1.13 at 100352, 1.00 at
// 200704; 1.17 at 50176 x 384, 1.04 at 200704; four a little more.  By tiles up to 512 deep 1.03 and more at every size tried (1.09 where a second or third
// round of tiles is all but empty).  Deeper, such a round costs what the launches save: second round filled to 0.05 / 0.09 / 0.14 / 0.16, 1024 deep 0.97 at
// 0.05 and 1.06 at 0.14, 768 deep 1.00 at 0.09 and 1.18 at 0.16; third round 0.98 at 0.11, 1.09 at 0.27.  And in many rounds the library's tiles, two
// SMs to one, are the faster: 768 deep 1.01 at 32 rounds, 0.99 at 48, 0.98 at 64, 1024 deep 1.00 at 42.
inline bool batch_pays(int count, long long rows, int K, int N, int slab_sms, int tile_sms) {
    const Route by = count >= 3 ? batch_route(count, rows, K, N, slab_sms, tile_sms) : Route::none;
    if (by != Route::tiles || K <= 512) return by != Route::none;
    const long long tiles = (rows + kM - 1) / kM * (N / kTile) * count, rounds = (tiles + tile_sms - 1) / tile_sms, last = tiles - (rounds - 1) * tile_sms;
    return rounds <= 40 && !((rounds == 2 || rounds == 3) && 8 * last < tile_sms);
}
// The key layer with its squared ReLU, which the tiles take in any depth.  By tiles / by slabs, us: 192 deep 12544 rows 9.6 / 9.8, 50176 28.5 / 25.0,
// 100352 51.9 / 42.2, 200704 99.2 / 78.4; 384 deep 12544 rows 17.8 / 19.6, 50176 60.6 / 60.4, 100352 120.7 / 116.3.
inline bool square_by_slabs(long long rows, int K, int N, int slab_sms) { return K <= 256 && slab_shape(rows, K, N) && slab_sms >= N / kSlab; }

}  // namespace lineartc
