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

// The key layer with its squared ReLU, which the tiles take in any depth.  By tiles / by slabs, us: 192 deep 12544 rows 9.6 / 9.8, 50176 28.5 / 25.0,
// 100352 51.9 / 42.2, 200704 99.2 / 78.4; 384 deep 12544 rows 17.8 / 19.6, 50176 60.6 / 60.4, 100352 120.7 / 116.3.
inline bool square_by_slabs(long long rows, int K, int N, int slab_sms) { return K <= 256 && slab_shape(rows, K, N) && slab_sms >= N / kSlab; }

}  // namespace lineartc
