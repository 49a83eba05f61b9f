#include "linear_routes.h"

extern "C" int batch_route(int count, long long rows, int K, int N, int slab_sms, int tile_sms) {
    return static_cast<int>(lineartc::batch_route(count, rows, K, N, slab_sms, tile_sms));
}
extern "C" int batch_pays(int count, long long rows, int K, int N, int slab_sms, int tile_sms) {
    return lineartc::batch_pays(count, rows, K, N, slab_sms, tile_sms) ? 1 : 0;
}
extern "C" int square_by_slabs(long long rows, int K, int N, int slab_sms) { return lineartc::square_by_slabs(rows, K, N, slab_sms) ? 1 : 0; }
