// The one-pass chase (fp_chase_tile.cuh) over fields of one shape.
#include "fp_chase_tile.cuh"
#include "fp_internal.h"

#include <climits>

namespace fpb
{
namespace
{
// Fields of one shape back to back, in place.
struct TileFieldIO
{
    double*   f;
    long long ny;
    __device__ __forceinline__ const double* in(int i, int j) const { return f + i * ny + j; }
    __device__ __forceinline__ double*       out(int i, int j) const { return f + i * ny + j; }
    __device__ __forceinline__ static constexpr bool store() { return true; }
    __device__ __forceinline__ void stage() const {}
    template <int Ri> __device__ __forceinline__ void mods(double (&)[Ri], double&, bool, int, int, int) const {}
    template <int Ri>
    __device__ __forceinline__ void take(double (&)[Ri], double, bool, int, int, int, int, bool) const {}
};
template <int W, int R>
__global__ void __launch_bounds__(kTileThreads, 1) k_chase_tile(double* __restrict__ f, int tiles, int skip,
                                                                const __grid_constant__ ChaseTileTab t)
{
    extern __shared__ double fp_tile_smem[];
    const long long b = blockIdx.x / tiles;
    const TileFieldIO io{f + b * (long long)t.nx * t.ny, t.ny};
    chase_tile<W, R>(t, (int)(blockIdx.x - b * tiles), skip, io, fp_tile_smem);
}

template <int W, int R> void launch(double* f, long long batch, int skip, const ChaseTileTab& t, cudaStream_t s)
{
    const int       threads = (t.P * W + 31) / 32 * 32;
    const int       tiles   = (t.ny + W - 1) / W;
    const long long grid    = batch * tiles;
    if (grid > (long long)INT_MAX) throw Error(3, "more than 2^31 tiles in one chase");
    k_chase_tile<W, R>
        <<<(unsigned)grid, threads, chase_tile_smem(threads, W, R) * sizeof(double), s>>>(f, tiles, skip, t);
    FPB_CHECK_LAUNCH();
}

}  // namespace

// Tile width: 8 wavenumbers (64-byte row pieces) with 8-row chunks, 4 (32 bytes, one sector) with 16-row ones, whose CTA
// is then 512 threads of 64 registers at 2048 rows, so that two tiles share an SM. us at W = 4 / 8 / 16: 8-row chunks 256 x
// 256 3.0 / 3.1 / 4.0, 256 x 8192 10.1 / 8.4 / 9.7; 16-row chunks 1000 x 1000 6.7 / 6.3 / 10, 1280 x 1280 11.1 / 13.4,
// 1536 x 1536 13.9 / 15.8, 2048 x 2048 21.6 / 21.1, 2048 x 512 7.2 / 11.
void launch_chase_tile(double* f, long long batch, int skip, const ChaseTileTab& t, cudaStream_t s)
{
    switch (t.R)
    {
        case 16: launch<4, 16>(f, batch, skip, t, s); break;
        case 8: launch<8, 8>(f, batch, skip, t, s); break;
        default: launch<8, 4>(f, batch, skip, t, s); break;
    }
}
}  // namespace fpb
