// One-pass partition chase: the Thomas solves along x of W neighbouring wavenumbers by one CTA that holds all
// their rows in registers, so that a field is read once and written once.
//
// Rows are cut into P chunks, the first e of R rows and the others of R - 1 (any nx up to 4096 but 2 and 5 divides so,
// tile_rows); thread (p, w) = (threadIdx.x / W, threadIdx.x % W) owns chunk p of wavenumber j = tile W + w. The last row
// of a chunk is its separator B_p; the rows before it satisfy  x_int = z_p - B_{p-1} g - B_p h,  z_p = T^-1 f_int,
// g = T^-1 e_first, h = T^-1 e_last, and the separators a tridiagonal system of size P whose Thomas factors
// depend on the wavenumber only and are tabulated:
//   -g_last B_{p-1} + (d - h_last - g'_first) B_p - h'_first B_{p+1} = f_sep - z_last - z'_first
// (primes: the next chunk). With Q_r = (-c_0) .. (-c_{r-1}), a pass is: the forward elimination
// y_r = (f_r - y_{r-1}) c_r of every chunk, whose values stay in registers, with z_first = sum Q_r y_r beside it; the
// separator system as two affine scans along p (shuffles inside a warp, the warps' compositions through shared
// memory); the back substitution x_r = y_r - c_r (x_{r+1} + Q_r B_{p-1}) from x = B_p. The pairs (c_r, Q_r) come from
// shared memory, one 16-byte read per row and sweep: with the factors read by four sweeps the kernel waited for
// shared memory (2048 x 2048: 27.5 -> 23.7 us with the pairs).
// Periodic x: the last row is a cut, beta = x_{nx-1}. The other separators are solved for beta = 0, the wrapped
// row gives beta, and their response v to beta = 1 (tabulated) is added.
// The result equals the sequential Thomas solve (chasing_method_base.cpp:24-52) and, for periodic x, the
// Sherman-Morrison solve (:178-197) up to round-off.
//
// What bounds it: one read and one write of the field (L2 or HBM); 2048 x 2048 in 21.7 us, 3.1 TB/s (the three-pass
// form: 48 us), 256 x 65536 in 81 us, 3.3 TB/s, 1000 x 1500 in 8.6 us (sequential sweep: 764 us); the load, compute
// and store phases of the few tiles an SM holds overlap little. At R = 16 the kernel stays at 64 registers, so that an
// SM holds 1024 threads of tiles, and the dependent chains at 15 steps. Only the last interior row of a chunk is
// conditional: with a bound on every row the selects took 5/6 of the instructions.
#pragma once

#include "fp_common.cuh"

#include <climits>

namespace fpb
{

constexpr int kTileThreads = 1024;  // largest CTA: kTileThreads / 4 chunks
constexpr int kTileMaxRows = kTileThreads / 4 * 16;

// Rows of the longer chunks for nx rows, whose chunks of R and R - 1 rows must add up to nx; 0 where none does (nx = 2
// and 5) or nx is beyond one CTA. 16 above 512 rows; 8 below, where a field gives few tiles and the pass is a chain of
// latencies. us at (R, W) = (8, 8) / (16, 4) / (16, 8), graph replays: 128 x 128 2.7 / 3.7 / 3.5, 512 x 512 4.2 / 3.8 /
// 4.2, 1024 x 512 7.4 / 4.7 / 6.1, 2048 x 512 - / 7.2 / 11; with more tiles (16, 8) is the better one from 192 to 1024
// rows, which the rule does not use: 384 x 8192 14.7 / 13.9 / 11.3, 512 x 8192 18.8 / 18.1 / 14.3, 1024 x 2048 14 / 11 / 9.
inline int tile_rows(int nx)
{
    if (nx > kTileMaxRows) return 0;
    for (int R : {16, 8, 4})
        if ((R < 16 || nx > 512) && (nx + R - 1) / R * (R - 1) <= nx) return R;
    return 0;
}

// Columns (fields x wavenumbers) up to which the one-pass kernel is the faster one on short columns. Most of a tile's
// lanes are idle there (nx = 8 is one chunk: 8 threads of a warp), which many columns pay for, while one thread per
// column (k_chase) is a chain of 2 nx steps that hides behind other columns; with periodic x it reads two more tables.
// us, sequential / one-pass, DD: 64 columns nx 3 2.2 / 2.5, 8 3.4 / 3.0, 16 5.3 / 3.3; 32768 columns 8 3.7 / 5.7, 16 5.7 /
// 5.9, 24 7.8 / 5.7; 262144 columns 8 9 / 23, 16 16 / 24, 24 24 / 25, 32 32 / 28; 127000 columns 33 16 / 24, 40 17 / 19.
inline long long tile_columns(int nx, bool periodic)
{
    struct Line
    {
        int       last;
        long long open, per;
    };
    constexpr long long never = LLONG_MAX;
    static const Line lines[] = {{4, 0, 24576},         {8, 8192, 32768},       {13, 24576, 65536},   {16, 32768, 196608},
                                 {20, 49152, 98304},    {24, 131072, never},    {27, 98304, never},   {32, never, never},
                                 {34, 65536, 98304},    {41, 98304, never}};
    for (const Line& l : lines)
        if (nx <= l.last) return periodic ? l.per : l.open;
    return never;
}

// The systems of one field: chunk layout and tables (chase_tile_tables builds them).
struct ChaseTileTab
{
    int           nx, ny;      // rows; wavenumbers of a row
    int           R, P, e;     // rows of a long chunk; chunks; the leading ones that are long
    int           end_neu;     // x+ Neumann: the last row's diagonal is d + 1
    int           per;         // periodic x
    int           types;       // 2: the first chunk has its own factors (x- Neumann)
    const double2* cq;         // [types][R - 1][ny] (c_r, Q_r): the other chunks, then the first one's
    const double* ends;        // [3][4][ny] g_first, g_last, h_first, h_last: chunk 0, other long ones, short ones
    const double* d;           // [ny] diagonals
    const double* cp;          // [P][ny] separator Thomas factors; the last row is formed in the kernel
    const double* iden;        // [P][ny] 1 / denominators
    const double* v;           // periodic: [P][ny] separators' response to beta = 1
    const double* ib;          // periodic: [ny] 1 / the wrapped row's denominator
};

// Shared memory (doubles) of a CTA of n threads with tiles of W wavenumbers.
__host__ __device__ __forceinline__ int chase_tile_smem(int n, int W, int R)
{
    return 4 * (R - 1) * W + 2 * n + 4 * (n / 32) * W + W;
}

// Inclusive affine scan over the chunks a warp holds (lane stride W), then over the CTA's warps: (a, b) of the
// thread's own map becomes the value of the composition of every map before and including it, applied to 0.
// REV: from the last chunk down. tw: the warps' compositions, nw x W. Contains one barrier.
template <int W, bool REV>
__device__ __forceinline__ double tile_scan(double a, double b, double2* tw)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5, w = lane % W;
#pragma unroll
    for (int o = W; o < 32; o <<= 1)
    {
        const double pa = REV ? __shfl_down_sync(0xffffffffu, a, o) : __shfl_up_sync(0xffffffffu, a, o);
        const double pb = REV ? __shfl_down_sync(0xffffffffu, b, o) : __shfl_up_sync(0xffffffffu, b, o);
        if (REV ? lane + o < 32 : lane >= o)
        {
            b = fma(a, pb, b);
            a *= pa;
        }
    }
    if (REV ? lane < W : lane >= 32 - W)
        tw[wid * W + w] = make_double2(a, b);
    __syncthreads();
    double y = 0;
#pragma unroll 4
    for (int k = 0; k < (REV ? nw - 1 - wid : wid); ++k)
    {
        const double2 m = tw[(REV ? nw - 1 - k : k) * W + w];
        y               = fma(m.x, y, m.y);
    }
    return fma(a, y, b);
}

// One tile. IO: in(i, j) the address of a right-hand side (rows ny apart); stage() loads what mods() needs into shared
// memory (a barrier follows); mods(y, fsep, lng, i0, li, j) turns the thread's values (interior rows i0 + r, separator
// row i0 + li) into right-hand sides; store() says whether the solution is written, to out(i, j), or handed to
// take(y, x, lng, p, i0, li, j, on) by all threads of a warp together (interior rows and separator, `on` where valid).
// skip: wavenumbers from ny - skip on are left alone. The tile's wavenumbers are tile W .. tile W + W - 1; blockDim.x a
// multiple of 32 of at least P W.
template <int W, int R, typename IO>
__device__ __forceinline__ void chase_tile(const ChaseTileTab& t, int tile, int skip, const IO& io, double* sm)
{
    constexpr int Ri  = R - 1;
    const int     n   = blockDim.x, tid = threadIdx.x;
    const int     w   = tid % W, p = tid / W, P = t.P, ny = t.ny;
    const int     j0  = tile * W + w;
    const bool    act = p < P && j0 < ny - skip;
    const int     j   = min(j0, ny - 1);  // idle lanes read their own tile's last column (another's is being stored)
    double2*      cs  = reinterpret_cast<double2*>(sm);  // [2][Ri][W]
    double2*      tw  = cs + 2 * Ri * W;                 // warps' compositions, forward and backward
    double2*      tw2 = tw + (n / 32) * W;
    double*       zf  = reinterpret_cast<double*>(tw2 + (n / 32) * W);  // [n] first interior values; later the separators
    double*       xs  = zf + n;                                         // [n]
    double*       sb  = xs + n;                                         // [W] beta
    const int     pc  = p < P ? p : P - 1;
    const int     i0  = pc * (R - 1) + min(pc, t.e);
    const bool    lng = pc < t.e;
    const int     li  = lng ? Ri : Ri - 1;  // interior rows; idle threads repeat the last chunk

    double y[Ri];
    auto   pin = io.in(i0, j);
#pragma unroll
    for (int r = 0; r < Ri; ++r, pin += ny) y[r] = r < Ri - 1 || lng ? (double)*pin : 0.0;
    double fsep = (double)*io.in(i0 + li, j);
    io.stage();
#pragma unroll 2
    for (int k = tid; k < t.types * Ri * W; k += n)
        cs[k] = __ldg(t.cq + (long long)(k / W) * ny + min(tile * W + k % W, ny - 1));
    // separator row of chunk p (the factors of the last row depend on its being last)
    double        inv = 0, cpv = 0, gl = 0;
    const double* en  = t.ends + (long long)(p == 0 ? 0 : p < t.e ? 1 : 2) * 4 * ny + j;
    if (p < P)
    {
        gl = __ldg(en + ny);
        if (p < P - 1)
        {
            inv = __ldg(t.iden + (long long)p * ny + j);
            cpv = __ldg(t.cp + (long long)p * ny + j);
        }
        else if (!t.per)
        {
            const double diag = (t.end_neu ? __ldg(t.d + j) + 1.0 : __ldg(t.d + j)) - __ldg(en + 3 * (long long)ny);
            inv = 1.0 / (p > 0 ? fma(gl, __ldg(t.cp + (long long)(p - 1) * ny + j), diag) : diag);
        }
    }
    __syncthreads();

    io.mods(y, fsep, lng, i0, li, j);
    const double2* c  = cs + (p == 0 && t.types > 1 ? Ri * W : 0) + w;
    double         zl = 0, z = 0;
#pragma unroll
    for (int r = 0; r < Ri; ++r)
        if (r < Ri - 1 || lng)
        {
            const double2 m = c[r * W];
            zl              = (y[r] - zl) * m.x;
            y[r]            = zl;
            z               = fma(m.y, zl, z);
        }
    zf[tid] = z;
    __syncthreads();

    const bool   sep = p < P - (t.per ? 1 : 0);  // rows of the separator system (the periodic cut is none of them)
    double       rhs = fsep - zl;
    if (p < P - 1) rhs -= zf[tid + W];
    double x = tile_scan<W, false>(sep ? (p > 0 ? gl * inv : 0.0) : 1.0, sep ? rhs * inv : 0.0, tw);
    x        = tile_scan<W, true>(sep ? -cpv : 1.0, sep ? x : 0.0, tw2);
    double bl;
    if (t.per)
    {
        xs[tid] = x;
        __syncthreads();
        if (p == P - 1)
        {
            double num = fsep - zl - zf[w];
            if (P > 1) num += gl * xs[tid - W] + __ldg(t.ends + 2 * (long long)ny + j) * xs[w];
            sb[w] = num * __ldg(t.ib + j);
        }
        __syncthreads();
        const double beta = sb[w];
        x                 = p < P - 1 ? fma(__ldg(t.v + (long long)p * ny + j), beta, x) : beta;
        zf[tid]           = x;
        __syncthreads();
        bl = p > 0 ? zf[tid - W] : beta;
    }
    else
    {
        xs[tid] = x;
        __syncthreads();
        bl = p > 0 ? xs[tid - W] : 0.0;
    }

    if (io.store())
    {
        if (act) *io.out(i0 + li, j) = x;
        auto po = io.out(i0 + Ri - 1, j);
#pragma unroll
        for (int r = Ri - 1; r >= 0; --r, po -= ny)
            if (r < Ri - 1 || lng)
            {
                const double2 m = c[r * W];
                x               = fma(-m.x, fma(m.y, bl, x), y[r]);
                if (act) *po = x;
            }
        return;
    }
    const double xsep = x;
#pragma unroll
    for (int r = Ri - 1; r >= 0; --r)
        if (r < Ri - 1 || lng)
        {
            const double2 m = c[r * W];
            y[r] = x = fma(-m.x, fma(m.y, bl, x), y[r]);
        }
    io.take(y, xsep, lng, p, i0, li, j, act);
}

// `batch` fields of t.nx x t.ny values back to back, solved in place; wavenumbers from ny - skip on are left alone.
void launch_chase_tile(double* f, long long batch, int skip, const ChaseTileTab& t, cudaStream_t s);

}  // namespace fpb
