// y-transforms of short rows as products with the transform's matrix on the FP64 tensor instruction
// (mma.sync.m8n8k4.f64). The matrices are those of PoissonFFT2D_* (pe/poisson/poisson_fft2d.cpp:19-465),
// tabulated on the device from exactly reduced angles; families with a reflection symmetry fold a row into its
// even and odd parts first, which halves the operations:
//   DD, NN forward   e_t = x_t + x_{n-1-t}, o_t = x_t - x_{n-1-t}; the even (odd) part gives every other mode
//   NN inverse       the even and odd modes separately give C and S; x_i = C_i + S_i, x_{n-1-i} = C_i - S_i
//   PP               cosine part from the even, sine part from the odd half of the row about its last point; the
//                    two outputs of a frequency are s1 (ta S + tb C)  (and the transpose for the inverse)
//   ND, DN           no reflection symmetry: the full matrix, its columns in two halves
// So a row needs n^2 (ND, DN: 2 n^2) operations, the fast transform of the awkward lengths of these families
// (n + 1, 2 n + 1) several hundred n: dense_rule says where the product is the faster one.
//
// A CTA takes BM rows whole into shared memory (folded), so that rows may be transformed in place, then runs over
// column tiles, streaming the table through a cp.async ring while eight warps accumulate in registers.
// A few rows give few CTAs: there a cluster shares a row tile, each CTA loading it and taking every CS-th column
// tile, with a cluster barrier between the loads and the first store.
// Rows need not be contiguous: element t of row r sits at r rs + t ts, so the middle axis of a 3D field is
// transformed where it lies (rs = 1, ts = nz).
//
// What bounds it: the FP64 tensor rate (37 TFLOP/s on 148 SMs at 1.965 GHz, the rate of the scalar FP64 pipe; the
// instruction's gain is 1/8 of the issue slots and operand reads). Measured on 16384 rows of 256 (DD): 63 us, 17
// TFLOP/s, 40 % of the pipe. At 4.2 M cells the time is about 15 us, the rows' loads and stores, which overlap little
// with the products, plus 0.19 us per cell of row length, 60 % of the pipe in the product loop (a third table stage, a
// deeper ring of half the size and a start of half the CTAs half a tile later all changed less than 3 %).
#pragma once

#include "fp_common.cuh"

namespace fpb
{

struct DenseTab  // one direction of one plan
{
    int           n, K, C;    // row length; folded inputs; columns of each of the two products
    int           ldb;        // row stride of the tables
    const double *te, *to;    // [K rounded to 16][ldb], zero beyond K x C
    const double *ta, *tb;    // PP: the family's cos / sin pairs
    double        s1;         // PP
};

struct DenseSeg  // slabs x rows rows of one length
{
    const void* in;
    void*       out;
    long long   slab;     // elements between slabs
    int         rows;     // rows of a slab
    int         slabs;
    int         rs, ts;   // element t of row r: r rs + t ts
    int         plan;     // its table is entry 2 plan of the launch's array
};

enum DenseOut
{
    DENSE_F64 = 0,
    DENSE_F32 = 1,
    DENSE_ACC = 2  // FP64 out += result
};

constexpr int kDenseBK = 16;
// Table stages in the ring: narrow column tiles multiply for less time than a fetch takes and keep more in flight in
// the same memory.
__host__ __device__ constexpr int dense_stages(int bn) { return bn <= 32 ? 4 : bn <= 48 ? 3 : 2; }

__host__ __device__ constexpr bool dense_fold(int kind) { return kind == 0 || kind == 1 || kind == 4; }
__host__ __device__ __forceinline__ int dense_lda(int K) { return (K + 15) / 16 * 16 + 4; }
// Shared memory (doubles) of a CTA with row tiles of bm rows and column tiles of bn.
__host__ __device__ __forceinline__ int dense_smem(bool fold, int K, int bm, int bn)
{
    return (fold ? 2 : 1) * bm * dense_lda(K) + dense_stages(bn) * 2 * kDenseBK * (bn + 4);
}

__device__ __forceinline__ void dense_mma(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ void dense_cp16(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ int nn_slot(int m, int n) { return m ? n - 1 - m : n - 1; }  // the reference's mode order

// The folded input pair t < K of a row; x(i) reads element i.
template <int KIND, int INV, typename X>
__device__ __forceinline__ void dense_in(const DenseTab& T, int t, const X& x, double& e, double& o)
{
    const int n = T.n;
    if (KIND == 0 || (KIND == 1 && !INV))
    {
        const double u = x(t), v = x(n - 1 - t);
        const bool   mid = 2 * t == n - 1;
        e                = mid ? u : u + v;
        o                = mid ? 0.0 : u - v;
    }
    else if (KIND == 1)
    {
        e = x(nn_slot(2 * t, n));
        o = 2 * t + 1 < n ? x(nn_slot(2 * t + 1, n)) : 0.0;
    }
    else if (KIND == 4 && !INV)
    {
        const int h = n / 2;
        const double u = x(t ? t - 1 : n - 1), v = (t == 0 || t == h) ? 0.0 : x(n - t - 1);
        e = u + v;
        o = (t == 0 || t == h) ? 0.0 : u - v;
    }
    else if (KIND == 4)
    {
        const int    h = n / 2, ja = 2 * t - 1, jb = 2 * t;
        const double a = t ? x(ja) : 0.0, b = t < h ? x(jb) : 0.0;
        e = T.s1 * ((t ? T.tb[ja] * a : 0.0) + (t < h ? T.tb[jb] * b : 0.0));
        o = T.s1 * ((t ? T.ta[ja] * a : 0.0) + (t < h ? T.ta[jb] * b : 0.0));
    }
    else
    {
        e = x(t);
        o = 0;
    }
}

// The outputs of two neighbouring columns c, c + 1 (c even) of both products; put(i, v) takes element i, put2(i, u, v)
// elements i and i + 1.
template <int KIND, int INV, typename P, typename P2>
__device__ __forceinline__ void dense_out(const DenseTab& T, int c, const double (&e)[2], const double (&o)[2],
                                          const P& put, const P2& put2)
{
    const int n = T.n;
    if (KIND == 0)
    {
#pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            const int i = 2 * (c + q);
            if (i + 1 < n) put2(i, e[q], o[q]);
            else if (i < n) put(i, e[q]);
        }
        return;
    }
    if (KIND == 2 || KIND == 3)
    {
        if (c + 1 < T.C) put2(c, e[0], e[1]);
        else if (c < T.C) put(c, e[0]);
        if (c + 1 + T.C < n) put2(c + T.C, o[0], o[1]);
        else if (c + T.C < n) put(c + T.C, o[0]);
        return;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
    {
        const int i = c + q;
        if (i >= T.C) continue;
        if (KIND == 1 && !INV)
        {
            put(nn_slot(2 * i, n), e[q]);
            if (2 * i + 1 < n) put(nn_slot(2 * i + 1, n), o[q]);
        }
        else if (KIND == 1)
        {
            put(i, e[q] + o[q]);
            if (n - 1 - i != i) put(n - 1 - i, e[q] - o[q]);
        }
        else if (!INV)
        {
            const int h = n / 2;
            if (i > 0) put(2 * i - 1, T.s1 * (T.ta[2 * i - 1] * o[q] + T.tb[2 * i - 1] * e[q]));
            if (i < h) put(2 * i, T.s1 * (T.ta[2 * i] * o[q] + T.tb[2 * i] * e[q]));
        }
        else
        {
            const int h = n / 2;
            if (i == 0) put(n - 1, e[q]);
            else if (i == h) put(h - 1, e[q]);
            else
            {
                put(i - 1, e[q] + o[q]);
                put(n - i - 1, e[q] - o[q]);
            }
        }
    }
}

// Work item = one row tile of one segment (segs == nullptr: `one`, with table `tv`; else a work list of segments whose
// plans are entries of `tabs`); blockIdx.x = item * CS + rank, CS the cluster size.
template <int KIND, int INV, int TM, int TN, int WM, int WN>
__global__ void __launch_bounds__(WM* WN * 32, 2)
    k_dense(const DenseSeg* __restrict__ segs, const long long* __restrict__ prefix, int nseg,
            const DenseTab* __restrict__ tabs, const DenseSeg one, const __grid_constant__ DenseTab tv, int in32,
            int omode, int CS)
{
    constexpr int  BM = TM * WM * 8, BN = TN * WN * 8, NT = WM * WN * 32, NS = dense_stages(TN * WN * 8), BK = kDenseBK;
    constexpr bool kFold = dense_fold(KIND);
    extern __shared__ __align__(16) double fp_dense_sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wn = warp / WM;

    const long long item = blockIdx.x / CS;
    const int       rank = (int)(blockIdx.x - item * CS);
    int             s    = 0;
    if (segs)
    {
        int lo = 0, hi = nseg - 1;
        while (lo < hi)
        {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(prefix + mid) <= item) lo = mid;
            else hi = mid - 1;
        }
        s = lo;
    }
    const DenseSeg  sg    = segs ? segs[s] : one;
    const DenseTab  T     = segs ? tabs[2 * sg.plan] : tv;
    const long long local = segs ? item - prefix[s] : item;
    const int       per   = (sg.rows + BM - 1) / BM;  // row tiles of a slab
    const int       slab  = (int)(local / per);
    const int       r0    = (int)(local - (long long)slab * per) * BM;
    const int       rows  = min(BM, sg.rows - r0);
    const long long base  = slab * sg.slab + (long long)r0 * sg.rs;
    const int       K = T.K, lda = dense_lda(K), nk = (K + BK - 1) / BK;
    double*         As = fp_dense_sm;
    double*         Bs = As + (kFold ? 2 : 1) * BM * lda;

    const int nct   = (T.C + BN - 1) / BN;
    const int mine  = rank < nct ? (nct - 1 - rank) / CS + 1 : 0;  // column tiles rank, rank + CS, ...
    const int iters = mine * nk;
    // table pieces of 16 bytes: two products x BK rows x BN / 2; the next fetch takes rows fk of column tile fc
    int  fk = 0, fc = rank;
    auto fetch = [&](int stage) {
        double* const b = Bs + stage * 2 * BK * (BN + 4);
        const long long o = (long long)fk * T.ldb + fc * BN;
#pragma unroll
        for (int q0 = 0; q0 < BK * BN; q0 += NT)
        {
            const int q = q0 + tid;
            if (BK * BN % NT != 0 && q >= BK * BN) break;
            const int par = q / (BK * BN / 2), z = q % (BK * BN / 2), kk = z / (BN / 2), cc = (z % (BN / 2)) * 2;
            dense_cp16(b + (par * BK + kk) * (BN + 4) + cc, (par ? T.to : T.te) + o + kk * T.ldb + cc);
        }
        fk += BK;
        if (fk >= nk * BK)
        {
            fk = 0;
            fc += CS;
        }
    };
#pragma unroll
    for (int i = 0; i < NS - 1; ++i)
    {
        if (i < iters) fetch(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // rows into shared memory, folded; zero beyond the rows and columns there are
    // kU pairs per thread are loaded before the first is stored (a load through a generic pointer cannot pass a store to
    // shared memory by itself)
    constexpr int kU = 8, NW = NT / 32;
    const int     Kp = nk * BK;
    auto          fill_rows = [&](auto* x0) {  // unit stride: lanes along the row
        const int st = (Kp + 31) / 32, items = BM / NW * st;
        int       r = warp, t = lane;
        for (int q0 = 0; q0 < items; q0 += kU)
        {
            double e[kU], o[kU];
            int    z[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                const auto* x  = x0 + (long long)r * sg.rs;
                const bool  in = r < BM && t < Kp;
                z[u]           = in ? r * lda + t : -1;
                e[u] = o[u] = 0;
                if (r < rows && t < K) dense_in<KIND, INV>(T, t, [=](int i) { return (double)x[i]; }, e[u], o[u]);
                t += 32;
                if (t >= st * 32)
                {
                    t = lane;
                    r += NW;
                }
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (z[u] >= 0)
                {
                    As[z[u]] = e[u];
                    if (kFold) As[BM * lda + z[u]] = o[u];
                }
        }
    };
    auto fill_cols = [&](auto* x0) {  // lanes across the rows
        const int   r = tid % BM;
        const auto* x = x0 + (long long)r * sg.rs;
        const int   ts = sg.ts;
        for (int t0 = tid / BM; t0 < Kp; t0 += kU * (NT / BM))
        {
            double e[kU], o[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                const int t = t0 + u * (NT / BM);
                e[u] = o[u] = 0;
                if (r < rows && t < K)
                    dense_in<KIND, INV>(T, t, [=](int i) { return (double)x[(long long)i * ts]; }, e[u], o[u]);
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                const int t = t0 + u * (NT / BM);
                if (t >= Kp) continue;
                As[r * lda + t] = e[u];
                if (kFold) As[(BM + r) * lda + t] = o[u];
            }
        }
    };
    if (sg.ts == 1)
    {
        if (in32) fill_rows(static_cast<const float*>(sg.in) + base);
        else fill_rows(static_cast<const double*>(sg.in) + base);
    }
    else fill_cols(static_cast<const double*>(sg.in) + base);  // the middle axis of FP64 fields
    if (CS > 1)  // every CTA of the cluster has read the rows before any of them stores
    {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    double acc[2][TM][TN][2];
    int    kc = 0, ct = rank;
    for (int i = 0; i < iters; ++i)
    {
        if (kc == 0)
#pragma unroll
            for (int par = 0; par < 2; ++par)
#pragma unroll
                for (int a = 0; a < TM; ++a)
#pragma unroll
                    for (int b = 0; b < TN; ++b) acc[par][a][b][0] = acc[par][a][b][1] = 0.0;
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();
        if (i + NS - 1 < iters) fetch((i + NS - 1) % NS);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double* b0 = Bs + (i % NS) * 2 * BK * (BN + 4) + (lane & 3) * (BN + 4) + wn * TN * 8 + (lane >> 2);
        const double* a0 = As + (wm * TM * 8 + (lane >> 2)) * lda + kc * BK + (lane & 3);
#pragma unroll
        for (int k = 0; k < BK / 4; ++k)
        {
            double av[kFold ? 2 : 1][TM], bv[2][TN];
#pragma unroll
            for (int par = 0; par < (kFold ? 2 : 1); ++par)
#pragma unroll
                for (int a = 0; a < TM; ++a) av[par][a] = a0[(par * BM + a * 8) * lda + k * 4];
#pragma unroll
            for (int par = 0; par < 2; ++par)
#pragma unroll
                for (int b = 0; b < TN; ++b) bv[par][b] = b0[(par * BK + k * 4) * (BN + 4) + b * 8];
#pragma unroll
            for (int par = 0; par < 2; ++par)
#pragma unroll
                for (int a = 0; a < TM; ++a)
#pragma unroll
                    for (int b = 0; b < TN; ++b) dense_mma(acc[par][a][b], av[kFold ? par : 0][a], bv[par][b]);
        }
        if (++kc < nk) continue;
        const int c0 = ct * BN + wn * TN * 8 + (lane & 3) * 2;
        kc = 0;
        ct += CS;
        // two elements in one store: unit stride, and every row starts on a pair
        const size_t esz = omode == DENSE_F32 ? 4 : 8;
        const bool   vec = sg.ts == 1 && sg.rs % 2 == 0 && (KIND == 0 || T.C % 2 == 0) &&
                         (reinterpret_cast<size_t>(sg.out) + base * esz) % (2 * esz) == 0;
        const bool   f64 = omode == DENSE_F64 && vec;
#pragma unroll
        for (int a = 0; a < TM; ++a)
        {
            const int r = wm * TM * 8 + a * 8 + (lane >> 2);
            if (r >= rows) continue;
            const long long ro = base + (long long)r * sg.rs;
            if (f64)  // the common case apart: its stores are one instruction each
            {
                double* const d = static_cast<double*>(sg.out) + ro;
                auto put  = [=](int q, double v) { d[q] = v; };
                auto put2 = [=](int q, double u, double v) { *reinterpret_cast<double2*>(d + q) = make_double2(u, v); };
#pragma unroll
                for (int b = 0; b < TN; ++b) dense_out<KIND, INV>(T, c0 + b * 8, acc[0][a][b], acc[1][a][b], put, put2);
                continue;
            }
            auto put = [&](int q, double v) {
                const long long z = ro + (long long)q * sg.ts;
                if (omode == DENSE_F32) static_cast<float*>(sg.out)[z] = (float)v;
                else if (omode == DENSE_ACC) static_cast<double*>(sg.out)[z] += v;
                else static_cast<double*>(sg.out)[z] = v;
            };
            auto put2 = [&](int q, double u, double v) {
                if (!vec)
                {
                    put(q, u);
                    put(q + 1, v);
                    return;
                }
                if (omode == DENSE_F32)
                {
                    *reinterpret_cast<float2*>(static_cast<float*>(sg.out) + ro + q) = make_float2((float)u, (float)v);
                    return;
                }
                double2*      d = reinterpret_cast<double2*>(static_cast<double*>(sg.out) + ro + q);  // DENSE_ACC
                const double2 w = *d;
                *d              = make_double2(u + w.x, v + w.y);
            };
#pragma unroll
            for (int b = 0; b < TN; ++b) dense_out<KIND, INV>(T, c0 + b * 8, acc[0][a][b], acc[1][a][b], put, put2);
        }
    }
}

}  // namespace fpb
