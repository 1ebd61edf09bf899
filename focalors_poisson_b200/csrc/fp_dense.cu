// Tables and launches of the dense y-transforms (fp_dense.cuh).
#include "fp_dense.h"

#include <algorithm>
#include <climits>

namespace fpb
{
namespace
{
// Entry (i, j) of the full forward matrix of ND and DN (fp_transform.cuh out_value): out_j = sum_i M(i, j) f_i.
__device__ double full_entry(int kind, int n, int i, int j, double s1, const double* ta, const double* tb)
{
    const int       L   = 2 * n + 1;
    const long long q   = (long long)(i + 1) * (j + 1) % L;
    double          sn, cs;
    sincospi(2.0 * (double)q / (double)L, &sn, &cs);
    if (kind == K_DN) return (((i ^ j) & 1) ? -s1 : s1) * sn;
    return ((i & 1) ? s1 : -s1) * (tb[j] * cs + ta[j] * sn);
}

// te / to [rows][ldb]: the two products' matrices, zero beyond K x C.
__global__ void k_dense_tables(int kind, int inv, int n, int K, int C, int rows, int ldb, double* te, double* to,
                               double s1, double s2, const double* ta, const double* tb)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= rows * ldb) return;
    const int t = q / ldb, c = q - t * ldb;
    double    e = 0, o = 0;
    if (t < K && c < C)
    {
        if (kind == K_DD)  // sqrt(2/(n+1)) sin(pi (t+1)(k+1)/(n+1)), k = 2c and 2c + 1
        {
            const long long L2 = 2LL * (n + 1);
            e = s1 * sinpi((double)((long long)(t + 1) * (2 * c + 1) % L2) / (double)(n + 1));
            if (2 * c + 1 < n) o = s1 * sinpi((double)((long long)(t + 1) * (2 * c + 2) % L2) / (double)(n + 1));
        }
        else if (kind == K_NN)  // mode m at point i: sqrt(1/n), -sqrt(2/n) cos(pi m (2i+1) / 2n)
        {
            const int  i  = inv ? c : t, m0 = 2 * (inv ? t : c);
            const auto w  = [&](int m) {
                return (m ? -s1 : s2) * cospi((double)((long long)m * (2 * i + 1) % (4LL * n)) / (double)(2 * n));
            };
            e = w(m0);
            if (m0 + 1 < n) o = w(m0 + 1);
        }
        else if (kind == K_PP)  // frequency h - c (forward) or h - t (inverse)
        {
            const int       h = n / 2;
            const long long k = (long long)(inv ? h - t : h - c) * (inv ? c : t) % n;
            sincospi(2.0 * (double)k / (double)n, &o, &e);
        }
        else
        {
            const int c2 = c + C;
            e = inv ? full_entry(kind, n, c, t, s1, ta, tb) : full_entry(kind, n, t, c, s1, ta, tb);
            if (c2 < n) o = inv ? full_entry(kind, n, c2, t, s1, ta, tb) : full_entry(kind, n, t, c2, s1, ta, tb);
        }
    }
    te[q] = e;
    to[q] = o;
}
}  // namespace

// Where the lines lie, by row length n, rows of a run, storage of the FFT it replaces and whether that FFT is one of
// its own length (7-smooth n + 1, n or 2 n + 1: direct) or a convolution of twice the length, two to three times as
// dear. Time of the product over the FFT's, forward + inverse, in place:
//   rows                   128  1024  2048  3072  4736  4768  8192 32768
//   FP64 DD  95 direct     .87   .97   .97  1.32   .83   .97   .72   .67
//   FP64 DD 127 direct     .90  1.00  1.06  1.42  1.00  1.17   .89   .86
//   FP64 DD 159 direct    1.14  1.27  1.52  1.79  1.23  1.57  1.13  1.09
//   FP64 DD 192            .75   .80   .99  1.02   .69   .96   .66   .58
//   FP64 DD 256            .53   .75  1.19  1.26   .83  1.20   .95   .78
//   FP64 NN  64 direct     .83   .82   .82   .80   .66   .77   .58   .55
//   FP64 NN  96 direct     .91   .92  1.04  1.38   .82  1.01   .74   .72
//   FP64 PP  60 direct     .87   .82   .55   .52   .50   .55   .39   .34
//   FP64 PP  96 direct    1.16  1.06   .84  1.11   .72   .89   .61   .59
//   FP64 PP 144 direct    1.32  1.33  1.05  1.19   .87  1.11   .75   .72
//   FP64 DN 121 direct     .73   .79  1.05  1.27   .68   .97   .74   .75
//   FP64 DN 187 direct    1.24  1.33  2.00  1.91  1.23  1.99  1.38  1.35
//   FP64 DN 192            .69   .76  1.04   .91   .62  1.04   .70   .62
//   FP64 DN 224            .50   .86  1.24  1.13   .77  1.26   .85   .76
//   FP32 DD 127 direct    1.01  1.08  1.13  1.57  1.23  1.23  1.03   .93
//   FP32 DD 192            .85   .89  1.14  1.21   .96  1.10   .82   .69
//   FP32 PP 144 direct    1.36  1.40  1.44  1.21   .96  1.16   .82   .78
//   FP32 DN 192            .89   .95  1.36  1.26  1.00  1.38   .97   .80
// The steps are waves of 32-row tiles, 148 and 296 of them (4736 and 9472 rows), and the change of launch shape at
// 2560 or 3200 rows. Where they cross 1 the FFT takes the rows between, one range per band; beside it up to a tenth, at
// a few lengths two or three in the first rows of a wave, is left. FP32 rows keep FP64 arithmetic in the product and have
// the faster FFT, so their lines are lower.
namespace
{
constexpr int kNever = INT_MAX;
struct DenseBand  // row lengths up to `last` (from the band before)
{
    int last, from, to;  // FFT for `from` <= rows < `to`
};
using Bands = std::vector<DenseBand>;
const Bands& dense_bands(int kind, bool direct, bool f32)
{
    // [FP64 / FP32][family][convolution / direct]
    static const Bands b[2][4][2] = {
        {{{{144, 0, 0}, {199, 2048, 3584}, {256, 1536, 8192}}, {{63, 0, 0}, {96, 2048, 3584}, {127, 2048, 7168}}},
         {{{96, 0, 0}}, {{64, 0, 0}, {96, 2048, 3584}}},
         {{{199, 0, 0}, {224, 2048, 3584}},
          {{64, 0, 0}, {127, 2048, 3584}, {190, 0, kNever}, {224, 1024, kNever}}},
         {{{144, 0, 0}}, {{60, 0, 0}, {126, 0, 2048}, {144, 0, 7168}}}},
        {{{{144, 0, 0}, {199, 1536, 6144}, {224, 1536, kNever}},
          {{63, 0, 0}, {96, 2560, 4736}, {127, 1536, 12288}}},
         {{{96, 0, 0}}, {{64, 0, 0}, {96, 1024, 5632}}},
         {{{128, 0, 0}, {144, 2048, 14208}, {175, 1536, kNever}, {192, 1536, 8192}},
          {{64, 0, 0}, {80, 2048, 7168}, {121, 1536, 14208}}},
         {{{144, 0, 0}}, {{60, 0, 0}, {126, 0, 3200}, {144, 0, 7168}}}}};
    const int family = kind == K_DD ? 0 : kind == K_NN ? 1 : kind == K_PP ? 3 : 2;
    return b[f32][family][direct];
}
}  // namespace

DenseRule dense_rule(int kind, int n, bool f32)
{
    DenseRule r;
    for (const DenseBand& b : dense_bands(kind, fft_direct(fft_length(kind, n)), f32))
        if (n <= b.last)
        {
            r.from = b.from;
            r.to   = b.to == kNever ? LLONG_MAX : b.to;
            break;
        }
    return r;
}

DensePlan::DensePlan(int kind_, int n_) : kind(kind_), n(n_)
{
    const KindTables kt = kind_tables(kind, n);
    s1                  = kt.s1;
    if (kind == K_ND || kind == K_PP)
    {
        ta = upload(kt.a);
        tb = upload(kt.b);
    }
    const DenseTab t    = tab(false);
    const int      rows = (t.K + kDenseBK - 1) / kDenseBK * kDenseBK;
    for (int inv = 0; inv < (kind == K_DD || kind == K_DN ? 1 : 2); ++inv)
    {
        te[inv].alloc((size_t)rows * t.ldb * sizeof(double));
        to[inv].alloc((size_t)rows * t.ldb * sizeof(double));
        k_dense_tables<<<(rows * t.ldb + 255) / 256, 256>>>(kind, inv, n, t.K, t.C, rows, t.ldb, te[inv].as<double>(),
                                                           to[inv].as<double>(), kt.s1, kt.s2, ta.as<double>(),
                                                           tb.as<double>());
        FPB_CHECK_LAUNCH();
    }
    FPB_CUDA(cudaStreamSynchronize(0));  // the tables are read on any stream
}

DenseTab DensePlan::tab(bool inverse) const
{
    const int d = inverse && (kind == K_NN || kind == K_ND || kind == K_PP) ? 1 : 0;
    DenseTab  t{};
    t.n   = n;
    t.C   = kind == K_PP ? n / 2 + 1 : (n + 1) / 2;
    t.K   = dense_fold(kind) ? t.C : n;
    t.ldb = (t.C + 79 + 15) / 16 * 16;  // any column tile of up to 80 stays inside
    t.te  = te[d].as<double>();
    t.to  = to[d].as<double>();
    t.ta  = ta.as<double>();
    t.tb  = tb.as<double>();
    t.s1  = s1;
    return t;
}

namespace
{
// Launch shapes. 0-3: 32-row tiles of 32, 48, 64 or 80 columns, eight warps as 4 x 2 (two CTAs per SM up to 256
// columns folded, so that one loads or stores while the other multiplies); 4: 8-row tiles whose columns a cluster
// shares, for few rows.
constexpr int kCfgs = 5, kSmall = 4, kCfgBM[kCfgs] = {32, 32, 32, 32, 8}, kCfgBN[kCfgs] = {32, 48, 64, 80, 32},
              kCfgThreads[kCfgs] = {256, 256, 256, 256, 128};

template <int KIND, int INV> const void* dense_kernel(int cfg)
{
    switch (cfg)
    {
        case 0: return (const void*)k_dense<KIND, INV, 1, 2, 4, 2>;
        case 1: return (const void*)k_dense<KIND, INV, 1, 3, 4, 2>;
        case 2: return (const void*)k_dense<KIND, INV, 2, 2, 2, 4>;
        case 3: return (const void*)k_dense<KIND, INV, 1, 5, 4, 2>;
        default: return (const void*)k_dense<KIND, INV, 1, 1, 1, 4>;
    }
}
const void* dense_kernel(int kind, bool inverse, int cfg)
{
    switch (kind)
    {
        case K_DD: return dense_kernel<K_DD, 0>(cfg);
        case K_NN: return inverse ? dense_kernel<K_NN, 1>(cfg) : dense_kernel<K_NN, 0>(cfg);
        case K_PP: return inverse ? dense_kernel<K_PP, 1>(cfg) : dense_kernel<K_PP, 0>(cfg);
        default: return dense_kernel<K_ND, 0>(cfg);  // ND and DN: the direction is in the table
    }
}
}  // namespace

DenseShape dense_shape(int kind, const std::vector<DenseLoad>& loads)
{
    const bool fold = dense_fold(kind);
    int        maxK = 0, maxC = 0;
    long long  rows = 0;
    for (const DenseLoad& l : loads)
    {
        maxK = std::max(maxK, l.K);
        maxC = std::max(maxC, l.C);
        rows += l.rows;
    }
    auto smem = [&](int c) { return (size_t)dense_smem(fold, maxK, kCfgBM[c], kCfgBN[c]) * sizeof(double); };
    DenseShape sh;
    sh.cfg = kSmall;
    // From 80 tiles of 32 rows on (100 where the products are narrow), the column tile with the least work, padding
    // included. us, large / small tiles, FP64: 2560 rows DD 120 10.1 / 8.1, DD 160 14.2 / 15.9; 3200 rows DD 64 5.6 / 5.1,
    // DD 128 9.7 / 10.8, DD 160 14.3 / 17.6, ND 192 19.4 / 24.2.
    if (rows >= (maxC <= 64 ? 100LL : 80LL) * kCfgBM[0])
    {
        double best = 0;
        for (int c = 0; c < kSmall; ++c)
        {
            double w = 0;
            for (const DenseLoad& l : loads)
                w += (double)l.rows * l.K * ((l.C + kCfgBN[c] - 1) / kCfgBN[c] * kCfgBN[c]);
            if (smem(c) <= max_dynamic_smem() && (sh.cfg == kSmall || w <= best))
            {
                best   = w;
                sh.cfg = c;
            }
        }
    }
    sh.bm      = kCfgBM[sh.cfg];
    sh.smem    = smem(sh.cfg);
    sh.cluster = 1;
    if (sh.cfg == kSmall)
        while (sh.cluster < 4 && 2 * sh.cluster <= (maxC + kCfgBN[kSmall] - 1) / kCfgBN[kSmall]) sh.cluster *= 2;
    return sh;
}

void dense_launch(int kind, bool inverse, const DenseShape& sh, const DenseSeg* segs, const long long* prefix, int nseg,
                  const DenseTab* tabs, const DenseSeg& one, const DenseTab& tv, long long items, bool in32, int omode,
                  cudaStream_t s)
{
    if (items <= 0) return;
    if (items * sh.cluster > (long long)INT_MAX) throw Error(3, "more than 2^31 tiles in one transform");
    const void* fn = dense_kernel(kind, inverse, sh.cfg);
    allow_max_dynamic_smem(fn);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim            = dim3((unsigned)(items * sh.cluster));
    cfg.blockDim           = dim3(kCfgThreads[sh.cfg]);
    cfg.dynamicSmemBytes   = sh.smem;
    cfg.stream             = s;
    cudaLaunchAttribute at[1];
    at[0].id               = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = sh.cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs              = at;
    cfg.numAttrs           = sh.cluster > 1 ? 1 : 0;
    int   in32i = in32 ? 1 : 0, cs = sh.cluster;
    void* args[] = {(void*)&segs, (void*)&prefix, (void*)&nseg, (void*)&tabs, (void*)&one, (void*)&tv, &in32i, &omode, &cs};
    FPB_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
    FPB_CHECK_LAUNCH();
}

namespace
{
void run_seg(const DensePlan& p, bool inverse, const DenseSeg& sg, bool in32, int omode, cudaStream_t s)
{
    const DenseTab   t    = p.tab(inverse);
    const DenseShape sh   = dense_shape(p.kind, {{t.K, t.C, (long long)sg.rows * sg.slabs}});
    const long long  per  = (sg.rows + sh.bm - 1) / sh.bm;
    dense_launch(p.kind, inverse, sh, nullptr, nullptr, 1, nullptr, sg, t, per * sg.slabs, in32, omode, s);
}
}  // namespace

void dense_rows(const DensePlan& p, bool inverse, const void* in, void* out, long long rows, bool in32, int omode,
                cudaStream_t s)
{
    run_seg(p, inverse, DenseSeg{in, out, 0, (int)rows, 1, p.n, 1, 0}, in32, omode, s);
}

void dense_middle(const DensePlan& p, bool inverse, const double* in, double* out, long long slabs, int inner,
                  cudaStream_t s)
{
    if (slabs > (long long)INT_MAX) throw Error(3, "more than 2^31 slabs in one transform");
    run_seg(p, inverse, DenseSeg{in, out, (long long)p.n * inner, inner, (int)slabs, 1, inner, 0}, false, DENSE_F64, s);
}
}  // namespace fpb
