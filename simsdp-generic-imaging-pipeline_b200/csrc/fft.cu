// 2-D complex FFT (FFTW convention: sign -1 forward, +1 inverse,
// unnormalised; fft_run.c:23-83) and the fused imaging transforms of the
// FFT pipeline.
//
// A transform is a row pass and a column pass.  A line of N points is a
// Stockham autosort FFT, N = 16 16 ... and a last radix 8, 4 or 2, with 16
// points per thread: in a stage a thread takes R points at stride N / R,
// multiplies point t by the twiddle W_{Ns R}^{t k} (k = butterfly index mod
// the span Ns done so far), does an R-point DFT in registers (16 = 4 x 4, 8 =
// 2 x 4) and writes the outputs to their sorted places; shared memory is
// touched once per stage, and the first stage reads, the last stage writes
// global memory directly.  Row CTAs hold one or more whole rows.  Column CTAs
// hold four adjacent columns (one 32-byte sector per row) of up to 2048
// points, or eight of 1024 at 4096 and 8192 points; those columns are spread
// over a cluster of Q CTAs: CTA c transforms the rows = c mod Q, and a radix-Q
// step over distributed shared memory joins them.  (A CTA that held all of an
// 8192-point column had room for one column: 8 bytes of every sector, 1290 us
// a pass.)
// Row / column pass of the imaging transforms: 2048^2 10-12 / 18-19 us, 8192^2
// 135-150 / 288-318 us (with full complex transforms 13-14 / 24-26 and
// 225-238 / 450-494; the kernels before those 55 / 36 and 980 / 1290).  Rows
// are bound by the L1 data path (75 % of its wavefronts in four stages at
// 8192: shared memory and twiddle loads), columns by one tag lookup per 32 or
// 64 bytes and the barriers of two 512-thread CTAs per SM.
// Twiddles come from tables built in double: exp(-2 pi i k / N), and per
// stage in the order in which the lanes of a warp read them.
// The inverse is the forward transform with real and imaginary parts
// swapped on the way in and on the way out.
//
// The checkerboard fftshift (fft_run.c:14, 96, 114) is applied while the
// first pass loads and while the second pass stores, and the taper
// correction (convolution_correction_run.c:4-35) in the second pass's store.
// An image is real, so both imaging transforms do half of the arithmetic and
// the second pass reads half of the array:
//   image -> grid: a row line is two image rows as real and imaginary part
//     (LOAD_REAL_PAIR), taken apart into columns 0 .. N / 2 of both rows
//     (STORE_PAIR); the column pass transforms those columns (LOAD_HALF) and
//     writes each result and its conjugate at the mirrored cell
//     (STORE_MIRROR).
//   grid -> image: the real part of the inverse transform is the inverse
//     transform of the grid's Hermitian part, (Z(k) + conj Z(-k)) / 2; the
//     row pass forms and transforms its rows 0 .. N / 2 (LOAD_HERMITIAN), the
//     column pass packs two columns into one line (LOAD_PACKED, the other
//     half of a column from its conjugate symmetry) and gets their pixels as
//     real and imaginary part (STORE_REAL_TAPER).
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include <cooperative_groups.h>

#include "common.cuh"

namespace sdp {

namespace cg = cooperative_groups;

// What a pass reads and writes (see the head of the file for the imaging
// transforms' four).
enum { LOAD_PLAIN = 0, LOAD_REAL_PAIR = 1, LOAD_HERMITIAN = 2, LOAD_HALF = 3, LOAD_PACKED = 4 };
enum { STORE_PLAIN = 0, STORE_PAIR = 1, STORE_MIRROR = 2, STORE_REAL_TAPER = 3 };

// Lines of a pass.
__host__ __device__ constexpr int fft_lines(int ld, int n)
{
    return ld == LOAD_REAL_PAIR || ld == LOAD_PACKED ? n / 2 : ld == LOAD_HERMITIAN || ld == LOAD_HALF ? n / 2 + 1 : n;
}

// Stages of an N-point line: radix 16, the last one 2^(log2 N mod 4).
__host__ __device__ constexpr int fft_stages(int log2n) { return log2n / 4 + (log2n % 4 ? 1 : 0); }
__host__ __device__ constexpr int fft_radix(int log2n, int st) { return st < log2n / 4 ? 16 : 1 << (log2n % 4); }
// First entry of stage st in the packed twiddles of a line: stage st holds
// (R - 1) Ns entries W_{Ns R}^{t k} at (t - 1) Ns + k.
__host__ __device__ constexpr int fft_tw_offset(int log2n, int st)
{
    int o = 0, ns = 1;
    for (int s = 0; s < st; ++s) {
        if (s > 0) o += (fft_radix(log2n, s) - 1) * ns;
        ns *= fft_radix(log2n, s);
    }
    return o;
}
__host__ __device__ constexpr int fft_tw_entries(int log2n) { return fft_tw_offset(log2n, fft_stages(log2n)); }
// log2 of the column points in one CTA: whole columns up to 2048 points, then
// 1024 points of eight columns (half the cluster's CTAs are worth less than
// 64 contiguous bytes: 4096^2 226 -> 216 us, 8192^2 942 -> 886 us for both
// imaging transforms against 2048 points of four; at 2048^2 60 -> 63), up to
// eight CTAs per cluster.
__host__ __device__ constexpr int fft_column_part(int log2n) { return log2n <= 11 ? log2n : (log2n <= 13 ? 10 : log2n - 3); }

__global__ void k_twiddles(int N, float2 *tw)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
        double s, c;
        sincospi(__ddiv_rn(2.0 * (double)k, (double)N), &s, &c);
        tw[k] = make_float2((float)c, (float)(-s));
    }
}

// Packed twiddles of stages 1.. of a 2^log2n-point line.
__global__ void k_twiddles_packed(int log2n, float2 *tw)
{
    const int total = fft_tw_entries(log2n);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int st = 1, ns = 16;
        while (e >= fft_tw_offset(log2n, st + 1)) {
            ns *= fft_radix(log2n, st);
            ++st;
        }
        const int r = fft_radix(log2n, st), q = e - fft_tw_offset(log2n, st);
        const int t = q / ns + 1, k = q % ns;
        double s, c;
        sincospi(__ddiv_rn(2.0 * (double)(t * k), (double)(ns * r)), &s, &c);
        tw[e] = make_float2((float)c, (float)(-s));
    }
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 swapped(float2 a) { return make_float2(a.y, a.x); }
// times -i
__device__ __forceinline__ float2 rot90(float2 a) { return make_float2(a.y, -a.x); }

__device__ __forceinline__ void dft2(float2 &a, float2 &b)
{
    const float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

__device__ __forceinline__ void dft4(float2 &a0, float2 &a1, float2 &a2, float2 &a3)
{
    const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2);
    const float2 t2 = cadd(a1, a3), t3 = rot90(csub(a1, a3));
    a0 = cadd(t0, t2);
    a2 = csub(t0, t2);
    a1 = cadd(t1, t3);
    a3 = csub(t1, t3);
}

// exp(-2 pi i j / 16) for j = 0..15 written as constants of cos/sin(pi j / 8)
__device__ __forceinline__ float2 w16(int j)
{
    const float c1 = 0.92387953251128674f, s1 = 0.38268343236508978f, h = 0.70710678118654752f;
    switch (j & 15) {
    case 0: return make_float2(1.f, 0.f);
    case 1: return make_float2(c1, -s1);
    case 2: return make_float2(h, -h);
    case 3: return make_float2(s1, -c1);
    case 4: return make_float2(0.f, -1.f);
    case 5: return make_float2(-s1, -c1);
    case 6: return make_float2(-h, -h);
    case 7: return make_float2(-c1, -s1);
    case 8: return make_float2(-1.f, 0.f);
    case 9: return make_float2(-c1, s1);
    case 10: return make_float2(-h, h);
    case 11: return make_float2(-s1, c1);
    case 12: return make_float2(0.f, 1.f);
    case 13: return make_float2(s1, c1);
    case 14: return make_float2(h, h);
    default: return make_float2(c1, s1);
    }
}

// In-register R-point forward DFT of a[0 .. R - 1] (natural order in and out).
template <int R>
__device__ __forceinline__ void dft_r(float2 *a)
{
    if constexpr (R == 2) {
        dft2(a[0], a[1]);
    } else if constexpr (R == 4) {
        dft4(a[0], a[1], a[2], a[3]);
    } else if constexpr (R == 8) {
        // n = m + 2 l (m < 2, l < 4); k = k1 + 4 k2
        dft4(a[0], a[2], a[4], a[6]);
        dft4(a[1], a[3], a[5], a[7]);
        // twiddle W8^{k1} on the odd half, then 2-point DFTs
        float2 x[8];
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            float2 o = a[2 * k1 + 1];
            if (k1 == 2) o = rot90(o);
            else if (k1) o = cmulf(o, w16(2 * k1));
            const float2 e = a[2 * k1];
            x[k1] = cadd(e, o);
            x[k1 + 4] = csub(e, o);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = x[i];
    } else if constexpr (R == 16) {
        // n = m + 4 l; inner DFT4 over l for each m, twiddle W16^{m k1}, outer DFT4 over m
#pragma unroll
        for (int m = 0; m < 4; ++m) dft4(a[m], a[m + 4], a[m + 8], a[m + 12]);
#pragma unroll
        for (int m = 1; m < 4; ++m)
#pragma unroll
            for (int k1 = 1; k1 < 4; ++k1)
                a[m + 4 * k1] = m * k1 == 4 ? rot90(a[m + 4 * k1]) : cmulf(a[m + 4 * k1], w16(m * k1));
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) dft4(a[4 * k1], a[4 * k1 + 1], a[4 * k1 + 2], a[4 * k1 + 3]);
        // a[4 k1 + k2] holds X[k1 + 4 k2]: transpose the 4 x 4 index
        float2 t[16];
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) t[k1 + 4 * k2] = a[4 * k1 + k2];
#pragma unroll
        for (int i = 0; i < 16; ++i) a[i] = t[i];
    }
}

__device__ __forceinline__ float checker(int r, int c) { return ((r + c) & 1) ? -1.f : 1.f; }

struct FftArgs {
    const void *in;
    void *out;
    const float2 *tw;       // exp(-2 pi i k / N), k < N (the join of column parts)
    const float2 *twp;      // packed stage twiddles of the CTA's lines
    const float *prolate;   // taper table (STORE_REAL_TAPER)
    int swap;               // LOAD_PLAIN (rows), STORE_PLAIN (columns): real and imaginary parts swapped
};

// Sizes of a pass: G x G array, lines of 2^LOG2N points.
template <bool ROWS, int LOG2N>
struct Pass {
    static constexpr int N = 1 << LOG2N;
    static constexpr int LOG2M = ROWS ? LOG2N : fft_column_part(LOG2N);  // of the part in one CTA
    static constexpr int M = 1 << LOG2M;
    static constexpr int Q = N / M;  // CTAs per cluster
    // lines per CTA: rows up to 128 threads, columns a sector
    static constexpr int L = ROWS ? (N >= 2048 ? 1 : (2048 / N < N ? 2048 / N : N)) : (LOG2N == 12 || LOG2N == 13 ? 8 : 4);
    static constexpr int THREADS = L * M / 16;
    static constexpr int kMinBlocks = THREADS >= 32 ? 1024 / THREADS : 32;  // 64 registers a thread
    // one padding element after every 16: the first stage writes at a stride
    // of 16 points, which would otherwise put a warp's stores on few banks
    static constexpr int kSmem = (L * M + L * M / 16) * (int)sizeof(float2);
    __device__ static __forceinline__ int sidx(int l, int i)
    {
        const int k = ROWS ? l * M + i : i * L + l;
        return k + (k >> 4);
    }
    // butterfly b of a radix-R stage: line l, index j in it
    template <int R>
    __device__ static __forceinline__ void split(int b, int &l, int &j)
    {
        constexpr int per_line = M / R;
        if (ROWS) {
            l = b / per_line;
            j = b % per_line;
        } else {
            l = b % L;
            j = b / L;
        }
    }
};

// Point i of line `line`.
template <bool ROWS, int LD>
__device__ __forceinline__ float2 load_point(const FftArgs &A, int N, int line, int i)
{
    if (LD == LOAD_REAL_PAIR) {
        const float *in = static_cast<const float *>(A.in) + (size_t)(2 * line) * N + i;
        const float a = checker(0, i);  // of the even row
        return make_float2(__ldg(in) * a, -(__ldg(in + N) * a));
    }
    const float2 *in = static_cast<const float2 *>(A.in);
    if (LD == LOAD_HERMITIAN) {
        const float2 a = __ldg(in + (size_t)line * N + i);
        const float2 b = __ldg(in + (size_t)((N - line) & (N - 1)) * N + ((N - i) & (N - 1)));
        const float h = 0.5f * checker(line, i);
        return make_float2((a.y - b.y) * h, (a.x + b.x) * h);  // swapped
    }
    if (LD == LOAD_PACKED) {
        const int j = i <= N / 2 ? i : N - i;
        const float2 *p = in + (size_t)j * N + 2 * line;
        float2 y1 = swapped(__ldg(p)), y2 = swapped(__ldg(p + 1));  // (the row pass left them swapped)
        // rows 0 and N / 2 of the symmetric half are real
        const float sg = (j == 0 || j == N / 2) ? 0.f : (i <= N / 2 ? 1.f : -1.f);
        y1.y *= sg;
        y2.y *= sg;
        return make_float2(y1.y + y2.x, y1.x - y2.y);  // y1 + i y2, swapped
    }
    float2 v = ROWS ? __ldg(in + (size_t)line * N + i) : __ldg(in + (size_t)i * N + line);
    if (ROWS && A.swap) v = swapped(v);
    return v;
}

__device__ __forceinline__ float taper_pixel(const FftArgs &A, int N, int r, int c, float x)
{
    const int half = N / 2;
    const int dc = abs(c - half), dr = abs(r - half);
    float taper = __fmul_rn(__ldg(A.prolate + dc), __ldg(A.prolate + dr));
    if (dc == 1229 || dr == 1229) taper = 0.f;
    // |taper| > 1E-10 as doubles: 1E-10f is the first float above it
    return fabsf(taper) >= 1E-10f ? __fdiv_rn(x * checker(r, c), taper) : 0.f;
}

template <bool ROWS, int STO>
__device__ __forceinline__ void store_point(const FftArgs &A, int N, int line, int i, float2 v)
{
    if (STO == STORE_REAL_TAPER) {
        // the two columns' pixels are the real and imaginary part after the swap
        float *out = static_cast<float *>(A.out) + (size_t)i * N + 2 * line;
        out[0] = taper_pixel(A, N, i, 2 * line, v.y);
        out[1] = taper_pixel(A, N, i, 2 * line + 1, v.x);
        return;
    }
    float2 *out = static_cast<float2 *>(A.out);
    if (STO == STORE_MIRROR) {
        const float a = checker(i, line);
        out[(size_t)i * N + line] = make_float2(v.x * a, v.y * a);
        if (line > 0 && line < N / 2)
            out[(size_t)((N - i) & (N - 1)) * N + (N - line)] = make_float2(v.x * a, -(v.y * a));
        return;
    }
    if (!ROWS && A.swap) v = swapped(v);
    if (ROWS)
        out[(size_t)line * N + i] = v;
    else
        out[(size_t)i * N + line] = v;
}

// Stage ST and all that follow.  A thread first reads all of its butterflies
// (16 points) into registers; a barrier separates those reads from the
// writes, so one shared buffer serves in place.
template <bool ROWS, int LOG2N, int LD, int STO, int ST, int NS>
__device__ __forceinline__ void run_stages(const FftArgs &A, float2 *__restrict__ s, int first, int part)
{
    using P = Pass<ROWS, LOG2N>;
    constexpr int NST = fft_stages(P::LOG2M);
    constexpr int R = fft_radix(P::LOG2M, ST), NB = 16 / R, per_line = P::M / R;
    constexpr bool FIRST = ST == 0, LAST = ST == NST - 1, GLOBAL = LAST && P::Q == 1 && STO != STORE_PAIR;
    constexpr int lines = fft_lines(LD, P::N);
    constexpr bool kWhole = lines % P::L == 0;  // no CTA has lines past the last
    float2 a[16];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        int l, j;
        P::template split<R>(threadIdx.x + q * P::THREADS, l, j);
#pragma unroll
        for (int t = 0; t < R; ++t) {
            const int i = j + t * per_line;
            if (FIRST) {
                a[q * R + t] =
                    load_point<ROWS, LD>(A, P::N, kWhole ? first + l : min(first + l, lines - 1), i * P::Q + part);
            } else {
                a[q * R + t] = s[P::sidx(l, i)];
            }
        }
    }
    if (!FIRST && !GLOBAL) __syncthreads();  // reads of this stage complete before in-place writes
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        int l, j;
        P::template split<R>(threadIdx.x + q * P::THREADS, l, j);
        const int k = j & (NS - 1);
        if (!FIRST) {
            const float2 *tw = A.twp + fft_tw_offset(P::LOG2M, ST) + k;
#pragma unroll
            for (int t = 1; t < R; ++t) a[q * R + t] = cmulf(a[q * R + t], __ldg(tw + (t - 1) * NS));
        }
        dft_r<R>(a + q * R);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int t = 0; t < R; ++t) {
            const int i = base + t * NS;
            if (GLOBAL) {
                if (kWhole || first + l < lines) store_point<ROWS, STO>(A, P::N, first + l, i, a[q * R + t]);
            } else {
                s[P::sidx(l, i)] = a[q * R + t];
            }
        }
    }
    if constexpr (!LAST) {
        __syncthreads();  // writes visible to the next stage
        run_stages<ROWS, LOG2N, LD, STO, ST + 1, NS * R>(A, s, first, part);
    }
}

// One pass over all lines of a G x G array (ROWS: lines are rows).
template <bool ROWS, int LOG2N, int LD, int STO>
__global__ void __launch_bounds__(Pass<ROWS, LOG2N>::THREADS, Pass<ROWS, LOG2N>::kMinBlocks) k_fft_pass(FftArgs A)
{
    using P = Pass<ROWS, LOG2N>;
    extern __shared__ float2 s[];
    const int first = (int)(blockIdx.x / P::Q) * P::L;
    const int part = (int)(blockIdx.x % P::Q);  // the rank in the cluster
    run_stages<ROWS, LOG2N, LD, STO, 0, 1>(A, s, first, part);
    if constexpr (STO == STORE_PAIR) {
        // Z = A + i B of two real rows: A(k) = (Z(k) + conj Z(-k)) / 2,
        // B(k) = (Z(k) - conj Z(-k)) / 2i, k = 0 .. N / 2
        __syncthreads();
        constexpr int H = P::N / 2 + 1;
        for (int e = threadIdx.x; e < P::L * H; e += P::THREADS) {
            const int l = e / H, k = e - l * H;
            if (first + l >= fft_lines(LD, P::N)) break;
            const float2 z = s[P::sidx(l, k)], m = s[P::sidx(l, (P::N - k) & (P::N - 1))];
            float2 *out = static_cast<float2 *>(A.out) + (size_t)(2 * (first + l)) * P::N + k;
            out[0] = make_float2(0.5f * (z.x + m.x), 0.5f * (z.y - m.y));
            out[P::N] = make_float2(0.5f * (z.y + m.y), 0.5f * (m.x - z.x));
        }
    }
    if constexpr (P::Q > 1) {
        // X[k + M q] = sum over c of W_Q^{c q} W_N^{c k} Y_c[k]: CTA `part`
        // takes its share of the k's from all parts
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        constexpr int KQ = P::M / P::Q;
        const float2 *src[P::Q];
#pragma unroll
        for (int c = 0; c < P::Q; ++c) src[c] = cluster.map_shared_rank(s, c);
#pragma unroll
        for (int q = 0; q < 16 / P::Q; ++q) {
            const int e = threadIdx.x + q * P::THREADS, l = e % P::L, k = part * KQ + e / P::L;
            float2 a[P::Q];
#pragma unroll
            for (int c = 0; c < P::Q; ++c) a[c] = src[c][P::sidx(l, k)];
#pragma unroll
            for (int c = 1; c < P::Q; ++c) a[c] = cmulf(a[c], __ldg(A.tw + c * k));
            dft_r<P::Q>(a);
#pragma unroll
            for (int c = 0; c < P::Q; ++c)
                if (fft_lines(LD, P::N) % P::L == 0 || first + l < fft_lines(LD, P::N))
                    store_point<ROWS, STO>(A, P::N, first + l, k + P::M * c, a[c]);
        }
        cluster.sync();  // the other CTAs have read this one's shared memory
    }
}

struct TwKey {
    int dev, n;
    bool operator==(const TwKey &o) const { return dev == o.dev && n == o.n; }
};
struct TwHash {
    size_t operator()(const TwKey &k) const { return (size_t)k.dev * 1000003u + (size_t)k.n; }
};

static std::mutex g_tw_mutex;
static std::unordered_map<TwKey, float2 *, TwHash> g_tw;

// Twiddle tables for size N on the current device (allocated on first use,
// kept): exp(-2 pi i k / N), k < N, then the packed stage tables of a row and
// of a column part.
int fft_twiddles(int N, cudaStream_t st, const float2 **out)
{
    int dev = 0;
    SDP_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_tw_mutex);
    auto it = g_tw.find({dev, N});
    if (it != g_tw.end()) {
        *out = it->second;
        return SDP_OK;
    }
    int log2n = 0;
    while ((1 << log2n) < N) ++log2n;
    float2 *p = nullptr;
    const size_t row = (size_t)fft_tw_entries(log2n), col = (size_t)fft_tw_entries(fft_column_part(log2n));
    SDP_CUDA_TRY(cudaMalloc(&p, sizeof(float2) * ((size_t)N + row + col)));
    k_twiddles<<<std::max(1, std::min(1024, N / 256 + 1)), 256, 0, st>>>(N, p);
    k_twiddles_packed<<<64, 256, 0, st>>>(log2n, p + N);
    k_twiddles_packed<<<64, 256, 0, st>>>(fft_column_part(log2n), p + N + row);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        cudaFree(p);
        return cuda_error(e, "FFT twiddle tables");
    }
    g_tw[{dev, N}] = p;
    *out = p;
    return SDP_OK;
}

int check_fft_size(int G)
{
    if (G < 16 || G > 16384 || (G & (G - 1)) != 0)
        return set_error(SDP_ERR_RANGE, "FFT size %d must be a power of two in [16, 16384]", G);
    return SDP_OK;
}

template <bool ROWS, int LOG2N, int LD, int STO>
static int launch_pass_n(FftArgs A, cudaStream_t st)
{
    using P = Pass<ROWS, LOG2N>;
    auto fn = k_fft_pass<ROWS, LOG2N, LD, STO>;
    A.twp = A.tw + P::N + (P::Q > 1 ? fft_tw_entries(LOG2N) : 0);
    if (P::kSmem > 48 * 1024)
        SDP_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, P::kSmem));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((fft_lines(LD, P::N) + P::L - 1) / P::L * P::Q);
    cfg.blockDim = dim3(P::THREADS);
    cfg.dynamicSmemBytes = P::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = P::Q;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = P::Q > 1 ? 1 : 0;
    SDP_CUDA_TRY(cudaLaunchKernelEx(&cfg, fn, A));
    return SDP_OK;
}

template <bool ROWS, int LD, int STO>
static int launch_pass(int G, const void *in, void *out, const float2 *tw, const float *prolate, bool swap,
                       cudaStream_t st)
{
    const FftArgs A{in, out, tw, nullptr, prolate, swap ? 1 : 0};
    switch (G) {
    case 16: return launch_pass_n<ROWS, 4, LD, STO>(A, st);
    case 32: return launch_pass_n<ROWS, 5, LD, STO>(A, st);
    case 64: return launch_pass_n<ROWS, 6, LD, STO>(A, st);
    case 128: return launch_pass_n<ROWS, 7, LD, STO>(A, st);
    case 256: return launch_pass_n<ROWS, 8, LD, STO>(A, st);
    case 512: return launch_pass_n<ROWS, 9, LD, STO>(A, st);
    case 1024: return launch_pass_n<ROWS, 10, LD, STO>(A, st);
    case 2048: return launch_pass_n<ROWS, 11, LD, STO>(A, st);
    case 4096: return launch_pass_n<ROWS, 12, LD, STO>(A, st);
    case 8192: return launch_pass_n<ROWS, 13, LD, STO>(A, st);
    case 16384: return launch_pass_n<ROWS, 14, LD, STO>(A, st);
    default: return set_error(SDP_ERR_RANGE, "FFT size %d unsupported", G);
    }
}

}  // namespace sdp

using namespace sdp;

SDP_EXPORT int sdp_fft2d(int G, const sdp_float2 *in, sdp_float2 *out, int sign, void *stream)
{
    SDP_TRY(check_fft_size(G));
    SDP_CHECK_ARG(in && out, "NULL argument");
    SDP_CHECK_ARG(sign == -1 || sign == 1, "sign %d must be -1 or +1", sign);
    cudaStream_t st = as_stream(stream);
    const float2 *tw = nullptr;
    SDP_TRY(fft_twiddles(G, st, &tw));
    const bool inv = (sign == 1);
    SDP_TRY((launch_pass<true, LOAD_PLAIN, STORE_PLAIN>(G, in, out, tw, nullptr, inv, st)));
    SDP_TRY((launch_pass<false, LOAD_PLAIN, STORE_PLAIN>(G, out, out, tw, nullptr, inv, st)));
    return SDP_OK;
}

SDP_EXPORT int sdp_grid_to_image(int G, const sdp_float2 *grid, const float *prolate_ext, sdp_float2 *work,
                                 float *image, void *stream)
{
    SDP_TRY(check_fft_size(G));
    SDP_CHECK_ARG(grid && prolate_ext && work && image, "NULL argument");
    cudaStream_t st = as_stream(stream);
    const float2 *tw = nullptr;
    SDP_TRY(fft_twiddles(G, st, &tw));
    SDP_TRY((launch_pass<true, LOAD_HERMITIAN, STORE_PLAIN>(G, grid, work, tw, nullptr, false, st)));
    SDP_TRY((launch_pass<false, LOAD_PACKED, STORE_REAL_TAPER>(G, work, image, tw, prolate_ext, false, st)));
    return SDP_OK;
}

SDP_EXPORT int sdp_image_to_grid(int G, const float *image, sdp_float2 *work, sdp_float2 *grid, void *stream)
{
    SDP_TRY(check_fft_size(G));
    SDP_CHECK_ARG(image && work && grid, "NULL argument");
    cudaStream_t st = as_stream(stream);
    const float2 *tw = nullptr;
    SDP_TRY(fft_twiddles(G, st, &tw));
    SDP_TRY((launch_pass<true, LOAD_REAL_PAIR, STORE_PAIR>(G, image, work, tw, nullptr, false, st)));
    SDP_TRY((launch_pass<false, LOAD_HALF, STORE_MIRROR>(G, work, grid, tw, nullptr, false, st)));
    return SDP_OK;
}
