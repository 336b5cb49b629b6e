// Tiled GEMM over asynchronous copies: the plain path's kernel for products
// whose operands are stored as the type they are computed in (binary32,
// binary64, and complex of both; binary32 also under the 16-bit precisions).
//
//   D[l,m,n] = op_D(alpha * sum_k A[l,m,k] B[l,k,n] + beta * op_C(C[l,m,n]))
//
// Operands are gathered in place, from any strides. A block (256 threads, 32
// to 256 for the tall tiles) owns a BM x BN tile; per BK-deep slice of the
// contraction every thread copies its share of the two operand tiles with cp.async into a ring of
// STAGES slices, [k][row] in shared memory whatever the operand's own order:
//   - rows contiguous, in 16-byte groups: one 16-byte copy per group;
//   - rows nearest, any alignment: one copy per element, lanes along rows;
//   - contraction nearest: one copy per element, the lanes of a warp on the
//     32-byte runs of several rows, so that whole sectors are read and the
//     transposed writes fall on different banks (row length BM + PAD).
// The offsets of the contracted coordinates come from a table in shared
// memory that all threads refill BATCH slices at a time, BATCH / 2 slices before
// its first use, so no index arithmetic stands between two slices. (The kernel
// before, which loaded through registers and resolved each slice's offsets
// between two barriers, ran 4096^3 binary32 in 3.75 ms: 0.49 of the FMA pipe.)
//
// Arithmetic: binary32 in 8 x 8 register tiles of paired multiply-adds
// (fma.rn.f32x2): a pair of rows meets a pair of columns once straight and
// once swapped, so only the columns' pair is turned and no operand is
// duplicated. Binary64 on the tensor cores' binary64 instruction
// (mma.m8n8k4, IEEE fused multiply-adds, contraction in ascending order): it has the
// CUDA cores' rate (37.1 against 36.4 TFLOP/s measured in registers) but reads a
// quarter of the operand words, which is what bounded the CUDA-core tile.
// Complex operands stay interleaved; conj(B) is computed as
// conj(conj(A) B), so only A's imaginary part takes a sign.
//
// Few tiles and a long contraction: the contraction is split over the blocks
// of a thread-block cluster (2, 4 or 8), whose partial tiles meet through
// distributed shared memory and are added in rank order, each block finishing
// its share of the tile: no workspace and no second launch. Where 8 ranks
// would each still walk more than some 10 slices, the splits go to a workspace
// and k_tile_final adds them in order. Both orders are fixed: a product gives
// the same bits in every run, alone or served.
#include <cstdio>
#include <cstring>
#include <type_traits>

#include "simt.cuh"

namespace tb {
namespace tile {

constexpr int MAXM = 8;        // modes per index class (more: k_simt)
constexpr int BATCH = 4;       // slices per refill of the offset tables

struct Map1 {  // coordinates of one index class -> offset in one operand
    int32_t n, pad;
    FastDiv f[MAXM];
    int64_t s[MAXM];
};
struct Map2 {  // ... -> offsets in C and D
    int32_t n, pad;
    FastDiv f[MAXM];
    int64_t c[MAXM], d[MAXM];
};

enum { COPY_VEC, COPY_PAIR, COPY_ROWS, COPY_K };  // how an operand tile is copied (above)

struct Params {
    const void* A;
    const void* B;
    const void* C;
    void* D;
    void* ws;                // split sums [split][l][m][n], or NULL
    double alpha, beta, alpha_im, beta_im;
    int64_t K, k_chunk;      // k_chunk: contraction length of one split (a multiple of BK)
    uint32_t M, N, L, tiles_m, tiles_n;
    int32_t tC, tD, round_in, beta_zero, conjA, flip, conjC, conjD, conjD_f32;
    int32_t a_copy, b_copy, a_half, b_half;  // *_half: complex elements not aligned to their size
    int32_t d_rows_fast, cluster;
    Map1 am, ak, al, bn, bk, bl;
    Map2 cm, cn, cl;
};

__device__ __forceinline__ int64_t offset1(const Map1& m, uint32_t i)
{
    int64_t o = 0;
    for (int j = 0; j + 1 < m.n; j++) {
        const uint32_t q = fdiv(i, m.f[j]);
        o += (int64_t)(i - q * m.f[j].d) * m.s[j];
        i = q;
    }
    return m.n ? o + (int64_t)i * m.s[m.n - 1] : 0;
}

__device__ __forceinline__ void offset2(const Map2& m, uint32_t i, int64_t& oc, int64_t& od)
{
    oc = od = 0;
    for (int j = 0; j < m.n; j++) {
        const uint32_t q = j + 1 < m.n ? fdiv(i, m.f[j]) : 0;
        const int64_t c = (int64_t)(j + 1 < m.n ? i - q * m.f[j].d : i);
        oc += c * m.c[j];
        od += c * m.d[j];
        i = q;
    }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// copies BYTES to shared memory, or writes zeros there (src is not read then).
// No memory clobber: what is copied is read only after a wait and a barrier,
// and the offset tables may stay in registers across copies.
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const char* src, bool in)
{
    const int n = in ? BYTES : 0;
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(n), "n"(BYTES));
}

// The elements (kk, r) of a ROWS x BK operand slice that thread t copies, each
// call of f covering a group along the rows: f(at(kk), kk, r). Along the rows
// a warp takes whole contracted values, its lanes the groups of rows.
template <int NT, int E, int ROWS, int BK, typename A, typename F>
__device__ __forceinline__ void for_own(int mode, int t, A&& at, F&& f)
{
    constexpr int NW = NT / 32;
    const int w = t >> 5, lane = t & 31;
    auto along_rows = [&](auto n) {
        constexpr int N = decltype(n)::value, G = ROWS / N;  // groups of N rows
        constexpr int LR = G > 16 ? 32 : G > 8 ? 16 : G > 4 ? 8 : G > 2 ? 4 : 2, KP = 32 / LR;
        const int lr = lane % LR, lk = lane / LR;
#pragma unroll
        for (int u = 0; u < (BK + NW * KP - 1) / (NW * KP); u++) {
            const int kk = w * KP + lk + u * NW * KP;
            if (BK % (NW * KP) && kk >= BK) continue;
            const int64_t o = at(kk);
#pragma unroll
            for (int j = 0; j < (G + LR - 1) / LR; j++) {
                const int g = lr + j * LR;
                if (G % LR == 0 || g < G) f(o, kk, g * N);
            }
        }
    };
    if (mode == COPY_VEC) {
        along_rows(std::integral_constant<int, 16 / E>());
    } else if (E == 4 && mode == COPY_PAIR) {
        along_rows(std::integral_constant<int, 2>());
    } else if (mode == COPY_ROWS) {
        along_rows(std::integral_constant<int, 1>());
    } else {
        // KS lanes along the contraction (32 bytes), RS rows per warp
        constexpr int KS = 32 / E, RS = 32 / KS, KB = BK / KS, UNITS = ROWS * BK / 32;
        static_assert(BK % KS == 0 && ROWS % RS == 0, "whole units of a warp");
        const int kl = lane % KS, rl = lane / KS;
#pragma unroll
        for (int u = 0; u < (UNITS + NW - 1) / NW; u++) {
            const int q = w + NW * u, kk = (q % KB) * KS + kl;
            if (UNITS % NW == 0 || q < UNITS) f(at(kk), kk, (q / KB) * RS + rl);
        }
    }
}

// One slice of an operand: rows < rows_in and kk < k_in exist, the rest is
// zero. The tables hold byte offsets, 0 for what does not exist, so that every
// address lies in the operand.
template <int NT, int E, int ROWS, int LD, int BK>
__device__ __forceinline__ void copy_slice(uint32_t dst, const char* base, const int64_t* row, const int64_t* kof,
                                           int rows_in, int k_in, int mode, int half, int t)
{
    auto at = [&](int kk) { return kof[kk]; };
    auto place = [&](int kk, int r) { return dst + (uint32_t)(kk * LD + r) * E; };
    if (mode == COPY_VEC)
        for_own<NT, E, ROWS, BK>(COPY_VEC, t, at, [&](int64_t o, int kk, int r) {
            copy_async<16>(place(kk, r), base + o + row[r], r < rows_in && kk < k_in);
        });
    else if (E == 4 && mode == COPY_PAIR)
        for_own<NT, E, ROWS, BK>(COPY_PAIR, t, at, [&](int64_t o, int kk, int r) {
            copy_async<8>(place(kk, r), base + o + row[r], r < rows_in && kk < k_in);
        });
    else if (E >= 8 && half)  // complex elements aligned to their parts only
        for_own<NT, E, ROWS, BK>(mode, t, at, [&](int64_t o, int kk, int r) {
            const bool in = r < rows_in && kk < k_in;
            copy_async<(E >= 8 ? E / 2 : 4)>(place(kk, r), base + o + row[r], in);
            copy_async<(E >= 8 ? E / 2 : 4)>(place(kk, r) + E / 2, base + o + row[r] + E / 2, in);
        });
    else if (mode == COPY_ROWS)
        for_own<NT, E, ROWS, BK>(COPY_ROWS, t, at, [&](int64_t o, int kk, int r) {
            copy_async<E>(place(kk, r), base + o + row[r], r < rows_in && kk < k_in);
        });
    else
        for_own<NT, E, ROWS, BK>(COPY_K, t, at, [&](int64_t o, int kk, int r) {
            copy_async<E>(place(kk, r), base + o + row[r], r < rows_in && kk < k_in);
        });
}

// ---------------------------------------------------------------------------
// Arithmetic of a tile: acc += A-slice B-slice, and the accumulators written
// to shared memory for the epilogue.

__device__ __forceinline__ void fma_pair(uint64_t& d, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t swapped(uint64_t x)
{
    uint64_t y;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tmov.b64 %0, {hi, lo};\n\t}" : "=l"(y) : "l"(x));
    return y;
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi)
{
    uint64_t y;
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "r"(lo), "r"(hi));
    return y;
}
__device__ __forceinline__ float lo_of(uint64_t x) { return __uint_as_float((uint32_t)x); }
__device__ __forceinline__ float hi_of(uint64_t x) { return __uint_as_float((uint32_t)(x >> 32)); }

// binary32: TM x TN per thread, rows and columns in groups of 4 (columns of 2
// where TN = 2); the lanes of a warp span 8 row and 4 column groups, so that
// a warp's vector reads of A and of B are one 128- and one 64-byte wavefront
template <int BM_, int BN_, int TM, int TN, int MINB_>
struct Real32 {
    using T = float;
    static constexpr bool CPLX = false;
    static constexpr int NT = 256, BM = BM_, BN = BN_, BK = 16, STAGES = 4, E = 4, PAD = 4, MINB = MINB_;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    static constexpr int RT = BM / TM, CT = BN / TN, GN = TN < 4 ? TN : 4;
    static_assert(RT * CT == NT, "one register tile per thread");
    uint64_t acc[TM / 2][TN / 2][2];
    int tr, tc;

    __device__ __forceinline__ void start(int t)
    {
        const int w = t >> 5, lane = t & 31;
        tr = (w % (RT / 8)) * 8 + lane % 8;
        tc = (w / (RT / 8)) * 4 + lane / 8;
#pragma unroll
        for (int i = 0; i < TM / 2; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) acc[i][j][0] = acc[i][j][1] = 0;
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int, int)
    {
        const float* a_at = (const float*)As + tr * 4;
        const float* b_at = (const float*)Bs + tc * GN;
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            uint64_t a[TM / 2], b[TN / 2], bs[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {
                const ulonglong2 q = *(const ulonglong2*)(a_at + kk * LDA + (i / 4) * (RT * 4));
                a[i / 2] = q.x;
                a[i / 2 + 1] = q.y;
            }
#pragma unroll
            for (int j = 0; j < TN; j += GN) {
                if constexpr (GN == 4) {
                    const ulonglong2 q = *(const ulonglong2*)(b_at + kk * LDB + (j / 4) * (CT * 4));
                    b[j / 2] = q.x;
                    b[j / 2 + 1] = q.y;
                } else {
                    b[j / 2] = *(const unsigned long long*)(b_at + kk * LDB);
                }
            }
#pragma unroll
            for (int j = 0; j < TN / 2; j++) bs[j] = swapped(b[j]);
#pragma unroll
            for (int i = 0; i < TM / 2; i++)
#pragma unroll
                for (int j = 0; j < TN / 2; j++) {
                    fma_pair(acc[i][j][0], a[i], b[j]);
                    fma_pair(acc[i][j][1], a[i], bs[j]);
                }
        }
    }
    // put(row, column, value) for every output of the thread
    template <typename F>
    __device__ __forceinline__ void each(int, F&& put)
    {
#pragma unroll
        for (int i = 0; i < TM / 2; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                const int r = (2 * i / 4) * (RT * 4) + tr * 4 + (2 * i) % 4;
                const int c = (2 * j / GN) * (CT * GN) + tc * GN + (2 * j) % GN;
                put(r, c, lo_of(acc[i][j][0]));
                put(r + 1, c + 1, hi_of(acc[i][j][0]));
                put(r, c + 1, lo_of(acc[i][j][1]));
                put(r + 1, c, hi_of(acc[i][j][1]));
            }
    }
};

// complex of binary32: 4 x 4 complex outputs per thread as (re, im) pairs
template <int BM_, int BN_>
struct Complex32 {
    using T = float;
    static constexpr bool CPLX = true;
    static constexpr int NT = 256, BM = BM_, BN = BN_, BK = 16, STAGES = 3, E = 8, PAD = 4, MINB = 2;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    static constexpr int TM = 4, TN = 4, RT = BM / TM, CT = BN / TN;
    static_assert(RT * CT == NT, "one register tile per thread");
    uint64_t acc[TM][TN];
    int tr, tc;

    __device__ __forceinline__ void start(int t)
    {
        const int w = t >> 5, lane = t & 31;
        tr = (w % (RT / 8)) * 8 + lane % 8;
        tc = (w / (RT / 8)) * 4 + lane / 8;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[i][j] = 0;
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int, int conjA)
    {
        const float2* a_at = (const float2*)As + tr * 2;
        const float2* b_at = (const float2*)Bs + tc * 2;
        // the second multiply-add of a product: (re, im) += (-ai, ai) (bi, br),
        // the signs turned for conj(A)
        const uint32_t s_re = conjA ? 0u : 0x80000000u, s_im = conjA ? 0x80000000u : 0u;
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            uint64_t ar[TM], ai[TM], b[TN], bs[TN];
#pragma unroll
            for (int i = 0; i < TM; i += 2) {
                const float4 q = *(const float4*)(a_at + kk * LDA + (i / 2) * (RT * 2));
                const uint32_t x = __float_as_uint(q.x), y = __float_as_uint(q.y), z = __float_as_uint(q.z),
                               w = __float_as_uint(q.w);
                ar[i] = pack2(x, x);
                ar[i + 1] = pack2(z, z);
                ai[i] = pack2(y ^ s_re, y ^ s_im);
                ai[i + 1] = pack2(w ^ s_re, w ^ s_im);
            }
#pragma unroll
            for (int j = 0; j < TN; j += 2) {
                const ulonglong2 q = *(const ulonglong2*)(b_at + kk * LDB + (j / 2) * (CT * 2));
                b[j] = q.x;
                b[j + 1] = q.y;
                bs[j] = swapped(q.x);
                bs[j + 1] = swapped(q.y);
            }
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    fma_pair(acc[i][j], ar[i], b[j]);
                    fma_pair(acc[i][j], ai[i], bs[j]);
                }
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(int flip, F&& put)
    {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) {
                const float im = hi_of(acc[i][j]);
                put((i / 2) * (RT * 2) + tr * 2 + i % 2, (j / 2) * (CT * 2) + tc * 2 + j % 2,
                    make_float2(lo_of(acc[i][j]), flip ? -im : im));
            }
    }
};

// The tall tiles of products with few columns (mode-n products with a small
// rank), where the multiply-adds and the load path matter as much as in the
// wide tile: a warp owns one group of TN columns, its lanes 8 rows each (two
// groups of 4), so a register tile costs 8 + TN words of shared memory for 8
// TN multiply-adds; BN is the column count rounded up to groups of 8 or 12.
template <int CT, int TN>
struct Slim32 {
    using T = float;
    static constexpr bool CPLX = false;
    static constexpr int NT = 32 * CT, BM = 256, BN = CT * TN, BK = 8, STAGES = 4, E = 4, PAD = 4;
    static constexpr int MINB = NT <= 96 ? 4 : NT <= 160 ? 3 : 2;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    uint64_t acc[4][TN / 2][2];
    int row, col;

    __device__ __forceinline__ void start(int t)
    {
        row = (t & 31) * 4;
        col = (t >> 5) * TN;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) acc[i][j][0] = acc[i][j][1] = 0;
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int kn, int)
    {
        const float* a_at = (const float*)As + row;
        const float* b_at = (const float*)Bs + col;
#pragma unroll 4
        for (int kk = 0; kk < kn; kk++) {
            uint64_t a[4], as[4], b[TN / 2];
            const ulonglong2 q0 = *(const ulonglong2*)(a_at + kk * LDA), q1 = *(const ulonglong2*)(a_at + kk * LDA + 128);
            a[0] = q0.x;
            a[1] = q0.y;
            a[2] = q1.x;
            a[3] = q1.y;
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const ulonglong2 q = *(const ulonglong2*)(b_at + kk * LDB + j);
                b[j / 2] = q.x;
                b[j / 2 + 1] = q.y;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) as[i] = swapped(a[i]);
#pragma unroll
            for (int j = 0; j < TN / 2; j++)
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int i = h ? 3 - u : u;
                        fma_pair(acc[i][j][h], h ? as[i] : a[i], b[j]);
                    }
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(int, F&& put)
    {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < TN / 2; j++) {
                const int r = row + (i / 2) * 128 + (i % 2) * 2, c = col + 2 * j;
                put(r, c, lo_of(acc[i][j][0]));
                put(r + 1, c + 1, hi_of(acc[i][j][0]));
                put(r + 1, c, lo_of(acc[i][j][1]));
                put(r, c + 1, hi_of(acc[i][j][1]));
            }
    }
};

// ... of complex binary32: 4 rows (two groups of 2) and 8 columns a thread
template <int CT>
struct SlimComplex32 {
    using T = float;
    static constexpr bool CPLX = true;
    static constexpr int NT = 32 * CT, BM = 128, BN = CT * 8, BK = 8, STAGES = 4, E = 8, PAD = 4;
    static constexpr int MINB = NT <= 96 ? 4 : 2;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    uint64_t acc[4][8];
    int row, col;

    __device__ __forceinline__ void start(int t)
    {
        row = (t & 31) * 2;
        col = (t >> 5) * 8;
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = 0;
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int kn, int conjA)
    {
        const float2* a_at = (const float2*)As + row;
        const float2* b_at = (const float2*)Bs + col;
        const uint32_t s_re = conjA ? 0u : 0x80000000u, s_im = conjA ? 0x80000000u : 0u;
#pragma unroll 2
        for (int kk = 0; kk < kn; kk++) {
            uint64_t ar[4], ai[4];
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const float4 q = *(const float4*)(a_at + kk * LDA + (i / 2) * 64);
                const uint32_t x = __float_as_uint(q.x), y = __float_as_uint(q.y), z = __float_as_uint(q.z),
                               w = __float_as_uint(q.w);
                ar[i] = pack2(x, x);
                ar[i + 1] = pack2(z, z);
                ai[i] = pack2(y ^ s_re, y ^ s_im);
                ai[i + 1] = pack2(w ^ s_re, w ^ s_im);
            }
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const ulonglong2 q = *(const ulonglong2*)(b_at + kk * LDB + j);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint64_t b = h ? q.y : q.x, bs = swapped(b);
#pragma unroll
                    for (int i = 0; i < 4; i++) fma_pair(acc[i][j + h], ar[i], b);
#pragma unroll
                    for (int i = 0; i < 4; i++) fma_pair(acc[3 - i][j + h], ai[3 - i], bs);
                }
            }
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(int flip, F&& put)
    {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float im = hi_of(acc[i][j]);
                put(row + (i / 2) * 64 + i % 2, col + j, make_float2(lo_of(acc[i][j]), flip ? -im : im));
            }
    }
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// binary64: WGM x WGN warps, each a grid of 8 x 8 fragments; a lane reads
// A[row lane/4][k lane%4] and B[k lane%4][column lane/4]. Rows of BM + 4
// words put the 16 lanes of a half-warp on different banks.
template <int BM_, int BN_, int WGM, int WGN, int MINB_>
struct Real64 {
    using T = double;
    static constexpr bool CPLX = false;
    static constexpr int NT = 256, BM = BM_, BN = BN_, BK = 16, STAGES = 3, E = 8, PAD = 4, MINB = MINB_;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    static constexpr int WM = BM / WGM, WN = BN / WGN, FM = WM / 8, FN = WN / 8;
    static_assert(WGM * WGN * 32 == NT, "8 warps");
    double acc[FM][FN][2];
    int g, q, wm, wn;

    __device__ __forceinline__ void start(int t)
    {
        const int w = t >> 5, lane = t & 31;
        g = lane >> 2;
        q = lane & 3;
        wm = (w % WGM) * WM;
        wn = (w / WGM) * WN;
#pragma unroll
        for (int i = 0; i < FM; i++)
#pragma unroll
            for (int j = 0; j < FN; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int, int)
    {
        const double* a_at = (const double*)As + q * LDA + wm + g;
        const double* b_at = (const double*)Bs + q * LDB + wn + g;
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; k4++) {
            double a[FM], b[FN];
#pragma unroll
            for (int i = 0; i < FM; i++) a[i] = a_at[k4 * 4 * LDA + i * 8];
#pragma unroll
            for (int j = 0; j < FN; j++) b[j] = b_at[k4 * 4 * LDB + j * 8];
#pragma unroll
            for (int i = 0; i < FM; i++)
#pragma unroll
                for (int j = 0; j < FN; j++) mma_f64(acc[i][j], a[i], b[j]);
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(int, F&& put)
    {
#pragma unroll
        for (int i = 0; i < FM; i++)
#pragma unroll
            for (int j = 0; j < FN; j++) {
                put(wm + i * 8 + g, wn + j * 8 + 2 * q, acc[i][j][0]);
                put(wm + i * 8 + g, wn + j * 8 + 2 * q + 1, acc[i][j][1]);
            }
    }
};

// complex of binary64: the same fragments, real and imaginary parts read
// together (rows of BM + 2 words of 16 bytes: 8 lanes on different banks)
template <int BM_, int BN_, int WGM, int WGN>
struct Complex64 {
    using T = double;
    static constexpr bool CPLX = true;
    static constexpr int NT = 256, BM = BM_, BN = BN_, BK = 16, STAGES = 3, E = 16, PAD = 2, MINB = 2;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    static constexpr int WM = BM / WGM, WN = BN / WGN, FM = WM / 8, FN = WN / 8;
    static_assert(WGM * WGN * 32 == NT, "8 warps");
    double re[FM][FN][2], im[FM][FN][2];
    int g, q, wm, wn;

    __device__ __forceinline__ void start(int t)
    {
        const int w = t >> 5, lane = t & 31;
        g = lane >> 2;
        q = lane & 3;
        wm = (w % WGM) * WM;
        wn = (w / WGM) * WN;
#pragma unroll
        for (int i = 0; i < FM; i++)
#pragma unroll
            for (int j = 0; j < FN; j++) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
    }
    static __device__ __forceinline__ double signed_by(double x, uint64_t s)
    {
        return __longlong_as_double(__double_as_longlong(x) ^ (long long)s);
    }
    __device__ __forceinline__ void slice(const char* As, const char* Bs, int, int conjA)
    {
        const double2* a_at = (const double2*)As + q * LDA + wm + g;
        const double2* b_at = (const double2*)Bs + q * LDB + wn + g;
        const uint64_t top = 0x8000000000000000ull, s_re = conjA ? 0 : top, s_im = conjA ? top : 0;
#pragma unroll
        for (int k4 = 0; k4 < BK / 4; k4++) {
            double2 a[FM], b[FN];
#pragma unroll
            for (int i = 0; i < FM; i++) a[i] = a_at[k4 * 4 * LDA + i * 8];
#pragma unroll
            for (int j = 0; j < FN; j++) b[j] = b_at[k4 * 4 * LDB + j * 8];
#pragma unroll
            for (int i = 0; i < FM; i++) {
                const double minus = signed_by(a[i].y, s_re), plus = signed_by(a[i].y, s_im);
#pragma unroll
                for (int j = 0; j < FN; j++) {
                    mma_f64(re[i][j], a[i].x, b[j].x);
                    mma_f64(im[i][j], a[i].x, b[j].y);
                }
#pragma unroll
                for (int j = 0; j < FN; j++) {
                    mma_f64(re[i][j], minus, b[j].y);
                    mma_f64(im[i][j], plus, b[j].x);
                }
            }
        }
    }
    template <typename F>
    __device__ __forceinline__ void each(int flip, F&& put)
    {
#pragma unroll
        for (int i = 0; i < FM; i++)
#pragma unroll
            for (int j = 0; j < FN; j++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    put(wm + i * 8 + g, wn + j * 8 + 2 * q + h,
                        make_double2(re[i][j][h], flip ? -im[i][j][h] : im[i][j][h]));
    }
};

// ---------------------------------------------------------------------------

template <typename T, bool CPLX>
struct Value;
template <typename T>
struct Value<T, false> { using V = T; static __device__ T re(T v) { return v; } static __device__ T im(T) { return 0; }
                         static __device__ T sum(T a, T b) { return a + b; } };
template <>
struct Value<float, true> { using V = float2; static __device__ float re(float2 v) { return v.x; } static __device__ float im(float2 v) { return v.y; }
                            static __device__ float2 sum(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); } };
template <>
struct Value<double, true> { using V = double2; static __device__ double re(double2 v) { return v.x; } static __device__ double im(double2 v) { return v.y; }
                             static __device__ double2 sum(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); } };

template <class W>
struct Layout {  // shared memory of a block
    static constexpr int STAGE = W::BK * (W::LDA + W::LDB) * W::E;
    static constexpr int KT = BATCH * W::BK;
    // the finished tile, D's contiguous side fastest, padded like the slices
    static constexpr int TILE_R = W::BN * (W::BM + W::PAD) * W::E, TILE_C = W::BM * (W::BN + W::PAD) * W::E;
    static constexpr int RING = STAGE * W::STAGES;
    static constexpr int BODY = RING > TILE_R ? (RING > TILE_C ? RING : TILE_C) : (TILE_R > TILE_C ? TILE_R : TILE_C);
    static constexpr int BYTES = BODY + 8 * (3 * W::BM + 3 * W::BN + 4 * KT);
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the value at shared-memory address `at` of block `rank` of the cluster
__device__ __forceinline__ uint32_t remote(uint32_t at, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(rank));
    return r;
}
__device__ __forceinline__ void load_remote(uint32_t a, float& v)
{
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ void load_remote(uint32_t a, double& v)
{
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
__device__ __forceinline__ void load_remote(uint32_t a, float2& v)
{
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
}
__device__ __forceinline__ void load_remote(uint32_t a, double2& v)
{
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
}

// RND: binary32 operands rounded to the precision's 16-bit format, by the
// thread that copied them, once their slice has landed
template <class W, bool RND>
__global__ void __launch_bounds__(W::NT, W::MINB) k_tile(const __grid_constant__ Params p)
{
    using T = typename W::T;
    using VT = Value<T, W::CPLX>;
    using V = typename VT::V;
    using S = Layout<W>;
    constexpr int NT = W::NT, BM = W::BM, BN = W::BN, BK = W::BK, STAGES = W::STAGES, E = W::E, KT = S::KT;
    extern __shared__ __align__(16) char smem[];
    int64_t* aRow = (int64_t*)(smem + S::BODY);
    int64_t* bRow = aRow + BM;
    int64_t* kA = bRow + BN;       // [2][KT]
    int64_t* kB = kA + 2 * KT;
    // offsets in C (x) and D (y) of the tile's rows and columns
    longlong2* rowCD = (longlong2*)(kB + 2 * KT);
    longlong2* colCD = rowCD + BM;

    const int t = threadIdx.x;
    // neighbouring blocks share a row panel of A (the longer operand)
    const uint32_t tn = blockIdx.x % p.tiles_n, rest = blockIdx.x / p.tiles_n;
    const uint32_t tm = rest % p.tiles_m, l = rest / p.tiles_m;
    const uint32_t m0 = tm * BM, n0 = tn * BN;
    const int rows_a = p.M - m0 < BM ? (int)(p.M - m0) : BM, rows_b = p.N - n0 < BN ? (int)(p.N - n0) : BN;
    const int64_t kbeg = (int64_t)blockIdx.y * p.k_chunk;
    const int64_t kend = kbeg + p.k_chunk < p.K ? kbeg + p.k_chunk : p.K;
    const int slices = kend > kbeg ? (int)((kend - kbeg + BK - 1) / BK) : 0;

    auto fill_offsets = [&](int batch) {
        const int64_t k0 = kbeg + (int64_t)batch * KT;
        const int at = (batch & 1) * KT;
        for (int i = t; i < 2 * KT; i += NT) {
            const int64_t k = k0 + i % KT;
            (i < KT ? kA : kB - KT)[at + i] = k < kend ? E * offset1(i < KT ? p.ak : p.bk, (uint32_t)k) : 0;
        }
    };
    for (int i = t; i < BM + BN; i += NT) {
        if (i < BM) aRow[i] = i < rows_a ? E * (offset1(p.al, l) + offset1(p.am, m0 + i)) : 0;
        else bRow[i - BM] = i - BM < rows_b ? E * (offset1(p.bl, l) + offset1(p.bn, n0 + i - BM)) : 0;
    }
    static_assert(STAGES <= BATCH, "the first slices lie in the first refill");
    fill_offsets(0);
    fill_offsets(1);
    __syncthreads();

    const uint32_t ring = smem_addr(smem);
    auto issue = [&](int s) {
        if (s < slices) {
            const uint32_t dst = ring + (uint32_t)(s % STAGES) * S::STAGE;
            const int at = ((s / BATCH) & 1) * KT + (s % BATCH) * BK;
            const int64_t left = kend - kbeg - (int64_t)s * BK;
            const int k_in = left < BK ? (int)left : BK;
            copy_slice<NT, E, BM, W::LDA, BK>(dst, (const char*)p.A, aRow, kA + at, rows_a, k_in, p.a_copy, p.a_half, t);
            copy_slice<NT, E, BN, W::LDB, BK>(dst + BK * W::LDA * E, (const char*)p.B, bRow, kB + at, rows_b, k_in, p.b_copy,
                                          p.b_half, t);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    W w;
    w.start(t);
    // the first STAGES - 1 steps only copy (one place in the code issues copies)
#pragma unroll 1
    for (int s = 1 - STAGES; s < slices; s++) {
        const int q = s + STAGES - 1;
        if (s == -1) {
            // the offsets of C and D, while the first slices are on their way
            for (int i = t; i < BM + BN; i += NT) {
                int64_t oc = 0, od = 0, lc = 0, ld = 0;
                if (i < BM) {
                    if (i < rows_a) {
                        offset2(p.cl, l, lc, ld);
                        offset2(p.cm, m0 + i, oc, od);
                    }
                    rowCD[i] = make_longlong2(oc + lc, od + ld);
                } else {
                    if (i - BM < rows_b) offset2(p.cn, n0 + i - BM, oc, od);
                    colCD[i - BM] = make_longlong2(oc, od);
                }
            }
        }
        if (s >= 0) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        char* As = smem + ((s + STAGES) % STAGES) * S::STAGE;
        char* Bs = As + BK * W::LDA * E;
        if (RND && s >= 0) {
            auto round_own = [&](char* base, int ld, int mode) {
                return [=](int64_t, int kk, int r) {
                    float* x = (float*)base + kk * ld + r;
                    if (mode == COPY_VEC) {
                        float4 v = *(float4*)x;
                        v.x = round_in<float>(v.x, p.round_in);
                        v.y = round_in<float>(v.y, p.round_in);
                        v.z = round_in<float>(v.z, p.round_in);
                        v.w = round_in<float>(v.w, p.round_in);
                        *(float4*)x = v;
                    } else if (mode == COPY_PAIR) {
                        float2 v = *(float2*)x;
                        v.x = round_in<float>(v.x, p.round_in);
                        v.y = round_in<float>(v.y, p.round_in);
                        *(float2*)x = v;
                    } else {
                        *x = round_in<float>(*x, p.round_in);
                    }
                };
            };
            auto none = [](int) { return (int64_t)0; };
            for_own<NT, E, BM, BK>(p.a_copy, t, none, round_own(As, W::LDA, p.a_copy));
            for_own<NT, E, BN, BK>(p.b_copy, t, none, round_own(Bs, W::LDB, p.b_copy));
        }
        if (s >= 0) __syncthreads();  // slice s has landed; slice s - 1 has been read by all
        if (s >= 0 && q % BATCH == BATCH / 2 && (q / BATCH + 1) * BATCH < slices) fill_offsets(q / BATCH + 1);
        issue(q);
        if (s < 0) continue;
        const int64_t left = kend - kbeg - (int64_t)s * BK;
        w.slice(As, Bs, left < BK ? (int)left : BK, p.conjA);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // the tile to shared memory, D's contiguous side fastest
    V* tile = (V*)smem;
    const bool by_rows = p.d_rows_fast && !p.ws;
    const int sr = by_rows ? 1 : BN + W::PAD, sc = by_rows ? BM + W::PAD : 1;
    w.each(p.flip, [&](int r, int c, V v) { tile[r * sr + c * sc] = v; });
    const int ranks = p.cluster;
    if (ranks > 1) cluster_barrier();
    else __syncthreads();
    static_assert(BM * BN % 8 == 0, "equal shares of a tile for 2, 4 and 8 ranks");
    const int share = BM * BN / ranks, first = ranks > 1 ? (int)blockIdx.y * share : 0;
    // the sum of the ranks' partial results for output (r, c), in rank order
    auto summed = [&](int r, int c) {
        const int at = r * sr + c * sc;
        if (ranks == 1) return tile[at];
        const uint32_t a = ring + (uint32_t)(at * (int)sizeof(V));
        V x[8];  // the ranks' loads in flight together
#pragma unroll
        for (int z = 0; z < 8; z++)
            if (z < ranks) load_remote(remote(a, z), x[z]);
#pragma unroll
        for (int z = 1; z < 8; z++)
            if (z < ranks) x[0] = VT::sum(x[0], x[z]);
        return x[0];
    };
    auto place = [&](int e, int& r, int& c) {
        r = by_rows ? e % BM : e / BN;
        c = by_rows ? e / BM : e % BN;
        return e < first + share && r < rows_a && c < rows_b;
    };
    constexpr int STORED = W::CPLX ? (sizeof(T) == 4 ? T_C32 : T_C64) : (sizeof(T) == 4 ? T_F32 : T_F64);
    if (p.ws) {
        for (int e = first + t; e < first + share; e += NT) {
            int r, c;
            if (place(e, r, c))
                ((V*)p.ws)[(((int64_t)blockIdx.y * p.L + l) * p.M + m0 + r) * p.N + n0 + c] = summed(r, c);
        }
    } else if (p.tC == STORED && p.tD == STORED) {
        // C and D as they are computed. A warp takes lines of the tile along
        // D's contiguous side (32 outputs a step), so the line's offsets are
        // read once and a lane keeps those of its places: some 12 instructions
        // an output, where one index decoded per output took 60 and made half
        // of a small product's time. (And no code per storage type, unrolled:
        // it missed the instruction cache on each tile.)
        auto lines = [&](auto rows_fast) {
            constexpr bool RF = decltype(rows_fast)::value;
            constexpr int IN = RF ? BM : BN, OUT = RF ? BN : BM, IT = (IN + 31) / 32, NW = NT / 32;
            constexpr int OU = IT >= 8 || (IT >= 4 && sizeof(V) > 4) ? 1 : (sizeof(V) == 16 ? 4 : 8) / IT;  // lines at a time
            constexpr int Q = W::CPLX ? 2 : 1;
            const longlong2* inner = RF ? rowCD : colCD;
            const longlong2* outer = RF ? colCD : rowCD;
            const int n_in = RF ? rows_a : rows_b, n_out = RF ? rows_b : rows_a;
            const int o0 = ranks > 1 ? (int)blockIdx.y * (OUT / ranks) : 0;
            // the last rank finishes what the ranks' equal shares leave (a width of 12 has no eighths)
            const int o1 = min(n_out, ranks > 1 && (int)blockIdx.y + 1 < ranks ? o0 + OUT / ranks : OUT);
            const int lane = t & 31;
            int64_t ic[IT], id[IT];
#pragma unroll
            for (int i = 0; i < IT; i++) {
                const longlong2 q = lane + 32 * i < n_in ? inner[lane + 32 * i] : make_longlong2(0, 0);
                ic[i] = Q * q.x;
                id[i] = Q * q.y;
            }
#pragma unroll 1
            for (int o = o0 + (t >> 5); o < o1; o += NW * OU) {
                T cr[OU][IT], ci[OU][IT];
#pragma unroll
                for (int v = 0; v < OU; v++) {
                    const T* C = (const T*)p.C + Q * (o + v * NW < o1 ? outer[o + v * NW].x : 0);
#pragma unroll
                    for (int i = 0; i < IT; i++) {
                        cr[v][i] = ci[v][i] = 0;
                        if (p.beta_zero || o + v * NW >= o1 || lane + 32 * i >= n_in) continue;
                        cr[v][i] = C[ic[i]];
                        if (W::CPLX) ci[v][i] = C[ic[i] + Q - 1];
                    }
                }
#pragma unroll
                for (int v = 0; v < OU; v++) {
                    if (o + v * NW >= o1) break;
                    T* D = (T*)p.D + Q * outer[o + v * NW].y;
#pragma unroll
                    for (int i = 0; i < IT; i++) {
                        const int at = lane + 32 * i;
                        if (at >= n_in) continue;
                        const V x = RF ? summed(at, o + v * NW) : summed(o + v * NW, at);
                        T c = cr[v][i], vr, vi;
                        if (RND) c = round_in<T>(c, p.round_in);
                        simt::epilogue_value<T, W::CPLX, Params>(p, VT::re(x), VT::im(x), c, ci[v][i], vr, vi);
                        D[id[i]] = vr;
                        if (W::CPLX) D[id[i] + Q - 1] = vi;
                    }
                }
            }
        };
        if (by_rows) lines(std::true_type());
        else lines(std::false_type());
    } else {
#pragma unroll 1
        for (int e = first + t; e < first + share; e += NT) {
            int r, c;
            if (!place(e, r, c)) continue;
            const V x = summed(r, c);
            T cr = 0, ci = 0, vr, vi;
            if (!p.beta_zero) load_rounded<T>(p.C, rowCD[r].x + colCD[c].x, p.tC, p.round_in, cr, ci);
            simt::epilogue_value<T, W::CPLX, Params>(p, VT::re(x), VT::im(x), cr, ci, vr, vi);
            store_elem<T>(p.D, rowCD[r].y + colCD[c].y, p.tD, vr, vi);
        }
    }
    if (ranks > 1) cluster_barrier();  // no block leaves while its tile may be read
}

// adds the splits of every element of D in split order, then the epilogue (a
// split product has fewer than 148 tiles, so its outputs count in 32 bits)
template <typename T, bool CPLX>
__global__ void __launch_bounds__(256) k_tile_final(const __grid_constant__ Params p, int splits, FastDiv fn, FastDiv fm)
{
    using VT = Value<T, CPLX>;
    using V = typename VT::V;
    const V* w = (const V*)p.ws;
    const int64_t total = (int64_t)p.L * p.M * p.N;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t row = fdiv((uint32_t)e, fn), n = (uint32_t)e - row * fn.d;
        const uint32_t l = fdiv(row, fm), m = row - l * fm.d;
        V x = w[e];
        for (int z = 1; z < splits; z++) x = VT::sum(x, w[z * total + e]);
        int64_t cm, dm, cn, dn, cl, dl;
        offset2(p.cm, m, cm, dm);
        offset2(p.cn, n, cn, dn);
        offset2(p.cl, l, cl, dl);
        T cr = 0, ci = 0, vr, vi;
        if (!p.beta_zero) load_rounded<T>(p.C, cm + cn + cl, p.tC, p.round_in, cr, ci);
        simt::epilogue_value<T, CPLX, Params>(p, VT::re(x), VT::im(x), cr, ci, vr, vi);
        store_elem<T>(p.D, dm + dn + dl, p.tD, vr, vi);
    }
}

// ---------------------------------------------------------------------------
// host side

static void map1(Map1& m, const simt::Modes& s)
{
    m.n = s.n;
    for (int j = 0; j < s.n; j++) {
        m.f[j] = make_fastdiv((uint32_t)s.ext[j]);
        m.s[j] = s.s0[j];
    }
}
static void map2(Map2& m, const simt::Modes& s)
{
    m.n = s.n;
    for (int j = 0; j < s.n; j++) {
        m.f[j] = make_fastdiv((uint32_t)s.ext[j]);
        m.c[j] = s.s0[j];
        m.d[j] = s.s1[j];
    }
}

// Whether groups of w neighbouring rows (or contracted values) are `bytes`
// aligned bytes: their first mode has stride 1 and an extent divisible by w, and every other stride
// and the base keep the alignment.
static bool rows_in_groups(const simt::Modes& rows, const simt::Modes& ks, const simt::Modes& ls, const void* base, int w,
                           int bytes)
{
    if ((uintptr_t)base % (unsigned)bytes || rows.n < 1 || rows.s0[0] != 1 || rows.ext[0] % w) return false;
    for (int j = 1; j < rows.n; j++)
        if (rows.s0[j] % w) return false;
    for (int j = 0; j < ks.n; j++)
        if (ks.s0[j] % w) return false;
    for (int j = 0; j < ls.n; j++)
        if (ls.s0[j] % w) return false;
    return true;
}

struct Split {
    int cluster;   // blocks of a cluster that share a tile's contraction, or 1
    int splits;    // splits through the workspace, or 1
    int64_t chunk;
    size_t ws_bytes;
};

// About two blocks per SM in all; products of 148 tiles and more are not split,
// but for those of up to one and a half tiles per SM and more than 32 slices, in
// which half the SMs would wait for a second whole tile (160 tiles, 2909 terms 259
// / 213 us in two ranks; with 64 to 130 terms 0.74 to 0.96 of the speed). A split keeps at least two slices of the
// contraction (less would spend more on the meeting of the ranks than on the
// sums); a cluster serves up to 8, beyond that the workspace and its second
// launch pay once every one of 8 ranks would walk more than 11 slices (binary32),
// 10 (binary64, complex) or 8 (complex binary64). 8 ranks / workspace, us: binary32
// 1384 terms 16.6 / 17.8, 1660 terms 16.3 / 13.4; complex 1029 terms 38.5 / 42.9, 1338
// terms 29.2 / 18.4; binary64 1262 terms 12.1 / 12.9, 1329 terms 17.4 / 13.7; complex
// binary64 570 terms 23 / 21, 1811 terms 57.6 / 29.7; 16 slices where fewer than 16
// splits fill the GPU (32 tiles, 1651 terms 26.3 / 33.4). ws_limit: the scratch a
// product is charged for by a server (simt_scratch_bytes), which the workspace
// stays within.
static Split choose_split(int64_t tiles, int64_t K, int bk, int64_t outs, size_t elem, size_t ws_limit)
{
    Split r = {1, 1, K, 0};
    const int64_t slices = (K + bk - 1) / bk;
    r.chunk = slices * bk;
    if (tiles >= 222 || (tiles >= 148 && slices <= 32) || slices < 4) return r;
    const int64_t want = (2 * 148 + tiles - 1) / tiles;
    const int most = want < 16 ? 16 : elem == 4 ? 11 : elem == 8 ? 10 : 8;
    if (want > 8 && slices > 8 * most) {
        int64_t S = want < slices / 4 ? want : slices / 4;
        if (S > 1024) S = 1024;
        while (S > 1 && (double)S * (double)outs * (double)elem > (double)ws_limit) S /= 2;
        if (S > 8) {
            const int64_t per = (slices + S - 1) / S;
            r.chunk = per * bk;
            r.splits = (int)((slices + per - 1) / per);
            r.ws_bytes = (size_t)r.splits * (size_t)outs * elem;
            return r;
        }
    }
    int cs = 1;
    while (cs < 8 && cs < want && 2 * (2 * cs) <= slices) cs *= 2;
    r.cluster = cs;
    r.chunk = (slices + cs - 1) / cs * bk;
    return r;
}

template <class W, bool RND>
static cudaError_t launch(const simt::Params& sp, size_t ws_limit, cudaStream_t s)
{
    Params p;
    memset(&p, 0, sizeof(p));
    p.A = sp.A;
    p.B = sp.B;
    p.C = sp.C;
    p.D = sp.D;
    p.alpha = sp.alpha;
    p.beta = sp.beta;
    p.alpha_im = sp.alpha_im;
    p.beta_im = sp.beta_im;
    p.K = sp.K;
    p.M = (uint32_t)sp.M;
    p.N = (uint32_t)sp.N;
    p.L = (uint32_t)sp.L;
    p.tC = sp.tC;
    p.tD = sp.tD;
    p.round_in = sp.round_in;
    p.beta_zero = sp.beta_zero;
    p.conjA = (sp.conjA != 0) != (sp.conjB != 0);
    p.flip = sp.conjB;
    p.conjC = sp.conjC;
    p.conjD = sp.conjD;
    p.conjD_f32 = sp.conjD_f32;
    p.d_rows_fast = sp.d_rows_fast;
    auto copy_form = [](bool rows_fast, const simt::Modes& rows, const simt::Modes& ks, const simt::Modes& ls, const void* base) {
        if (!rows_fast) return (int)COPY_K;
        if (rows_in_groups(rows, ks, ls, base, 16 / W::E, 16)) return (int)COPY_VEC;
        return (int)(W::E == 4 && rows_in_groups(rows, ks, ls, base, 2, 8) ? COPY_PAIR : COPY_ROWS);
    };
    p.a_copy = copy_form(sp.a_rows_fast, sp.am, sp.ak, sp.al, sp.A);
    p.b_copy = copy_form(sp.b_rows_fast, sp.bn, sp.bk, sp.bl, sp.B);
    p.a_half = W::CPLX && (uintptr_t)sp.A % W::E != 0;
    p.b_half = W::CPLX && (uintptr_t)sp.B % W::E != 0;
    map1(p.am, sp.am);
    map1(p.ak, sp.ak);
    map1(p.al, sp.al);
    map1(p.bn, sp.bn);
    map1(p.bk, sp.bk);
    map1(p.bl, sp.bl);
    map2(p.cm, sp.cm);
    map2(p.cn, sp.cn);
    map2(p.cl, sp.cl);
    p.tiles_m = (p.M + W::BM - 1) / W::BM;
    p.tiles_n = (p.N + W::BN - 1) / W::BN;
    const int64_t blocks = (int64_t)p.tiles_m * p.tiles_n * sp.L;
    if (blocks <= 0 || blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
    const Split split = choose_split(blocks, sp.K, W::BK, sp.L * sp.M * sp.N, W::E, ws_limit);
    p.k_chunk = split.chunk;
    p.cluster = split.cluster;

    constexpr int smem = Layout<W>::BYTES;
    static int attr_done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_tile<W, RND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = 1;
    }
    if (split.splits > 1) {
        cudaError_t e = pool_alloc(&p.ws, split.ws_bytes, s);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks, (unsigned)(split.splits > 1 ? split.splits : split.cluster));
    cfg.blockDim = dim3(W::NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = (unsigned)split.cluster;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = split.cluster > 1 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_tile<W, RND>, p);
    count_launch();
    if (split.splits > 1) {
        if (e == cudaSuccess) {
            const int64_t total = sp.L * sp.M * sp.N;
            int64_t g = (total + 255) / 256;
            if (g > 148 * 16) g = 148 * 16;
            k_tile_final<typename W::T, W::CPLX>
                <<<(unsigned)g, 256, 0, s>>>(p, split.splits, make_fastdiv(p.N), make_fastdiv(p.M));
            count_launch();
            e = cudaGetLastError();
        }
        cudaFreeAsync(p.ws, s);
    }
    return e;
}

// Tiles by the shorter side N. Wide ones where both sides fill them (binary64
// 128 x 64, two blocks per SM with 32 accumulators a thread, or 64 x 64 where M
// is small; binary32 128 x 128 with two tiles per SM and, shared by the ranks of
// a cluster, with fewer where the contraction is long, sooner if operands lie
// along it: a 64 x 64 tile reads twice the shared memory per multiply-add and
// copies transposing, element by element, twice as often. 64 x 64 / 128 x 128,
// us: 634 x 480 x 2832 126 / 77, 817 x 1168 x 1972 in 2 batches, both operands along
// the contraction, 411 / 290; mean of 350 products 1.1 to 1.4 times from the lines
// on, 0.5 to 1.1 below them and with fewer than 16 tiles), 128 rows of 8 to 64 columns for narrow products, and for binary32 and its
// complex tall tiles as wide as N rounded up to 8 or 12, whose warps own a group
// of columns each.
// A block of those has only as many warps as groups, so they need rows for
// several warps per SM: with fewer, one or two warps an SM wait on every slice
// (57771 x 2 x 383 165 us, 76 in 128 x 16 tiles). Time in the general tile / in
// the tall one, 1600 random products: binary32 up to 48 columns 0.3 to 0.8
// below 4 warps an SM, about 1 at 5, 1.0 to 2.1 from 6 on; 49 to 60 columns 0.6 to
// 1.0 everywhere (no tall tile), 61 to 64 0.5 to 1.0 below 10 warps, 0.9 to 1.5
// above. Complex up to 16 columns 0.6 to 1.0 below 2 and 3 warps an SM, 1.1 to 1.4 above,
// 17 to 24 columns 1.02 to 1.10 from 24 on, 41 to 48 1.05 to 1.18 from 32 on where
// A lies along the contraction (0.8 to 0.97 else), other widths 0.7 to 1.0.
template <typename F>
static auto with_tile(const simt::Params& p, int compute, F&& f)
{
    const int w8 = (int)((p.N + 7) / 8);
    // whether full blocks of `rows` rows and `warps` warps put `per_sm` warps on every SM
    auto fills = [&](int rows, int warps, int per_sm) {
        return (double)p.M * (double)p.L * warps >= 148.0 * per_sm * rows;
    };
    switch (compute) {
    case TB_R64:
        if (p.N > 64) {
            if (p.M <= 64) return f(Real64<64, 64, 2, 4, 2>());
            return f(Real64<128, 64, 4, 2, 2>());
        }
        switch (w8) {
        case 1: return f(Real64<128, 8, 8, 1, 2>());
        case 2: return f(Real64<128, 16, 8, 1, 2>());
        case 3: return f(Real64<128, 24, 8, 1, 2>());
        case 4: return f(Real64<128, 32, 8, 1, 2>());
        case 5: return f(Real64<128, 40, 8, 1, 2>());
        case 6: return f(Real64<128, 48, 8, 1, 2>());
        case 7: return f(Real64<128, 56, 8, 1, 2>());
        default: return f(Real64<128, 64, 4, 2, 2>());
        }
    case TB_C32:
        if (p.N <= 8 && fills(128, 1, 2)) return f(SlimComplex32<1>());
        if (p.N > 8 && p.N <= 16 && fills(128, 2, 3)) return f(SlimComplex32<2>());
        if (p.N > 16 && p.N <= 24 && fills(128, 3, 24)) return f(SlimComplex32<3>());
        if (p.N > 40 && p.N <= 48 && !p.a_rows_fast && fills(128, 6, 32)) return f(SlimComplex32<6>());
        if (p.N <= 32) return f(Complex32<128, 32>());
        return f(Complex32<64, 64>());
    case TB_C64:
        if (p.N <= 32) return f(Complex64<128, 32, 4, 2>());
        return f(Complex64<64, 64, 2, 4>());
    default:
        if (p.N <= 12 && fills(256, 1, 6)) return p.N <= 8 ? f(Slim32<1, 8>()) : f(Slim32<1, 12>());
        if (p.N > 12 && p.N <= 24 && fills(256, 2, 6)) return p.N <= 16 ? f(Slim32<2, 8>()) : f(Slim32<2, 12>());
        if (p.N > 24 && p.N <= 32 && fills(256, 4, 6)) return f(Slim32<4, 8>());
        if (p.N > 32 && p.N <= 36 && fills(256, 3, 5)) return f(Slim32<3, 12>());
        if (p.N > 36 && p.N <= 40 && fills(256, 5, 6)) return f(Slim32<5, 8>());
        if (p.N > 40 && p.N <= 48 && fills(256, 4, 6)) return f(Slim32<4, 12>());
        if (p.N > 60 && p.N <= 64 && fills(256, 8, 10)) return f(Slim32<8, 8>());
        if (p.N <= 16) return f(Real32<128, 16, 4, 2, 2>());
        if (p.N <= 32) return f(Real32<128, 32, 4, 4, 2>());
        if (p.M > 64 && p.N > 64) {
            const double tiles = (double)((p.M + 127) / 128) * (double)((p.N + 127) / 128) * (double)p.L;
            const int along_k = !p.a_rows_fast + !p.b_rows_fast;
            if ((double)p.M * (double)p.N * (double)p.L >= 148.0 * 128 * 128 ||
                (tiles >= 16 && (along_k == 2 ? p.K >= 512 : p.K >= 1024 && (along_k || p.K >= 2048 || tiles < 128))))
                return f(Real32<128, 128, 8, 8, 2>());
        }
        return f(Real32<64, 64, 4, 4, 2>());
    }
}

}  // namespace tile

// Operands stored as the type they are computed in; binary32 may also be
// rounded to 16 bits. Coordinates fit 32-bit division. Two binary32 operands in
// 16-byte runs along a contraction of 1536 terms and more stay with k_simt, which
// loads four terms at once where this kernel copies one, as long as they have
// fewer than two 128 x 128 tiles per SM but more than 5 (k_simt / this kernel,
// us: 837 x 101 x 2416 38 / 48, 94 x 1773 x 1680 42 / 55, 392 x 68 x 42668 in 2
// batches 322 / 622, 1.04 on average; with 4 tiles 154 x 144 x 3720 52 / 24).
bool tile_takes(const simt::Params& p, int compute)
{
    static const int stored[4] = {T_F32, T_F64, T_C32, T_C64};  // by TB_R32 .. TB_C64
    const int t = stored[compute];
    if (p.tA != t || p.tB != t) return false;
    if (p.round_in != TB_ROUND_NONE && (compute != TB_R32 || p.round_in == TB_ROUND_F32)) return false;
    const int64_t lim = 1ll << 31;
    if (p.M >= lim || p.N >= lim || p.K >= lim || p.L >= lim || p.K < 1) return false;
    const simt::Modes* m[9] = {&p.am, &p.ak, &p.al, &p.bn, &p.bk, &p.bl, &p.cm, &p.cn, &p.cl};
    for (int j = 0; j < 9; j++)
        if (m[j]->n > tile::MAXM) return false;
    // (by the layout alone: where the buffers lie must not choose another order of the sums)
    if (compute == TB_R32 && !p.a_rows_fast && !p.b_rows_fast && p.M > 64 && p.N > 64 && p.K >= 1536 &&
        tile::rows_in_groups(p.ak, p.am, p.al, nullptr, 4, 16) && tile::rows_in_groups(p.bk, p.bn, p.bl, nullptr, 4, 16)) {
        const double tiles = (double)((p.M + 127) / 128) * (double)((p.N + 127) / 128) * (double)p.L;
        if (tiles >= 6 && (double)p.M * (double)p.N * (double)p.L < 148.0 * 128 * 128) return false;
    }
    return true;
}

// kind: the narrow kernel (simt.cu, NK_*; complex float 4 a row per thread, 6
// row vectors). Narrow kernels walk the rows persistently with B resident and
// win on many rows; with few of them, the serial staging of a long B and the
// few blocks cost more than everything else, and one row per thread reads
// eight times the shared memory per multiply-add. Measured (us, narrow / this
// one; rows x columns x contraction):
//   binary64 1.7M x 24 x 64 484 / 390, odd strides 554k x 37 x 201 1439 / 553,
//     4224 x 8 x 250 45 / 8, 10^4 x 33 x 100 70 / 20
//   row per thread, binary32 10^4 x 33 x 101 45 / 20, 1240 x 30 x 230 57 / 13,
//     but 505k x 21 x 129 250 / 286; complex 505k x 45 x 127 901 / 829
//   row vectors, binary32 4224 x 8 x 250 49 / 10, but 655k x 38 x 40 245 / 505;
//     complex 4224 x 8 x 250 61 / 16
// (contractions of up to 130 stay with the row vectors: 1 to 10 us either way).
// Up to 8 columns waste most of this kernel's columns or warps, so the narrow
// ones are ahead as soon as their rows fill the GPU once: binary32 41k x 6 x 68
// 21 / 80 and 115k x 7 x 269 97 / 139; complex, whose rows are streamed one by
// one, already 22k x 2 x 245 44 / 63; binary64 where the contraction is short,
// 286k x 4 x 117 78 / 104, but 109k x 1 x 222 at par and 44k x 3 x 258 58 / 34. From
// 9 columns the line rises with them: 12 columns 79k x 79 31 / 35, 48k x 337 105 / 87,
// 16 columns 113k x 231 89 / 107.
bool tile_over_narrow(const simt::Params& p, int compute, int kind)
{
    if (!tile_takes(p, compute)) return false;
    const double rows = (double)p.M * (double)p.L, cols = (double)p.N;
    const bool vectors = kind >= 5, few = p.N <= 8;
    if (compute == TB_R64) return few && rows >= 148.0 * 256 ? p.K > 130 : vectors ? p.K >= 64 : p.K > 64;
    if (compute == TB_C32 && few) return p.K > (vectors ? 130 : 64) && rows < 148.0 * 96;
    if (vectors) return p.K > 130 && rows < 148.0 * 256;
    if (compute == TB_C32) return p.K > 64 && (p.N > 12 || rows < 148.0 * 1024);
    if (rows < 148.0 * 256) return p.K > 64;
    // (from 13 columns tall tiles take over where the rows fill them)
    return p.K > 64 && !few && rows < 148.0 * 1024 && (rows < 148.0 * 40 * cols || (p.N > 12 && rows >= 148.0 * 768));
}

// tile, cluster and splits of a product that this kernel takes
void tile_describe(const simt::Params& p, int compute, size_t ws_limit, int out[4])
{
    tile::with_tile(p, compute, [&](auto w) {
        using W = decltype(w);
        const int64_t tiles = ((p.M + W::BM - 1) / W::BM) * ((p.N + W::BN - 1) / W::BN) * p.L;
        const tile::Split s = tile::choose_split(tiles, p.K, W::BK, p.L * p.M * p.N, W::E, ws_limit);
        out[0] = W::BM;
        out[1] = W::BN;
        out[2] = s.cluster;
        out[3] = s.splits;
    });
}

cudaError_t launch_tile(const simt::Params& p, int compute, size_t ws_limit, cudaStream_t s)
{
    return tile::with_tile(p, compute, [&](auto w) {
        using W = decltype(w);
        if constexpr (!W::CPLX && W::E == 4) {
            if (p.round_in != TB_ROUND_NONE) return tile::launch<W, true>(p, ws_limit, s);
        }
        return tile::launch<W, false>(p, ws_limit, s);
    });
}

}  // namespace tb
