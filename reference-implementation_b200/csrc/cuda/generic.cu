// CUDA-core product kernels for every shape, storage type and precision.
//
//   k_element_rows one thread per element of D, or for 4 or 8 of them along a
//                  mode that one operand lacks: walks the contracted
//                  coordinates and, inside, the unary coordinates of A and of
//                  B. This is the reference's loop nest
//                  (reference_implementation/src/product.c:338-399) with the
//                  outer loop spread over threads.
//   k_warp_rows    the same with a warp, its lanes along the contraction
//   k_elementwise, k_warpdot
//                  one element of D per thread, per warp: operands of types
//                  that are converted one by one as they are loaded
//   k_reduce       one block per element of D for few outputs with a long
//                  contraction: the contracted range is split over the
//                  block's threads and combined with warp shuffles.
//
// All evaluate D = op_D(alpha * sum op_A(A) op_B(B) + beta * op_C(C)) in the
// plan's compute domain (real/complex, binary32/binary64) and honour the
// plan's operand rounding for the 16-bit precisions.
#include <algorithm>
#include <cstdio>
#include <type_traits>
#include <utility>

#include "tb_common.cuh"

namespace tb {

struct GenParams {
    int32_t nF, nK, nUA, nUB;
    int32_t tA, tB, tC, tD;
    int32_t round_in, conjA, conjB, conjC, conjD, conjD_f32, beta_zero, small_F;
    int32_t warp, pad_;  // warp: one warp per output (warp_element), else one thread (element)
    int64_t sizeF, sizeK, sizeUA, sizeUB;
    double alpha_re, alpha_im, beta_re, beta_im;
    FastDiv fF[TB_MAXMODES];
    int64_t F_ext[TB_MAXMODES], F_sA[TB_MAXMODES], F_sB[TB_MAXMODES], F_sC[TB_MAXMODES], F_sD[TB_MAXMODES];
    int64_t K_ext[TB_MAXMODES], K_sA[TB_MAXMODES], K_sB[TB_MAXMODES];
    FastDiv fK[TB_MAXMODES];
    int64_t UA_ext[TB_MAXMODES], UA_s[TB_MAXMODES];
    int64_t UB_ext[TB_MAXMODES], UB_s[TB_MAXMODES];
};

// complex helpers on (re, im) pairs; CPLX=false keeps only the real part
template <typename R, bool CPLX>
__device__ __forceinline__ void cmac(R& sr, R& si, R ar, R ai, R br, R bi)
{
    if (CPLX) {
        sr = fma(ar, br, sr);
        sr = fma(-ai, bi, sr);
        si = fma(ar, bi, si);
        si = fma(ai, br, si);
    } else {
        sr = fma(ar, br, sr);
    }
}

// sum over the unary coordinates of one operand at base offset `off`, added in
// order, U loads in flight. k_reduce keeps one: with four it took 3 to 47%
// longer, with unary modes or without (a product of 20000 terms and 1000
// outputs, complex binary64, 227 -> 332 us), for registers it does not have.
template <typename R, bool CPLX, int U>
__device__ __forceinline__ void unary_sum(const void* base, int64_t off, int t, int conj, int rmode, int n,
                                          int64_t size, const int64_t* ext, const int64_t* str, R& re, R& im)
{
    if (n == 0) {
        load_rounded<R>(base, off, t, rmode, re, im);
        if (conj) im = -im;
        return;
    }
    re = 0;
    im = 0;
    int64_t c[TB_MAXMODES];
    for (int j = 0; j < n; j++) c[j] = 0;
    int64_t o = off;
    auto next = [&]() {
        for (int j = 0; j < n; j++) {
            o += str[j];
            if (++c[j] < ext[j]) break;
            o -= str[j] * ext[j];
            c[j] = 0;
        }
    };
    auto add = [&](R xr, R xi) {
        if (conj) xi = -xi;
        re += xr;
        im += xi;
        if (rmode != TB_ROUND_NONE) {  // the 16-bit precisions keep the running sum in 16 bits
            re = round_in<R>(re, rmode);
            im = round_in<R>(im, rmode);
        }
    };
    int64_t u = 0;
    if constexpr (U > 1) {
        for (; u + U <= size; u += U) {
            R xr[U], xi[U];
#pragma unroll
            for (int v = 0; v < U; v++) {
                load_elem<R>(base, o, t, xr[v], xi[v]);
                next();
            }
#pragma unroll
            for (int v = 0; v < U; v++) add(xr[v], xi[v]);
        }
    }
    for (; u < size; u++) {
        R xr, xi;
        load_elem<R>(base, o, t, xr, xi);
        add(xr, xi);
        next();
    }
}

// op_D(alpha * sum + beta * op_C(C)) into D, C's value (cr, ci) already loaded
template <typename R, bool CPLX>
__device__ __forceinline__ void finish_c(const GenParams& p, R sr, R si, R cr, R ci, void* D, int64_t oD)
{
    // alpha * sum
    R ar = (R)p.alpha_re, ai = (R)p.alpha_im;
    R accr, acci;
    if (CPLX) {
        accr = ar * sr - ai * si;
        acci = ar * si + ai * sr;
    } else {
        accr = ar * sr;
        acci = 0;
    }
    if (!p.beta_zero) {
        if (p.conjC) ci = -ci;
        R br = (R)p.beta_re, bi = (R)p.beta_im;
        if (CPLX) {
            accr += br * cr - bi * ci;
            acci += br * ci + bi * cr;
        } else {
            accr += br * cr;
        }
    }
    if (p.conjD) {
        if (p.conjD_f32) {
            accr = (R)(float)accr;
            acci = (R)(float)acci;
        }
        acci = -acci;
    }
    store_elem<R>(D, oD, p.tD, accr, acci);
}

template <typename R, bool CPLX>
__device__ __forceinline__ void finish(const GenParams& p, R sr, R si, const void* C, int64_t oC, void* D, int64_t oD)
{
    R cr = 0, ci = 0;
    if (!p.beta_zero) load_rounded<R>(C, oC, p.tC, p.round_in, cr, ci);
    finish_c<R, CPLX>(p, sr, si, cr, ci, D, oD);
}

// offsets in A, B, C and D of the free coordinates of output index i
__device__ __forceinline__ void free_offsets(const GenParams& p, int64_t i, int64_t& oA, int64_t& oB, int64_t& oC,
                                             int64_t& oD)
{
    oA = oB = oC = oD = 0;
    if (p.small_F) {
        uint32_t r = (uint32_t)i;
        for (int j = 0; j < p.nF; j++) {
            uint32_t q = fdiv(r, p.fF[j]);
            int64_t c = r - q * p.fF[j].d;
            r = q;
            oA += c * p.F_sA[j];
            oB += c * p.F_sB[j];
            oC += c * p.F_sC[j];
            oD += c * p.F_sD[j];
        }
    } else {
        int64_t r = i;
        for (int j = 0; j < p.nF; j++) {
            int64_t c = r % p.F_ext[j];
            r /= p.F_ext[j];
            oA += c * p.F_sA[j];
            oB += c * p.F_sB[j];
            oC += c * p.F_sC[j];
            oD += c * p.F_sD[j];
        }
    }
}

// unary loads in flight in the grouped launch and the request loop: their
// products with unary modes take 8 to 14% less time than with one (16-bit
// storage 3% more); four spill for binary32 complex in the grouped launch
template <typename R, bool CPLX>
constexpr int UNARY_LOADS = CPLX && sizeof(R) == 4 ? 2 : 4;

// one element of D: the reference's loop nest for output index i, U unary
// loads in flight
template <typename R, bool CPLX, int U>
__device__ __forceinline__ void element(const GenParams& p, const void* A, const void* B, const void* C, void* D,
                                        int64_t i)
{
    int64_t oA, oB, oC, oD;
    free_offsets(p, i, oA, oB, oC, oD);
    R sr = 0, si = 0;
    int64_t kc[TB_MAXMODES];
    for (int j = 0; j < p.nK; j++) kc[j] = 0;
    int64_t kA = oA, kB = oB;
    int64_t k0 = 0;
    if (p.nUA == 0 && p.nUB == 0) {
        // no unary modes: UNR terms' loads issued together, then their
        // multiply-adds in order (the same values and order as below)
        constexpr int UNR = (CPLX || sizeof(R) == 8) ? 4 : 8;
        for (; k0 + UNR <= p.sizeK; k0 += UNR) {
            R ar[UNR], ai[UNR], br[UNR], bi[UNR];
#pragma unroll
            for (int u = 0; u < UNR; u++) {
                load_rounded<R>(A, kA, p.tA, p.round_in, ar[u], ai[u]);
                load_rounded<R>(B, kB, p.tB, p.round_in, br[u], bi[u]);
                for (int j = 0; j < p.nK; j++) {
                    kA += p.K_sA[j];
                    kB += p.K_sB[j];
                    if (++kc[j] < p.K_ext[j]) break;
                    kA -= p.K_sA[j] * p.K_ext[j];
                    kB -= p.K_sB[j] * p.K_ext[j];
                    kc[j] = 0;
                }
            }
#pragma unroll
            for (int u = 0; u < UNR; u++) {
                if (p.conjA) ai[u] = -ai[u];
                if (p.conjB) bi[u] = -bi[u];
                cmac<R, CPLX>(sr, si, ar[u], ai[u], br[u], bi[u]);
            }
        }
    }
    for (int64_t k = k0; k < p.sizeK; k++) {
        R ar, ai, br, bi;
        unary_sum<R, CPLX, U>(A, kA, p.tA, p.conjA, p.round_in, p.nUA, p.sizeUA, p.UA_ext, p.UA_s, ar, ai);
        unary_sum<R, CPLX, U>(B, kB, p.tB, p.conjB, p.round_in, p.nUB, p.sizeUB, p.UB_ext, p.UB_s, br, bi);
        cmac<R, CPLX>(sr, si, ar, ai, br, bi);
        for (int j = 0; j < p.nK; j++) {
            kA += p.K_sA[j];
            kB += p.K_sB[j];
            if (++kc[j] < p.K_ext[j]) break;
            kA -= p.K_sA[j] * p.K_ext[j];
            kB -= p.K_sB[j] * p.K_ext[j];
            kc[j] = 0;
        }
    }
    finish<R, CPLX>(p, sr, si, C, oC, D, oD);
}

// Several outputs per thread (k_element_rows) or per warp (k_warp_rows): NR
// outputs along a free mode that one operand (the shared one) lacks. The
// shared operand's value is loaded once per term for all of them, the index
// arithmetic is done once, and the other operand's NR loads of a term are in
// flight together. Every output sums the same terms in the same order as
// element() or warp_element(), so the bits are those of the kernels that take
// one output at a time, of the grouped launches and of the request loop.
// One output per thread was bound by one load of the varying operand in flight
// for each of the shared one, one per warp by index arithmetic and shuffles:
// the 823 MB Hadamard product of 69 terms went from 621 to 209 us (3.9 TB/s),
// its form with the contraction contiguous from 1790 to 331 us, and the
// mixed-class product's unary sums, loads side by side and offsets from tables,
// from 40 to 17 us.
// The mode's place in p's free modes counts the groups: a group is NR
// neighbours, or, spread, every groups-th coordinate (so that the lanes of a
// warp still read neighbours when the mode is the one they walk).
struct RowGroup {
    int64_t ext, groups, inner;  // extent of the mode, its groups, outputs of p per group step
    int64_t v, c, d;             // from one row of a group to the next: in the varying operand, C, D
    int32_t swapped, spread;     // the varying operand, A here, is the product's B
};

// outputs of group index i of p
template <int NR>
__device__ __forceinline__ int rows_of(const RowGroup& g, int64_t i)
{
    const int64_t q = i / g.inner % g.groups;
    const int64_t n = g.spread ? (g.ext - q + g.groups - 1) / g.groups : g.ext - q * NR;
    return n < NR ? (int)n : NR;
}

// One warp per element of D for products whose contraction runs along an
// operand's contiguous mode while consecutive outputs do not (batched
// matrix-vector and Hadamard products with A stored contraction-fastest):
// the lanes take every 32nd term (lane j the terms j, j + 32, ...), so each
// load of the warp reads 32 neighbouring elements instead of 32 elements a
// whole row apart, and a shuffle tree adds the 32 partial sums (a fixed
// order: the same bits in every run).
template <typename R, bool CPLX, int U>
__device__ __forceinline__ void warp_element(const GenParams& p, const void* A, const void* B, const void* C, void* D,
                                             int64_t i, int lane)
{
    {
        int64_t oA, oB, oC, oD;
        free_offsets(p, i, oA, oB, oC, oD);
        R sr = 0, si = 0;
        auto term_offsets = [&](int64_t k, int64_t& kA, int64_t& kB) {
            kA = oA;
            kB = oB;
            uint32_t r = (uint32_t)k;
            for (int j = 0; j < p.nK; j++) {
                const uint32_t q = j + 1 < p.nK ? fdiv(r, p.fK[j]) : 0;
                const int64_t c = j + 1 < p.nK ? (int64_t)(r - q * p.fK[j].d) : (int64_t)r;
                r = q;
                kA += c * p.K_sA[j];
                kB += c * p.K_sB[j];
            }
        };
        int64_t k0 = lane;
        if (p.nUA == 0 && p.nUB == 0) {
            // the lane's next 4 terms loaded together, then added in order
            for (; k0 + 3 * 32 < p.sizeK; k0 += 4 * 32) {
                R ar[4], ai[4], br[4], bi[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    int64_t kA, kB;
                    term_offsets(k0 + 32 * u, kA, kB);
                    load_rounded<R>(A, kA, p.tA, p.round_in, ar[u], ai[u]);
                    load_rounded<R>(B, kB, p.tB, p.round_in, br[u], bi[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (p.conjA) ai[u] = -ai[u];
                    if (p.conjB) bi[u] = -bi[u];
                    cmac<R, CPLX>(sr, si, ar[u], ai[u], br[u], bi[u]);
                }
            }
        }
        for (int64_t k = k0; k < p.sizeK; k += 32) {
            int64_t kA, kB;
            term_offsets(k, kA, kB);
            R ar, ai, br, bi;
            unary_sum<R, CPLX, U>(A, kA, p.tA, p.conjA, p.round_in, p.nUA, p.sizeUA, p.UA_ext, p.UA_s, ar, ai);
            unary_sum<R, CPLX, U>(B, kB, p.tB, p.conjB, p.round_in, p.nUB, p.sizeUB, p.UB_ext, p.UB_s, br, bi);
            cmac<R, CPLX>(sr, si, ar, ai, br, bi);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sr += __shfl_xor_sync(0xffffffffu, sr, o);
            if (CPLX) si += __shfl_xor_sync(0xffffffffu, si, o);
        }
        if (lane == 0) finish<R, CPLX>(p, sr, si, C, oC, D, oD);
    }
}

// How the row kernels load A and B: NATIVE, both stored as R (pairs of R,
// aligned to the pair, for complex); STORED16, both in 16 bits, either kind
// (R = float). Nothing branches between a step's loads, so that they are in
// flight together; the precision's rounding is done on all of them afterwards.
// Operands of other types (ANY) keep the kernels that take one output at a
// time (k_elementwise, k_warpdot): in groups their loads, each behind a switch,
// waited for one another (16-bit operands, 531 terms x 4725 outputs: 17 -> 29 us).
enum { NATIVE, STORED16, ANY };

template <typename R, bool CPLX, int LOADS>
__device__ __forceinline__ void load_term(const void* base, int64_t off, int t, R& re, R& im)
{
    im = 0;
    if constexpr (LOADS == STORED16) {
        const unsigned short h = __ldg((const unsigned short*)base + off);
        re = t == T_BF16 ? (R)__uint_as_float((uint32_t)h << 16) : (R)__half2float(__ushort_as_half(h));
    } else if constexpr (CPLX && sizeof(R) == 4) {
        const float2 q = __ldg((const float2*)base + off);
        re = q.x;
        im = q.y;
    } else if constexpr (CPLX) {
        const double2 q = __ldg((const double2*)base + off);
        re = q.x;
        im = q.y;
    } else {
        re = __ldg((const R*)base + off);
    }
}

// loaded values rounded to the precision's operand format (binary32 only: the
// 16-bit precisions compute in it)
template <typename R, bool CPLX, int N>
__device__ __forceinline__ void round_terms(int rmode, R (&re)[N], R (&im)[N])
{
    if constexpr (sizeof(R) == 4) {
        if (rmode == TB_ROUND_NONE) return;
#pragma unroll
        for (int r = 0; r < N; r++) {
            re[r] = round_in<R>(re[r], rmode);
            if (CPLX) im[r] = round_in<R>(im[r], rmode);
        }
    }
}

// The offsets of a product's contracted and unary coordinates in shared
// memory: resolved by the block once, a coordinate per thread, where the loops
// over them would spend some 50 instructions a term on strides in parameter
// memory. Longer sums than the tables step through the coordinates, and so do
// the kernels that spread a step over 8 or 4 rows and have no unary modes, to
// which the tables gave nothing (35 to 39 us for a product of 10^6 outputs and
// 20 terms).
constexpr int TAB_K = 512, TAB_U = 128;

__device__ __forceinline__ bool k_tabled(const GenParams& p) { return p.sizeK <= TAB_K; }
__host__ __device__ __forceinline__ bool u_tabled(const GenParams& p) { return p.sizeUA <= TAB_U && p.sizeUB <= TAB_U; }

__device__ __forceinline__ void fill_tables(const GenParams& p, int64_t* ka, int64_t* kb, int64_t* ua, int64_t* ub)
{
    const int t = threadIdx.x, n = blockDim.x;
    if (k_tabled(p)) {
        for (int k = t; k < (int)p.sizeK; k += n) {
            uint32_t r = (uint32_t)k;
            int64_t oa = 0, ob = 0;
            for (int j = 0; j < p.nK; j++) {
                const uint32_t q = j + 1 < p.nK ? fdiv(r, p.fK[j]) : 0;
                const int64_t c = j + 1 < p.nK ? (int64_t)(r - q * p.fK[j].d) : (int64_t)r;
                r = q;
                oa += c * p.K_sA[j];
                ob += c * p.K_sB[j];
            }
            ka[k] = oa;
            kb[k] = ob;
        }
    }
    if (u_tabled(p)) {
        auto unary = [&](int64_t* tab, int size, int nU, const int64_t* ext, const int64_t* str) {
            for (int u = t; u < size; u += n) {
                uint32_t r = (uint32_t)u;
                int64_t o = 0;
                for (int j = 0; j < nU; j++) {
                    const uint32_t e = (uint32_t)ext[j], q = r / e;
                    o += (int64_t)(r - q * e) * str[j];
                    r = q;
                }
                tab[u] = o;
            }
        };
        if (p.nUA) unary(ua, (int)p.sizeUA, p.nUA, p.UA_ext, p.UA_s);
        if (p.nUB) unary(ub, (int)p.sizeUB, p.nUB, p.UB_ext, p.UB_s);
    }
    __syncthreads();
}

// unary_sum for NR rows side by side (offsets at[r] apart), from a table of
// offsets: U coordinates' loads in flight, added in order
template <typename R, bool CPLX, int LOADS, int NR, int U>
__device__ __forceinline__ void unary_rows(const void* base, int64_t off, const int64_t (&at)[NR], int t, int conj, int rmode,
                                           const int64_t* tab, int size, R (&re)[NR], R (&im)[NR])
{
#pragma unroll
    for (int r = 0; r < NR; r++) re[r] = im[r] = 0;
    auto some = [&](auto count, int u0) {
        constexpr int N = decltype(count)::value;
        R yr[N][NR], yi[N][NR];
#pragma unroll
        for (int u = 0; u < N; u++) {
            const int64_t o = off + tab[u0 + u];
#pragma unroll
            for (int r = 0; r < NR; r++) load_term<R, CPLX, LOADS>(base, o + at[r], t, yr[u][r], yi[u][r]);
        }
#pragma unroll
        for (int u = 0; u < N; u++)
#pragma unroll
            for (int r = 0; r < NR; r++) {
                re[r] += yr[u][r];
                im[r] += conj ? -yi[u][r] : yi[u][r];
                if (rmode != TB_ROUND_NONE) {  // the 16-bit precisions keep the running sum in 16 bits
                    re[r] = round_in<R>(re[r], rmode);
                    im[r] = round_in<R>(im[r], rmode);
                }
            }
    };
    int u = 0;
    for (; u + U <= size; u += U) some(std::integral_constant<int, U>(), u);
    for (; u < size; u++) some(std::integral_constant<int, 1>(), u);
}

// One term's values: B's (shared) and the NR rows' of A (varying),
// unary sums included, at contracted offsets kS and kV. (Several rows are only
// taken where the tables hold the unary modes.)
template <typename R, bool CPLX, int LOADS, int NR>
__device__ __forceinline__ void summed_term(const GenParams& p, const void* A, const void* B, int64_t kV, int64_t kS,
                                            const int64_t (&at)[NR], const int64_t* ua, const int64_t* ub, R (&vr)[NR],
                                            R (&vi)[NR], R& xr, R& xi)
{
    if (p.nUB == 0) {
        R yr[1], yi[1];
        load_term<R, CPLX, LOADS>(B, kS, p.tB, yr[0], yi[0]);
        round_terms<R, CPLX>(p.round_in, yr, yi);
        xr = yr[0];
        xi = p.conjB ? -yi[0] : yi[0];
    } else if (NR > 1 || u_tabled(p)) {
        const int64_t zero[1] = {0};
        R yr[1], yi[1];
        unary_rows<R, CPLX, LOADS, 1, 4>(B, kS, zero, p.tB, p.conjB, p.round_in, ub, (int)p.sizeUB, yr, yi);
        xr = yr[0];
        xi = yi[0];
    } else {
        unary_sum<R, CPLX, 4>(B, kS, p.tB, p.conjB, p.round_in, p.nUB, p.sizeUB, p.UB_ext, p.UB_s, xr, xi);
    }
    if (p.nUA == 0) {
#pragma unroll
        for (int r = 0; r < NR; r++) load_term<R, CPLX, LOADS>(A, kV + at[r], p.tA, vr[r], vi[r]);
        round_terms<R, CPLX>(p.round_in, vr, vi);
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (p.conjA) vi[r] = -vi[r];
    } else if (NR > 1 || u_tabled(p)) {
        unary_rows<R, CPLX, LOADS, NR, NR == 1 ? 4 : NR == 4 || !CPLX ? 2 : 1>(A, kV, at, p.tA, p.conjA, p.round_in, ua, (int)p.sizeUA, vr, vi);
    } else {
        unary_sum<R, CPLX, 4>(A, kV + at[0], p.tA, p.conjA, p.round_in, p.nUA, p.sizeUA, p.UA_ext, p.UA_s, vr[0], vi[0]);
    }
}

// NR outputs per thread: element() for each of them (NR = 1: the plain element kernel)
template <typename R, bool CPLX, int LOADS, int NR>
__global__ void __launch_bounds__(256) k_element_rows(GenParams p, RowGroup g,
                                                      const void* A, const void* B, const void* C, void* D)
{
    constexpr bool TABLES = NR == 1;
    __shared__ int64_t ka[TABLES ? TAB_K : 1], kb[TABLES ? TAB_K : 1], ua[TABLES ? TAB_U : 1], ub[TABLES ? TAB_U : 1];
    // terms whose loads are issued together: 8 to 16 loads of the varying operand
    constexpr int UNR = NR >= 8 ? 2 : NR > 1 ? 4 : (CPLX || sizeof(R) == 8) ? 4 : 8;
    if constexpr (TABLES) fill_tables(p, ka, kb, ua, ub);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.sizeF; i += stride) {
        int64_t oA, oB, oC, oD;
        free_offsets(p, i, oA, oB, oC, oD);
        const int rows = NR == 1 ? 1 : rows_of<NR>(g, i);
        int64_t at[NR];  // absent outputs repeat the first one's loads
#pragma unroll
        for (int r = 0; r < NR; r++) at[r] = r < rows ? r * g.v : 0;
        R sr[NR], si[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) sr[r] = si[r] = 0;
        int64_t kc[TB_MAXMODES], kV = oA, kS = oB;  // stepped through without a table
        if (!TABLES || !k_tabled(p))
            for (int j = 0; j < p.nK; j++) kc[j] = 0;
        auto offsets = [&](int64_t k, int64_t& v, int64_t& s) {
            if (TABLES && k_tabled(p)) {
                v = oA + ka[k];
                s = oB + kb[k];
                return;
            }
            v = kV;
            s = kS;
            for (int j = 0; j < p.nK; j++) {
                kV += p.K_sA[j];
                kS += p.K_sB[j];
                if (++kc[j] < p.K_ext[j]) break;
                kV -= p.K_sA[j] * p.K_ext[j];
                kS -= p.K_sB[j] * p.K_ext[j];
                kc[j] = 0;
            }
        };
        auto add = [&](int r, R vr, R vi, R xr, R xi) {
            if (g.swapped) cmac<R, CPLX>(sr[r], si[r], xr, xi, vr, vi);
            else cmac<R, CPLX>(sr[r], si[r], vr, vi, xr, xi);
        };
        auto terms = [&](auto count, int64_t k) {
            constexpr int U = decltype(count)::value;
            R vr[U][NR], vi[U][NR], xr[U], xi[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                int64_t v, s;
                offsets(k + u, v, s);
                load_term<R, CPLX, LOADS>(B, s, p.tB, xr[u], xi[u]);
#pragma unroll
                for (int r = 0; r < NR; r++) load_term<R, CPLX, LOADS>(A, v + at[r], p.tA, vr[u][r], vi[u][r]);
            }
            if (sizeof(R) == 4 && p.round_in != TB_ROUND_NONE) {
                round_terms<R, CPLX>(p.round_in, xr, xi);
#pragma unroll
                for (int u = 0; u < U; u++) round_terms<R, CPLX>(p.round_in, vr[u], vi[u]);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (p.conjB) xi[u] = -xi[u];
#pragma unroll
                for (int r = 0; r < NR; r++) add(r, vr[u][r], p.conjA ? -vi[u][r] : vi[u][r], xr[u], xi[u]);
            }
        };
        int64_t k = 0;
        if (NR > 1 || (p.nUA == 0 && p.nUB == 0)) {  // (unary modes run one row a thread)
            for (; k + UNR <= p.sizeK; k += UNR) terms(std::integral_constant<int, UNR>(), k);
            for (; k < p.sizeK; k++) terms(std::integral_constant<int, 1>(), k);
        } else {
            for (; k < p.sizeK; k++) {
                int64_t v, s;
                offsets(k, v, s);
                R vr[NR], vi[NR], xr, xi;
                summed_term<R, CPLX, LOADS, NR>(p, A, B, v, s, at, ua, ub, vr, vi, xr, xi);
#pragma unroll
                for (int r = 0; r < NR; r++) add(r, vr[r], vi[r], xr, xi);
            }
        }
        R cr[NR], ci[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) {
            cr[r] = ci[r] = 0;
            if (!p.beta_zero && r < rows) load_rounded<R>(C, oC + r * g.c, p.tC, p.round_in, cr[r], ci[r]);
        }
#pragma unroll
        for (int r = 0; r < NR; r++)
            if (r < rows) finish_c<R, CPLX>(p, sr[r], si[r], cr[r], ci[r], D, oD + r * g.d);
    }
}

// NR outputs per warp: warp_element for each of them (NR = 1: the plain warp
// kernel). The partial sums of the rows meet in one transposed shuffle tree,
// in which a lane hands away half of its rows at each step, so 8 rows take 9
// shuffles instead of 40 and end on 8 different lanes; each row's sum is that
// of the same tree as warp_element's. UNARY: some operand has unary modes.
template <typename R, bool CPLX, int LOADS, int NR, bool UNARY>
__global__ void __launch_bounds__(128, CPLX && NR == 8 ? (sizeof(R) == 4 ? 4 : 2) : sizeof(R) == 8 ? 4 : CPLX || UNARY ? 5 : 8)
    k_warp_rows(GenParams p, RowGroup g, const void* A, const void* B,
                const void* C, void* D)
{
    __shared__ int64_t ka[UNARY ? TAB_K : 1], kb[UNARY ? TAB_K : 1], ua[UNARY ? TAB_U : 1], ub[UNARY ? TAB_U : 1];
    constexpr int UNR = NR == 1 ? 4 : 2;  // terms of a lane whose loads are issued together
    if constexpr (UNARY) fill_tables(p, ka, kb, ua, ub);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int lane = threadIdx.x & 31;
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < p.sizeF; i += warps) {
        int64_t oA, oB, oC, oD;
        free_offsets(p, i, oA, oB, oC, oD);
        const int rows = NR == 1 ? 1 : rows_of<NR>(g, i);
        int64_t at[NR];  // absent outputs repeat the first one's loads
#pragma unroll
        for (int r = 0; r < NR; r++) at[r] = r < rows ? r * g.v : 0;
        R sr[NR], si[NR];
#pragma unroll
        for (int r = 0; r < NR; r++) sr[r] = si[r] = 0;
        auto offsets = [&](int64_t k, int64_t& v, int64_t& s) {
            v = oA;
            s = oB;
            if (UNARY && k_tabled(p)) {
                v += ka[k];
                s += kb[k];
                return;
            }
            uint32_t r = (uint32_t)k;
            for (int j = 0; j < p.nK; j++) {
                const uint32_t q = j + 1 < p.nK ? fdiv(r, p.fK[j]) : 0;
                const int64_t c = j + 1 < p.nK ? (int64_t)(r - q * p.fK[j].d) : (int64_t)r;
                r = q;
                v += c * p.K_sA[j];
                s += c * p.K_sB[j];
            }
        };
        auto add = [&](int r, R vr, R vi, R xr, R xi) {
            if (g.swapped) cmac<R, CPLX>(sr[r], si[r], xr, xi, vr, vi);
            else cmac<R, CPLX>(sr[r], si[r], vr, vi, xr, xi);
        };
        if constexpr (!UNARY) {
            for (int64_t k = lane; k < p.sizeK; k += UNR * 32) {
                R vr[UNR][NR], vi[UNR][NR], xr[UNR], xi[UNR];
#pragma unroll
                for (int u = 0; u < UNR; u++) {
                    if (k + 32 * u >= p.sizeK) continue;
                    int64_t v, s;
                    offsets(k + 32 * u, v, s);
                    load_term<R, CPLX, LOADS>(B, s, p.tB, xr[u], xi[u]);
#pragma unroll
                    for (int r = 0; r < NR; r++) load_term<R, CPLX, LOADS>(A, v + at[r], p.tA, vr[u][r], vi[u][r]);
                }
                if (sizeof(R) == 4 && p.round_in != TB_ROUND_NONE) {
#pragma unroll
                    for (int u = 0; u < UNR; u++) {
                        if (k + 32 * u >= p.sizeK) continue;
                        xr[u] = round_in<R>(xr[u], p.round_in);
                        if (CPLX) xi[u] = round_in<R>(xi[u], p.round_in);
                        round_terms<R, CPLX>(p.round_in, vr[u], vi[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < UNR; u++) {
                    if (k + 32 * u >= p.sizeK) continue;
                    if (p.conjB) xi[u] = -xi[u];
#pragma unroll
                    for (int r = 0; r < NR; r++) add(r, vr[u][r], p.conjA ? -vi[u][r] : vi[u][r], xr[u], xi[u]);
                }
            }
        } else {
            for (int64_t k = lane; k < p.sizeK; k += 32) {
                int64_t v, s;
                offsets(k, v, s);
                R vr[NR], vi[NR], xr, xi;
                summed_term<R, CPLX, LOADS, NR>(p, A, B, v, s, at, ua, ub, vr, vi, xr, xi);
#pragma unroll
                for (int r = 0; r < NR; r++) add(r, vr[r], vi[r], xr, xi);
            }
        }
        // step o: a lane keeps the upper or lower half of its rows by its bit o
        int row = 0, o = 16;
#pragma unroll
        for (int n = NR; n > 1; n /= 2, o /= 2) {
            const bool up = (lane & o) != 0;
            row += up ? n / 2 : 0;
#pragma unroll
            for (int r = 0; r < n / 2; r++) {
                const R give = up ? sr[r] : sr[r + n / 2], keep = up ? sr[r + n / 2] : sr[r];
                sr[r] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                if (CPLX) {
                    const R gi = up ? si[r] : si[r + n / 2], ki = up ? si[r + n / 2] : si[r];
                    si[r] = ki + __shfl_xor_sync(0xffffffffu, gi, o);
                }
            }
        }
        for (; o > 0; o /= 2) {
            sr[0] += __shfl_xor_sync(0xffffffffu, sr[0], o);
            if (CPLX) si[0] += __shfl_xor_sync(0xffffffffu, si[0], o);
        }
        if (lane % (32 / NR) == 0 && row < rows) finish<R, CPLX>(p, sr[0], si[0], C, oC + row * g.c, D, oD + row * g.d);
    }
}

template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) k_elementwise(GenParams p, const void* A, const void* B, const void* C, void* D)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.sizeF; i += stride)
        element<R, CPLX, 1>(p, A, B, C, D, i);
}

template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) k_warpdot(GenParams p, const void* A, const void* B, const void* C, void* D)
{
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < p.sizeF; i += warps)
        warp_element<R, CPLX, 1>(p, A, B, C, D, i, threadIdx.x & 31);
}

// Many independent products of the same compute domain in one launch:
// product j owns blocks [first[j], first[j+1]) and walks its elements with
// them. Descriptors and operand pointers live in device memory.
template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) k_elementwise_group(const GenParams* __restrict__ params,
                                                           const tb_ptrs* __restrict__ ptrs,
                                                           const int64_t* __restrict__ first, int n)
{
    int lo = 0, hi = n - 1;  // last j with first[j] <= blockIdx.x
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first[mid] <= (int64_t)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const GenParams& p = params[lo];
    const tb_ptrs q = ptrs[lo];
    const int64_t nb = first[lo + 1] - first[lo];
    if (p.warp) {
        const int64_t warps = nb * (blockDim.x >> 5);
        for (int64_t i = ((int64_t)blockIdx.x - first[lo]) * (blockDim.x >> 5) + (threadIdx.x >> 5); i < p.sizeF;
             i += warps)
            warp_element<R, CPLX, UNARY_LOADS<R, CPLX>>(p, q.A, q.B, q.C, q.D, i, threadIdx.x & 31);
        return;
    }
    const int64_t stride = nb * blockDim.x;
    for (int64_t i = ((int64_t)blockIdx.x - first[lo]) * blockDim.x + threadIdx.x; i < p.sizeF; i += stride)
        element<R, CPLX, UNARY_LOADS<R, CPLX>>(p, q.A, q.B, q.C, q.D, i);
}

template <typename R>
__device__ __forceinline__ R warp_sum(R v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Few outputs, long contraction: block (x, y) sums the y-th chunk of the
// contracted range of output x with all its threads (combined by warp
// shuffles). With one chunk the block finishes the output itself; with
// several, each chunk's sum goes to a workspace and k_reduce_final adds the
// chunks in order and finishes, so the result does not depend on scheduling.
template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) k_reduce(GenParams p, const void* A, const void* B, const void* C, void* D,
                                                int64_t chunk, R* ws)
{
    __shared__ R red[2][8];
    const int64_t kbeg = (int64_t)blockIdx.y * chunk;
    const int64_t kend = kbeg + chunk < p.sizeK ? kbeg + chunk : p.sizeK;
    for (int64_t i = blockIdx.x; i < p.sizeF; i += gridDim.x) {
        int64_t oA = 0, oB = 0, oC = 0, oD = 0;
        int64_t r = i;
        for (int j = 0; j < p.nF; j++) {
            int64_t c = r % p.F_ext[j];
            r /= p.F_ext[j];
            oA += c * p.F_sA[j];
            oB += c * p.F_sB[j];
            oC += c * p.F_sC[j];
            oD += c * p.F_sD[j];
        }
        R sr = 0, si = 0;
        for (int64_t k = kbeg + threadIdx.x; k < kend; k += blockDim.x) {
            uint32_t rk = (uint32_t)k;
            int64_t kA = oA, kB = oB;
            for (int j = 0; j < p.nK; j++) {
                uint32_t q = fdiv(rk, p.fK[j]);
                int64_t c = rk - q * p.fK[j].d;
                rk = q;
                kA += c * p.K_sA[j];
                kB += c * p.K_sB[j];
            }
            R ar, ai, br, bi;
            unary_sum<R, CPLX, 1>(A, kA, p.tA, p.conjA, p.round_in, p.nUA, p.sizeUA, p.UA_ext, p.UA_s, ar, ai);
            unary_sum<R, CPLX, 1>(B, kB, p.tB, p.conjB, p.round_in, p.nUB, p.sizeUB, p.UB_ext, p.UB_s, br, bi);
            cmac<R, CPLX>(sr, si, ar, ai, br, bi);
        }
        sr = warp_sum(sr);
        if (CPLX) si = warp_sum(si);
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l == 0) { red[0][w] = sr; red[1][w] = si; }
        __syncthreads();
        if (threadIdx.x == 0) {
            R tr = 0, ti = 0;
            for (int j = 0; j < (int)(blockDim.x >> 5); j++) { tr += red[0][j]; ti += red[1][j]; }
            if (ws) {
                ws[(blockIdx.y * p.sizeF + i) * 2] = tr;
                ws[(blockIdx.y * p.sizeF + i) * 2 + 1] = ti;
            } else {
                finish<R, CPLX>(p, tr, ti, C, oC, D, oD);
            }
        }
        __syncthreads();
    }
}

template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) k_reduce_final(GenParams p, const void* C, void* D, int chunks, const R* ws)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.sizeF; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t oC = 0, oD = 0, r = i;
        for (int j = 0; j < p.nF; j++) {
            int64_t c = r % p.F_ext[j];
            r /= p.F_ext[j];
            oC += c * p.F_sC[j];
            oD += c * p.F_sD[j];
        }
        R tr = 0, ti = 0;
        for (int z = 0; z < chunks; z++) {
            tr += ws[(z * p.sizeF + i) * 2];
            ti += ws[(z * p.sizeF + i) * 2 + 1];
        }
        finish<R, CPLX>(p, tr, ti, C, oC, D, oD);
    }
}

// chunks of the contraction for the reduction path: about 8 blocks per SM in
// all, every chunk at least 2048 terms long
static int reduce_chunks(int64_t outs, int64_t K)
{
    if (outs <= 0) return 1;
    int64_t S = (148 * 8 + outs - 1) / outs;
    const int64_t by_len = K / 2048;
    if (S > by_len) S = by_len;
    if (S > 4096) S = 4096;
    return S < 1 ? 1 : (int)S;
}

size_t reduce_scratch_bytes(const tb_plan* P, size_t real_bytes)
{
    const int S = reduce_chunks(P->F.size, P->K.size);
    return S > 1 ? (size_t)S * (size_t)P->F.size * 2 * real_bytes : 0;
}

static bool warpdot_ok(const GenParams& g);

static void fill_params(const tb_plan* P, GenParams& g)
{
    memset(&g, 0, sizeof(g));
    g.nF = P->F.n; g.nK = P->K.n; g.nUA = P->UA.n; g.nUB = P->UB.n;
    g.tA = P->tA; g.tB = P->tB; g.tC = P->tC; g.tD = P->tD;
    g.round_in = P->round_in;
    g.conjA = P->conjA; g.conjB = P->conjB; g.conjC = P->conjC; g.conjD = P->conjD;
    g.conjD_f32 = P->conjD_round_f32;
    g.beta_zero = P->beta_zero;
    g.sizeF = P->F.size; g.sizeK = P->K.size; g.sizeUA = P->UA.size; g.sizeUB = P->UB.size;
    g.alpha_re = P->alpha_re; g.alpha_im = P->alpha_im;
    g.beta_re = P->beta_re; g.beta_im = P->beta_im;
    g.small_F = P->F.size < (1ll << 31);
    for (int j = 0; j < P->F.n; j++) {
        g.F_ext[j] = P->F.ext[j];
        g.fF[j] = make_fastdiv(g.small_F ? (uint32_t)P->F.ext[j] : 1u);
        g.F_sA[j] = P->F.sA[j]; g.F_sB[j] = P->F.sB[j]; g.F_sC[j] = P->F.sC[j]; g.F_sD[j] = P->F.sD[j];
    }
    for (int j = 0; j < P->K.n; j++) {
        g.K_ext[j] = P->K.ext[j];
        g.fK[j] = make_fastdiv(P->K.size < (1ll << 31) ? (uint32_t)P->K.ext[j] : 1u);
        g.K_sA[j] = P->K.sA[j]; g.K_sB[j] = P->K.sB[j];
    }
    for (int j = 0; j < P->UA.n; j++) { g.UA_ext[j] = P->UA.ext[j]; g.UA_s[j] = P->UA.sA[j]; }
    for (int j = 0; j < P->UB.n; j++) { g.UB_ext[j] = P->UB.ext[j]; g.UB_s[j] = P->UB.sB[j]; }
    g.warp = warpdot_ok(g) ? 1 : 0;
}

// Element path kernel: the warp per output (k_warp_rows, k_warpdot)
//   - when an operand is contiguous along the contraction while consecutive
//     outputs step it by a stride other than 0 or 1 (one thread per output
//     would read it a row apart from lane to lane), for contractions of at
//     least 64 terms;
//   - when one thread per output makes less than a wave (fewer than 148 x 256
//     outputs) and each output sums at least 8 terms with at least 64 loads
//     in all (unary sums included): the lanes share the terms.
static bool warpdot_ok(const GenParams& g)
{
    if (g.sizeK >= (1ll << 31) || g.nK < 1 || g.nF < 1) return false;
    if (g.sizeF < 148 * 256 && g.sizeK >= 8 && (double)g.sizeK * (double)(g.sizeUA + g.sizeUB) >= 64.0) return true;
    if (g.sizeK < 64) return false;
    auto a = [](int64_t x) { return x < 0 ? -x : x; };
    // not when consecutive outputs already walk the other operand along its
    // contiguous mode (threads per output read that one in whole lines)
    const bool by_A = a(g.K_sA[0]) == 1 && a(g.F_sA[0]) > 1 && a(g.F_sB[0]) != 1;
    const bool by_B = a(g.K_sB[0]) == 1 && a(g.F_sB[0]) > 1 && a(g.F_sA[0]) != 1;
    return by_A || by_B;
}

static void swap_operands(GenParams& g)
{
    auto swap_all = [](int64_t* a, int64_t* b) {
        for (int j = 0; j < TB_MAXMODES; j++) std::swap(a[j], b[j]);
    };
    std::swap(g.tA, g.tB);
    std::swap(g.conjA, g.conjB);
    std::swap(g.nUA, g.nUB);
    std::swap(g.sizeUA, g.sizeUB);
    swap_all(g.F_sA, g.F_sB);
    swap_all(g.K_sA, g.K_sB);
    swap_all(g.UA_ext, g.UB_ext);
    swap_all(g.UA_s, g.UB_s);
}

// Puts free mode j of g into groups of nr (RowGroup): neighbours, the groups
// walked slowest, or spread, in place.
static void group_rows(GenParams& g, RowGroup& q, int j, int nr, bool spread)
{
    const int64_t e = g.F_ext[j], groups = (e + nr - 1) / nr;
    q.ext = e;
    q.groups = groups;
    q.spread = spread;
    if (g.F_sA[j] == 0) {  // the varying operand takes A's place
        q.swapped = 1;
        swap_operands(g);
    }
    const int64_t step = spread ? groups : 1, base = spread ? 1 : nr;
    const int64_t s[4] = {g.F_sA[j], g.F_sB[j], g.F_sC[j], g.F_sD[j]};
    q.v = step * s[0];
    q.c = step * s[2];
    q.d = step * s[3];
    const int64_t others = g.sizeF / e;
    q.inner = 1;
    int at = j;
    if (spread) {
        for (int i = 0; i < j; i++) q.inner *= g.F_ext[i];
    } else {
        q.inner = others;
        for (; at + 1 < g.nF; at++) {
            g.F_ext[at] = g.F_ext[at + 1];
            g.fF[at] = g.fF[at + 1];
            g.F_sA[at] = g.F_sA[at + 1];
            g.F_sB[at] = g.F_sB[at + 1];
            g.F_sC[at] = g.F_sC[at + 1];
            g.F_sD[at] = g.F_sD[at + 1];
        }
    }
    g.F_ext[at] = groups;
    g.fF[at] = make_fastdiv(g.small_F ? (uint32_t)groups : 1u);
    g.F_sA[at] = s[0] * base;
    g.F_sB[at] = s[1] * base;
    g.F_sC[at] = s[2] * base;
    g.F_sD[at] = s[3] * base;
    g.sizeF = others * groups;
}

static int stored_bytes(int t)
{
    switch (t) {
    case T_F32: return 4;
    case T_F64: return 8;
    case T_C32: return 8;
    case T_C64: return 16;
    default: return 2;
    }
}

static bool one_operand_lacks(const GenParams& g, int j) { return (g.F_sA[j] == 0) != (g.F_sB[j] == 0); }

// Rows per thread of k_element_rows, or 1: a mode that one
// operand lacks, other than the walk's first one (whose neighbours the lanes
// of a warp read), and of several the one along which D is nearest; where
// only the first one qualifies, spread over it as long as 8 neighbours are
// left to the lanes (32 bytes of binary32). 8 or 4 rows as long as the threads
// fill the GPU about once (148 x 1024) and the mode more than half a group: the
// rows it lacks still cost loads (modes of 4, against one output a thread: 8
// rows 0.70 to 1.43, 4 rows 1.05 to 1.76; modes of 2: 4 rows 0.83 to 1.6, one
// row 1.04 and more).
static int thread_rows(GenParams& g, RowGroup& q)
{
    if (g.nUA || g.nUB || g.sizeK < 1) return 1;
    int best = -1;
    auto a = [](int64_t x) { return x < 0 ? -x : x; };
    for (int j = 1; j < g.nF; j++)
        if (one_operand_lacks(g, j) && 2 * g.F_ext[j] > 4 && (best < 0 || a(g.F_sD[j]) < a(g.F_sD[best]))) best = j;
    const bool spread = best < 0;
    if (spread) {
        if (g.nF < 1 || !one_operand_lacks(g, 0)) return 1;
        best = 0;
    }
    const int64_t e = g.F_ext[best], others = g.sizeF / e;
    for (int nr = 8; nr >= 4; nr /= 2) {
        const int64_t groups = (e + nr - 1) / nr;
        if (2 * e <= nr || others * groups < 148 * 1024 || (spread && groups < 8)) continue;
        group_rows(g, q, best, nr, spread);
        return nr;
    }
    return 1;
}

// Rows per warp of k_warp_rows, or 1: 8 or 4 rows as long as 8 warps per SM
// have work and the mode fills half a group; of the modes that one operand
// lacks the one with the fewest loads (a group's NR of the varying operand and
// one of the shared, over rounds of the 16 warps per SM that run at a time),
// of equal ones the nearest in D.
// One row where unary modes are longer than the offset tables: a group would
// step through them row by row, with one row's loads in flight (133 unary
// values, 51 terms, 5664 outputs 231 us in k_warpdot, 322 in groups of 4); and
// where a lane reads runs of 64 bytes and more along one: the 32 lanes' lines of
// 8 rows do not stay in L1 (75 contiguous complex values, 26 terms, 18513 outputs
// 235 us in k_warpdot, 710 in groups of 8, below 200 with one row).
static int warp_rows(GenParams& g, RowGroup& q)
{
    auto long_runs = [](int n, const int64_t* ext, const int64_t* str, int t) {
        return n > 0 && (str[0] == 1 || str[0] == -1) && ext[0] * stored_bytes(t) >= 64;
    };
    if (!u_tabled(g) || long_runs(g.nUA, g.UA_ext, g.UA_s, g.tA) || long_runs(g.nUB, g.UB_ext, g.UB_s, g.tB)) return 1;
    auto a = [](int64_t x) { return x < 0 ? -x : x; };
    for (int nr = 8; nr >= 4; nr /= 2) {
        int best = -1;
        double best_cost = 0;
        for (int j = 0; j < g.nF; j++) {
            const int64_t e = g.F_ext[j], groups = g.sizeF / e * ((e + nr - 1) / nr);
            if (!one_operand_lacks(g, j) || 2 * e < nr || groups < 148 * 8) continue;
            const double uv = (double)(g.F_sA[j] ? g.sizeUA : g.sizeUB), us = (double)(g.F_sA[j] ? g.sizeUB : g.sizeUA);
            const double cost = (double)((groups + 148 * 16 - 1) / (148 * 16)) * (nr * uv + us);
            if (best < 0 || cost < best_cost || (cost == best_cost && a(g.F_sD[j]) < a(g.F_sD[best]))) {
                best = j;
                best_cost = cost;
            }
        }
        if (best < 0) continue;
        group_rows(g, q, best, nr, false);
        return nr;
    }
    return 1;
}

// How the row kernels would load the operands of a product computed in the
// type of storage `stored`.
static int loads_of(const GenParams& g, int stored)
{
    if (g.tA == stored && g.tB == stored) return NATIVE;
    return stored == T_F32 && g.tA >= T_F16 && g.tB >= T_F16 ? STORED16 : ANY;
}

// Rows per step of the row kernels, g then in groups, or 0: one output at a
// time. A single term without a mode to group by gains nothing from the offset
// tables and pays for filling them (binary32, 889200 outputs 12.1 us without,
// 14.6 with; 0.97 on average over 283 products, 0.81 at worst), and a rounded
// complex one nothing from groups (3.9 million outputs 64 us one by one, 77 in
// groups of 8). Unary modes beyond the tables, rounded or of 16 bits, convert
// one value after the other whichever kernel sums them, and the tables' shared
// memory is missing from L1 (135 rounded complex values, 36 terms, 7350 outputs
// 293 us in k_warpdot, 655 in k_warp_rows).
static int rows_of_step(GenParams& g, RowGroup& q, int loads)
{
    if (loads == ANY || (!u_tabled(g) && (loads == STORED16 || g.round_in != TB_ROUND_NONE))) return 0;
    if (g.warp) return warp_rows(g, q);
    const bool one_term = g.sizeK == 1 && !g.nUA && !g.nUB;
    if (one_term && g.tA == T_C32 && g.round_in != TB_ROUND_NONE) return 0;
    const int nr = thread_rows(g, q);
    return nr == 1 && one_term ? 0 : nr;
}

template <typename R, bool CPLX, int LOADS>
static void launch_rows(const GenParams& g, const RowGroup& q, int nr, const tb_ptrs* d, cudaStream_t s)
{
    const int per = g.warp ? 4 : 256, threads = g.warp ? 128 : 256;  // groups and threads of a block
    int64_t blocks = (g.sizeF + per - 1) / per;
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    void (*kern)(GenParams, RowGroup, const void*, const void*, const void*, void*);
    if (g.warp && (g.nUA || g.nUB))
        kern = nr == 8 ? k_warp_rows<R, CPLX, LOADS, 8, true>
               : nr == 4 ? k_warp_rows<R, CPLX, LOADS, 4, true> : k_warp_rows<R, CPLX, LOADS, 1, true>;
    else if (g.warp)
        kern = nr == 8 ? k_warp_rows<R, CPLX, LOADS, 8, false>
               : nr == 4 ? k_warp_rows<R, CPLX, LOADS, 4, false> : k_warp_rows<R, CPLX, LOADS, 1, false>;
    else
        kern = nr == 8 ? k_element_rows<R, CPLX, LOADS, 8>
               : nr == 4 ? k_element_rows<R, CPLX, LOADS, 4> : k_element_rows<R, CPLX, LOADS, 1>;
    kern<<<(unsigned)blocks, threads, 0, s>>>(g, q, q.swapped ? d->B : d->A, q.swapped ? d->A : d->B, d->C, d->D);
}

template <typename R, bool CPLX>
static cudaError_t launch_typed(GenParams& g, int path, const tb_ptrs* d, cudaStream_t s)
{
    constexpr int stored = sizeof(R) == 4 ? (CPLX ? T_C32 : T_F32) : (CPLX ? T_C64 : T_F64);
    if (path == TB_PATH_REDUCE && g.sizeK < (1ll << 31)) {
        const int S = reduce_chunks(g.sizeF, g.sizeK);
        int64_t bx = g.sizeF < 148 * 16 ? g.sizeF : 148 * 16;
        if (bx < 1) bx = 1;
        if (S == 1) {
            k_reduce<R, CPLX><<<(unsigned)bx, 256, 0, s>>>(g, d->A, d->B, d->C, d->D, g.sizeK, (R*)nullptr);
            count_launch();
            return cudaGetLastError();
        }
        const int64_t chunk = (g.sizeK + S - 1) / S;
        const int chunks = (int)((g.sizeK + chunk - 1) / chunk);
        void* ws = nullptr;
        cudaError_t e = pool_alloc(&ws, (size_t)chunks * (size_t)g.sizeF * 2 * sizeof(R), s);
        if (e != cudaSuccess) return e;
        k_reduce<R, CPLX><<<dim3((unsigned)bx, (unsigned)chunks), 256, 0, s>>>(g, d->A, d->B, d->C, d->D, chunk,
                                                                            (R*)ws);
        e = cudaGetLastError();
        if (e == cudaSuccess) {
            int64_t b2 = (g.sizeF + 255) / 256;
            if (b2 > 148 * 8) b2 = 148 * 8;
            k_reduce_final<R, CPLX><<<(unsigned)b2, 256, 0, s>>>(g, d->C, d->D, chunks, (const R*)ws);
            e = cudaGetLastError();
        }
        count_launch(2);
        cudaFreeAsync(ws, s);
        return e;
    }
    const uintptr_t pair = CPLX ? 2 * sizeof(R) : 1;  // complex pairs are loaded whole
    const bool aligned = (uintptr_t)d->A % pair == 0 && (uintptr_t)d->B % pair == 0;
    const int loads = aligned ? loads_of(g, stored) : ANY;
    RowGroup q;
    memset(&q, 0, sizeof(q));
    const int nr = rows_of_step(g, q, loads);
    if (nr == 0) {
        const int per = g.warp ? 8 : 256;  // outputs of a block
        const int64_t most = 148 * (g.warp ? 32 : 64), blocks = std::max<int64_t>(1, std::min((g.sizeF + per - 1) / per, most));
        (g.warp ? k_warpdot<R, CPLX> : k_elementwise<R, CPLX>)<<<(unsigned)blocks, 256, 0, s>>>(g, d->A, d->B, d->C, d->D);
    } else if (loads == NATIVE) {
        launch_rows<R, CPLX, NATIVE>(g, q, nr, d, s);
    } else if constexpr (sizeof(R) == 4 && !CPLX) {
        launch_rows<R, CPLX, STORED16>(g, q, nr, d, s);
    }
    count_launch();
    return cudaGetLastError();
}

size_t group_descriptor_bytes(int n)
{
    return (size_t)n * sizeof(GenParams) + (size_t)n * sizeof(tb_ptrs) + (size_t)(n + 1) * sizeof(int64_t) + 64;
}

// Fills `host` (pinned, group_descriptor_bytes(n)) with the descriptors of n
// products of one compute domain, copies it to `dev` and launches one grouped
// kernel. The host buffer must stay untouched until the copy has run.
cudaError_t launch_generic_group(const tb_plan* const* P, const tb_ptrs* d, int n, void* host, void* dev,
                                 cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    char* h = (char*)host;
    GenParams* hp = (GenParams*)h;
    tb_ptrs* hq = (tb_ptrs*)(h + (size_t)n * sizeof(GenParams));
    int64_t* hf = (int64_t*)(h + (size_t)n * (sizeof(GenParams) + sizeof(tb_ptrs)));
    int64_t blocks = 0;
    for (int j = 0; j < n; j++) {
        fill_params(P[j], hp[j]);
        hq[j] = d[j];
        hf[j] = blocks;
        // warp-per-output products: 8 outputs per block
        int64_t b = hp[j].warp ? (P[j]->F.size + 7) / 8 : (P[j]->F.size + 255) / 256;
        if (b > 148 * 8) b = 148 * 8;
        if (b < 1) b = 1;
        blocks += b;
    }
    hf[n] = blocks;
    const size_t bytes = group_descriptor_bytes(n);
    cudaError_t e = cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    char* dv = (char*)dev;
    const GenParams* dp = (const GenParams*)dv;
    const tb_ptrs* dq = (const tb_ptrs*)(dv + (size_t)n * sizeof(GenParams));
    const int64_t* df = (const int64_t*)(dv + (size_t)n * (sizeof(GenParams) + sizeof(tb_ptrs)));
    if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
    switch (P[0]->compute) {
    case TB_R32: k_elementwise_group<float, false><<<(unsigned)blocks, 256, 0, s>>>(dp, dq, df, n); break;
    case TB_R64: k_elementwise_group<double, false><<<(unsigned)blocks, 256, 0, s>>>(dp, dq, df, n); break;
    case TB_C32: k_elementwise_group<float, true><<<(unsigned)blocks, 256, 0, s>>>(dp, dq, df, n); break;
    default: k_elementwise_group<double, true><<<(unsigned)blocks, 256, 0, s>>>(dp, dq, df, n); break;
    }
    count_launch();
    return cudaGetLastError();
}

// Copy of one operand (its free, contracted and unary modes) into a dense
// buffer whose first mode is the first output mode and whose other modes
// follow in free, contracted, unary order, so that the element kernel reads
// it along its walk of the outputs instead of one line per lane. Element
// values are copied as stored (2-byte elements, or 4-byte words).
struct StageParams {
    const unsigned char* src;
    unsigned char* dst;
    int32_t n, words;  // modes; 4-byte words per element (0: one 2-byte element)
    int64_t size;
    int64_t s[3 * TB_MAXMODES];  // source strides, in elements
    FastDiv f[3 * TB_MAXMODES];
};

__global__ void __launch_bounds__(256) k_stage(StageParams p)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.size; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t r = (uint32_t)i;
        int64_t o = 0;
        for (int j = 0; j < p.n; j++) {
            const uint32_t q = fdiv(r, p.f[j]);
            o += (int64_t)(r - q * p.f[j].d) * p.s[j];
            r = q;
        }
        if (p.words == 0) {
            ((uint16_t*)p.dst)[i] = __ldg((const uint16_t*)p.src + o);
        } else {
            for (int w = 0; w < p.words; w++)
                ((uint32_t*)p.dst)[i * p.words + w] = __ldg((const uint32_t*)p.src + o * p.words + w);
        }
    }
}

// The operand `side` (0 A, 1 B) of the element path copied into scratch in
// the order of the output walk; g's strides and d's pointer then refer to
// the copy. *ws: the scratch, to be freed after the element kernel.
static cudaError_t stage_operand(const tb_plan* P, int side, GenParams& g, tb_ptrs& d, void** ws, cudaStream_t s)
{
    StageParams sp;
    memset(&sp, 0, sizeof(sp));
    int64_t* F_s = side ? g.F_sB : g.F_sA;
    int64_t* K_s = side ? g.K_sB : g.K_sA;
    int64_t* U_s = side ? g.UB_s : g.UA_s;
    const tb_modes& U = side ? P->UB : P->UA;
    int n = 0;
    int64_t acc = 1;
    auto add = [&](int64_t ext, int64_t& stride) {
        sp.s[n] = stride;
        sp.f[n] = make_fastdiv((uint32_t)ext);
        n++;
        stride = acc;
        acc *= ext;
    };
    for (int j = 0; j < P->F.n; j++)
        if (F_s[j] != 0) add(P->F.ext[j], F_s[j]);
    for (int j = 0; j < P->K.n; j++) add(P->K.ext[j], K_s[j]);
    for (int j = 0; j < U.n; j++) add(U.ext[j], U_s[j]);
    if (acc >= (1ll << 31)) return cudaErrorInvalidValue;
    const int tY = side ? P->tB : P->tA;
    const int eb = stored_bytes(tY);
    sp.n = n;
    sp.words = eb / 4;
    sp.size = acc;
    sp.src = (const unsigned char*)(side ? d.B : d.A);
    cudaError_t e = pool_alloc(ws, (size_t)acc * (size_t)eb, s);
    if (e != cudaSuccess) return e;
    sp.dst = (unsigned char*)*ws;
    int64_t blocks = (acc + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_stage<<<(unsigned)blocks, 256, 0, s>>>(sp);
    count_launch();
    if (side) d.B = *ws;
    else d.A = *ws;
    return cudaGetLastError();
}

cudaError_t launch_generic(const tb_plan* P, const tb_ptrs* d, cudaStream_t s, int* kernels)
{
    GenParams g;
    fill_params(P, g);
    *kernels = 1;
    tb_ptrs dd = *d;
    void* ws = nullptr;
    if (P->path == TB_PATH_GENERIC && P->elem_stage && !g.warp) {
        cudaError_t e = stage_operand(P, P->elem_stage - 1, g, dd, &ws, s);
        if (e != cudaSuccess) {
            if (ws) cudaFreeAsync(ws, s);
            return e;
        }
        *kernels = 2;
    }
    cudaError_t e = cudaErrorInvalidValue;
    switch (P->compute) {
    case TB_R32: e = launch_typed<float, false>(g, P->path, &dd, s); break;
    case TB_R64: e = launch_typed<double, false>(g, P->path, &dd, s); break;
    case TB_C32: e = launch_typed<float, true>(g, P->path, &dd, s); break;
    case TB_C64: e = launch_typed<double, true>(g, P->path, &dd, s); break;
    }
    if (ws) cudaFreeAsync(ws, s);
    return e;
}

}  // namespace tb

// ---------------------------------------------------------------------------
// Device-resident request loop (host side: host/loop.c). A persistent kernel
// of G blocks serves small products as they arrive, without a launch per
// product. The host writes product t's descriptor into slot t % R of a ring
// in page-locked host memory mapped into the device, then the slot's
// sequence word (t + 1) last. Block 0 polls that word (system-scope acquire
// loads, a short sleep between polls), copies the descriptor into the same
// slot of a ring in device memory and raises its device sequence word; the
// other blocks poll the device word (an L2 read instead of a PCIe read).
// Every block then computes its share of D's elements (element i on block
// i / 256 mod G) with the element kernel's own per-output function, so the
// bits equal TAPP_execute_product's on the element path; the last block to
// finish (an arrival counter per slot) publishes t + 1 in the host slot's
// completion word after a system fence. A block that sees no new product for
// idle_ns stores the ticket it waits for in device memory and returns, so
// the loop never spins without a bound; the host relaunches it when
// products arrive again and the last launch has ended.
namespace tb {

struct LoopSlot {
    GenParams p;
    tb_ptrs q;
    int32_t compute;
    int32_t warp;    // 1: one warp per output (the kernel TAPP_execute_product would run)
    int64_t seq;     // t + 1 once the descriptor of ticket t is complete (written last)
    int64_t done;    // t + 1 once ticket t's D is written
    int64_t pad2[6];
};

struct LoopParams {
    LoopSlot* slots;      // device pointer of the mapped ring
    LoopSlot* dslots;     // ring in device memory: block 0's copies
    int64_t* dseq;        // device memory: t + 1 once dslots[t % R] holds ticket t
    int* arrive;          // device memory: blocks done with the slot's current ticket
    int64_t* next;        // device memory: per block, the ticket it serves next
    int32_t nslots;
    int32_t pad;
    unsigned long long idle_ns;
};

__device__ __forceinline__ unsigned long long loop_now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ int64_t ld_acquire_sys(const int64_t* p)
{
    int64_t v;
    asm volatile("ld.acquire.sys.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int64_t ld_acquire_gpu(const int64_t* p)
{
    int64_t v;
    asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_sys(int64_t* p, int64_t v)
{
    asm volatile("st.release.sys.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void st_release_gpu(int64_t* p, int64_t v)
{
    asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <typename R, bool CPLX>
__device__ __forceinline__ void loop_product(const GenParams& p, const tb_ptrs& q, int warp)
{
    if (warp) {
        const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
        for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < p.sizeF; i += warps)
            warp_element<R, CPLX, UNARY_LOADS<R, CPLX>>(p, q.A, q.B, q.C, q.D, i, threadIdx.x & 31);
        return;
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.sizeF; i += stride)
        element<R, CPLX, UNARY_LOADS<R, CPLX>>(p, q.A, q.B, q.C, q.D, i);
}

// three blocks an SM: 80 registers. Left to itself the compiler held the four
// products' code in 64 and spilled 452 bytes.
__global__ void __launch_bounds__(256, 3) k_request_loop(LoopParams lp)
{
    __shared__ GenParams sp;
    __shared__ tb_ptrs sq;
    __shared__ int scomp, swarp, go;
    const int b = blockIdx.x;
    int64_t t = lp.next[b];
    unsigned long long last = loop_now_ns();
    for (;;) {
        const int64_t s = t % lp.nslots;
        LoopSlot* hs = &lp.slots[s];
        LoopSlot* ds = &lp.dslots[s];
        if (threadIdx.x == 0) {
            // block 0 watches the host ring, the others the device copy
            const int64_t* word = b == 0 ? &hs->seq : &lp.dseq[s];
            int posted = 0;
            for (;;) {
                if ((b == 0 ? ld_acquire_sys(word) : ld_acquire_gpu(word)) == t + 1) {
                    posted = 1;
                    break;
                }
                if (loop_now_ns() - last > lp.idle_ns) break;
                __nanosleep(b == 0 ? 256 : 128);
            }
            go = posted;
        }
        __syncthreads();
        if (!go) break;
        {
            // the descriptor into shared memory: from host memory on block 0
            // (which also fills the device copy), from the device copy elsewhere
            const volatile int64_t* src = (const volatile int64_t*)(b == 0 ? &hs->p : &ds->p);
            int64_t* dst = (int64_t*)&sp;
            int64_t* dcopy = (int64_t*)&ds->p;
            for (int w = threadIdx.x; w < (int)(sizeof(GenParams) / 8); w += blockDim.x) {
                const int64_t v = src[w];
                dst[w] = v;
                if (b == 0) dcopy[w] = v;
            }
            if (threadIdx.x == 0) {
                const volatile tb_ptrs* vq = b == 0 ? &hs->q : &ds->q;
                sq.A = vq->A;
                sq.B = vq->B;
                sq.C = vq->C;
                sq.D = vq->D;
                scomp = *(const volatile int32_t*)(b == 0 ? &hs->compute : &ds->compute);
                swarp = *(const volatile int32_t*)(b == 0 ? &hs->warp : &ds->warp);
                if (b == 0) {
                    ds->q = sq;
                    ds->compute = scomp;
                    ds->warp = swarp;
                }
            }
        }
        __syncthreads();
        if (b == 0 && threadIdx.x == 0) {
            __threadfence();
            st_release_gpu(&lp.dseq[s], t + 1);  // the device copy is complete
        }
        switch (scomp) {
        case TB_R32: loop_product<float, false>(sp, sq, swarp); break;
        case TB_R64: loop_product<double, false>(sp, sq, swarp); break;
        case TB_C32: loop_product<float, true>(sp, sq, swarp); break;
        default: loop_product<double, true>(sp, sq, swarp); break;
        }
        __syncthreads();  // this block's outputs of the product written
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&lp.arrive[s], 1) == (int)gridDim.x - 1) {
                // the last block: every output is written
                lp.arrive[s] = 0;
                __threadfence_system();
                st_release_sys(&hs->done, t + 1);
            }
        }
        t++;
        last = loop_now_ns();
    }
    if (threadIdx.x == 0) lp.next[b] = t;
}

size_t loop_slot_bytes() { return sizeof(LoopSlot); }

// Fills ring slot `slot` (host memory) with a product's descriptor, all
// but the sequence word.
void loop_fill(void* slot, const tb_plan* P, const tb_ptrs* d)
{
    LoopSlot* s = (LoopSlot*)slot;
    fill_params(P, s->p);
    if (P->path == TB_PATH_NOOP) s->p.sizeF = 0;  // nothing to write (empty D, or a precision left as is)
    s->q = *d;
    s->compute = P->compute;
    s->warp = s->p.warp;
}

// device state of a loop: the ring copy, its sequence words, the arrival
// counters and the per-block tickets (zeroed; every block starts at ticket 0)
size_t loop_state_bytes(int nslots, int blocks)
{
    return (size_t)nslots * (sizeof(LoopSlot) + sizeof(int64_t) + sizeof(int)) + (size_t)blocks * sizeof(int64_t) + 64;
}

cudaError_t loop_launch(void* slots_dev, void* state, int nslots, int blocks, unsigned long long idle_ns,
                        cudaStream_t s)
{
    LoopParams lp;
    char* st = (char*)state;
    lp.slots = (LoopSlot*)slots_dev;
    lp.dslots = (LoopSlot*)st;
    lp.dseq = (int64_t*)(st + (size_t)nslots * sizeof(LoopSlot));
    lp.next = lp.dseq + nslots;
    lp.arrive = (int*)(lp.next + blocks);
    lp.nslots = nslots;
    lp.pad = 0;
    lp.idle_ns = idle_ns;
    k_request_loop<<<blocks, 256, 0, s>>>(lp);
    count_launch();
    return cudaGetLastError();
}

}  // namespace tb

// Kernel of the element path for a plan: 0 threads, 1 warps. *rows: outputs of
// a step along a mode (0: no row kernel), *spread and *swapped: RowGroup's, for
// operands aligned to their elements. No device call.
extern "C" int tbk_generic_kernel(const tb_plan* P, int* rows, int* spread, int* swapped)
{
    static const int stored[4] = {T_F32, T_F64, T_C32, T_C64};  // by TB_R32 .. TB_C64
    tb::GenParams g;
    tb::fill_params(P, g);
    tb::RowGroup q;
    memset(&q, 0, sizeof(q));
    *rows = tb::rows_of_step(g, q, tb::loads_of(g, stored[P->compute]));
    *spread = q.spread;
    *swapped = q.swapped;
    return g.warp;
}
