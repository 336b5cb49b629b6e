// Launch parameters of the CUDA-core products in their turned L/M/N/K view
// (simt.cu), shared with the tiled GEMM (tile.cu).
#pragma once

#include "tb_common.cuh"

namespace tb {
namespace simt {

struct Modes {
    int32_t n, pad;
    int64_t ext[TB_MAXMODES];
    int64_t s0[TB_MAXMODES];
    int64_t s1[TB_MAXMODES];
};

struct Params {
    const void* A;
    const void* B;
    const void* C;
    void* D;
    int32_t tA, tB, tC, tD, round_in, beta_zero, a_rows_fast, b_rows_fast;
    int64_t M, N, K, L;
    double alpha, beta, alpha_im, beta_im;
    int32_t conjA, conjB, conjC, conjD, conjD_f32, d_rows_fast;
    Modes am, ak, al;  // A: rows (M), contraction, batch (s0 = stride in A)
    Modes bn, bk, bl;  // B: rows (N), contraction, batch (s0 = stride in B)
    Modes cm, cn, cl;  // C (s0) and D (s1) strides of M, N, L modes
    int32_t tiles_m, tiles_n;
    int64_t k_chunk;   // contraction length of one split (multiple of BK)
    void* ws;          // split sums [split][l][m][n][plane], or NULL: epilogue in place
    int32_t a_vec, b_vec;  // operand read 16 bytes at a time (see vec_side)
};

// D = op_D(alpha * acc + beta * op_C(C)) for one element whose C value
// (cr, ci) is already loaded (rounded, not yet conjugated)
template <typename T, bool CPLX, typename P>
__device__ __forceinline__ void epilogue_value(const P& p, T xr, T xi, T cr, T ci, T& out_r, T& out_i)
{
    const T ar = (T)p.alpha, ai = (T)p.alpha_im, br = (T)p.beta, bi = (T)p.beta_im;
    T vr = ar * xr - (CPLX ? ai * xi : (T)0);
    T vi = CPLX ? ar * xi + ai * xr : (T)0;
    if (!p.beta_zero) {
        if (p.conjC) ci = -ci;
        vr = fma(br, cr, vr);
        if (CPLX) {
            vr = fma(-bi, ci, vr);
            vi = fma(br, ci, fma(bi, cr, vi));
        }
    }
    if (p.conjD) {
        if (p.conjD_f32) {
            vr = (T)(float)vr;
            vi = (T)(float)vi;
        }
        vi = -vi;
    }
    out_r = vr;
    out_i = vi;
}

}  // namespace simt

// tile.cu: the tiled GEMM over asynchronous copies; its split sums stay within ws_limit bytes
bool tile_takes(const simt::Params& p, int compute);
// ... and whether it takes a product that the narrow kernels could run
bool tile_over_narrow(const simt::Params& p, int compute, int kind);
void tile_describe(const simt::Params& p, int compute, size_t ws_limit, int out[4]);
cudaError_t launch_tile(const simt::Params& p, int compute, size_t ws_limit, cudaStream_t s);

}  // namespace tb
