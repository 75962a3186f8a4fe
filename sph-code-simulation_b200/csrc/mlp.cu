// mlp.cu — tensor-core inference and training of the learned Riemann guess.
//
// Network (mlp.cuh): 5 scaled inputs (padded to 16) -> 64 -> 64 -> 64 -> 1,
// SiLU, BF16 weights / activations, FP32 accumulation.  Every matrix product
// is a warp-level mma.sync.m16n8k16 (bf16 x bf16 -> f32) on a 16-row tile:
//   * a layer's f32 accumulator fragments (two adjacent 8-column n-tiles) are
//     exactly the bf16 A-operand fragment of the next layer's k-tile, so the
//     three hidden layers stay in registers;
//   * training puts activations and dZ of a block's rows into shared memory,
//     and each warp sums its own part of dW = dZ^T A_prev in registers (the
//     transposed operands are read by ldmatrix.trans), one global add per
//     weight and block.
// Training keeps FP32 master parameters and Adam moments; the BF16 image the
// kernels read is rebuilt after every update.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>
#include <cuda_runtime.h>

#include "context.cuh"
#include "mlp.cuh"

namespace sphgpu {

namespace {

constexpr int LDW0 = 24;  // padded smem row lengths (bf16) for conflict-free fragment loads
constexpr int LDW = 72;

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ unsigned pack_bf16(f32x2 v)
{
    float lo, hi;
    unpack2(v, lo, hi);
    return pack_bf16(lo, hi);
}

__device__ __forceinline__ void mma16816(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma1688(float (&d)[4], unsigned a0, unsigned a1, unsigned b0)
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

// Four 8x8 bf16 matrices; the lane's address is row lane & 7 of matrix lane >> 3.
template <bool TRANS>
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], const __nv_bfloat16* row)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(row);
    if(TRANS) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    } else {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
    }
}

// Shared-memory copy of the network; the biases negated (SiLU takes -z).
struct __align__(16) SmemNet {
    __nv_bfloat16 w0[MLP_H * LDW0];
    __nv_bfloat16 w1[MLP_H * LDW];
    __nv_bfloat16 w2[MLP_H * LDW];
    float w3[MLP_H];
    float nb[3][MLP_H];
    float b3;
};

template <int THREADS>
__device__ __forceinline__ void load_net(SmemNet& s, const MlpDev& m)
{
    const uint4* w = reinterpret_cast<const uint4*>(m.w);   // 8 bf16 each
    for(int k = threadIdx.x; k < MLP_H * MLP_INP / 8; k += THREADS) {
        *reinterpret_cast<uint4*>(&s.w0[(k / 2) * LDW0 + (k % 2) * 8]) = __ldg(&w[IMG_W0 / 8 + k]);
    }
    for(int k = threadIdx.x; k < MLP_H * MLP_H / 8; k += THREADS) {
        *reinterpret_cast<uint4*>(&s.w1[(k / 8) * LDW + (k % 8) * 8]) = __ldg(&w[IMG_W1 / 8 + k]);
        *reinterpret_cast<uint4*>(&s.w2[(k / 8) * LDW + (k % 8) * 8]) = __ldg(&w[IMG_W2 / 8 + k]);
    }
    for(int k = threadIdx.x; k < MLP_H; k += THREADS) {
        s.w3[k] = m.f[IMGF_W3 + k];
        s.nb[0][k] = -m.f[IMGF_B0 + k];
        s.nb[1][k] = -m.f[IMGF_B1 + k];
        s.nb[2][k] = -m.f[IMGF_B2 + k];
    }
    if(threadIdx.x == 0) s.b3 = m.f[IMGF_B3];
}

// Two SiLUs of z = acc + bias, from the negated bias: z / (1 + exp(-z)).  With
// nz = -z and q = -1 / (1 + exp(-z)) every negation is in an operand, and two
// values share each packed operation.  The reciprocal is rcp.approx and one
// Newton step by fused operations, which rounds correctly for every argument
// from 1 on (each of the 2^23 significands compared with the division); the
// clamp keeps exp's overflow out of the step, where the result is 0 as before.
__device__ __forceinline__ f32x2 silu2(float acc0, float acc1, f32x2 nb, f32x2& nz, f32x2& q)
{
    const f32x2 one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
    nz = fma2(pack2(acc0, acc1), minus, nb);
    float z0, z1, x0, x1;
    unpack2(nz, z0, z1);
    unpack2(add2(pack2(__expf(z0), __expf(z1)), one), x0, x1);
    x0 = fminf(x0, FLT_MAX);
    x1 = fminf(x1, FLT_MAX);
    const f32x2 y = pack2(rcp_approx(-x0), rcp_approx(-x1));
    q = fma2(fma2(pack2(x0, x1), y, one), y, y);
    return mul2(nz, q);
}
// and the derivative s (1 + z (1 - s)) of the same pair, s = -q
__device__ __forceinline__ f32x2 dsilu2(f32x2 nz, f32x2 q)
{
    const f32x2 one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
    return mul2(q, fma2(nz, add2(q, one), minus));
}

// n-tile j of x W^T for a warp's 16-row tile: two reads of four 8x8 matrices
// cover K = 64.
__device__ __forceinline__ void ntile_mma(const __nv_bfloat16* w, int j, const unsigned (&act)[4][4], float (&c)[4],
                                          int lane)
{
    const __nv_bfloat16* row = w + (8 * j + (lane & 7)) * LDW + (lane >> 3) * 8;
    unsigned b[2][4];
    ldsm4<false>(b[0], row);
    ldsm4<false>(b[1], row + 32);
    c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
    for(int kk = 0; kk < 4; ++kk) {
        mma16816(c, act[kk][0], act[kk][1], act[kk][2], act[kk][3], b[kk >> 1][2 * (kk & 1)],
                 b[kk >> 1][2 * (kk & 1) + 1]);
    }
}

constexpr int IBLK = 128;
constexpr int IRES = 5;   // resident blocks per SM (4: 370 us, 6: 373, both for 3 M rows)

// y[row] for feature rows (8 bf16 per row, 5 used).
//
// Bound by the special-function unit: a row takes 192 exponentials and 192
// reciprocals, 24 cycles of an SM, against 10 of its tensor unit (measured: 78 %
// and 29 % busy, 34 cycles a row).  The products therefore stay on the
// warp-level form, whose accumulators are in registers where SiLU needs them,
// and the 20 KB of weights are loaded once per resident block: 3 M rows 626 us
// (16 blocks per SM, 4-byte fragment loads, two branches around each reciprocal)
// -> 363.  Two 16-row tiles per warp (half the weight reads) were slower, 424.
__global__ void __launch_bounds__(IBLK, IRES) k_mlp_infer(MlpDev m, const uint4* __restrict__ feat,
                                                          float* __restrict__ y, long long rows)
{
    __shared__ SmemNet s;
    load_net<IBLK>(s, m);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long warp = ((long long)blockIdx.x * IBLK + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * IBLK) >> 5;
    const unsigned* x = reinterpret_cast<const unsigned*>(feat);
    for(long long base = warp * 16; base < rows; base += nwarps * 16) {
        const long long lo = base + g, hi = lo + 8;
        const unsigned x_lo = lo < rows ? __ldg(&x[4 * lo + t]) : 0u, x_hi = hi < rows ? __ldg(&x[4 * hi + t]) : 0u;
        // n-tile by n-tile through each layer: a tile's accumulators go straight
        // through SiLU into the next layer's operand
        unsigned act[4][4];
        float ylo = 0.f, yhi = 0.f;
#pragma unroll
        for(int layer = 0; layer < 3; ++layer) {
            const __nv_bfloat16* w = layer == 1 ? s.w1 : s.w2;
            unsigned next[4][4], b0[4];
#pragma unroll
            for(int j = 0; j < 8; ++j) {
                float c[4] = {0.f, 0.f, 0.f, 0.f};
                if(layer == 0) {
                    if((j & 3) == 0) ldsm4<false>(b0, s.w0 + (8 * j + lane) * LDW0);
                    mma1688(c, x_lo, x_hi, b0[j & 3]);
                } else {
                    ntile_mma(w, j, act, c, lane);
                }
                const f32x2 nb = *reinterpret_cast<const f32x2*>(&s.nb[layer][8 * j + 2 * t]);
                f32x2 nz, q;
                const f32x2 alo = silu2(c[0], c[1], nb, nz, q), ahi = silu2(c[2], c[3], nb, nz, q);
                if(layer < 2) {
                    next[j >> 1][2 * (j & 1)] = pack_bf16(alo);
                    next[j >> 1][2 * (j & 1) + 1] = pack_bf16(ahi);
                } else {   // output: y = a3 . w3 + b3
                    const float wl = s.w3[8 * j + 2 * t], wh = s.w3[8 * j + 2 * t + 1];
                    float a0, a1;
                    unpack2(alo, a0, a1);
                    ylo += a0 * wl + a1 * wh;
                    unpack2(ahi, a0, a1);
                    yhi += a0 * wl + a1 * wh;
                }
            }
            if(layer == 2) break;
#pragma unroll
            for(int e = 0; e < 16; ++e) act[e / 4][e % 4] = next[e / 4][e % 4];
        }
        // reduced over the 4 lanes of a row group
        ylo += __shfl_xor_sync(FULL_MASK, ylo, 1);
        ylo += __shfl_xor_sync(FULL_MASK, ylo, 2);
        yhi += __shfl_xor_sync(FULL_MASK, yhi, 1);
        yhi += __shfl_xor_sync(FULL_MASK, yhi, 2);
        if(t == 0) {
            if(lo < rows) y[lo] = ylo + s.b3;
            if(hi < rows) y[hi] = yhi + s.b3;
        }
    }
}

// --------------------------------------------------------------- training
// A block takes TROWS rows at a time, 16 per warp: forward and backward of the
// warp's own rows in registers, activations and dZ to shared memory (bf16, the
// operands' own precision), then every warp sums dW of its own 16 outputs x 32
// inputs of both 64 x 64 matrices over the block's rows, in registers until the
// block's end.  (Summing each 16-row product into shared memory by f32 atomics
// instead took 1.59 ms for 500 K rows; 0.19 now, bound by the latency of 8 warps
// per SM, each with 255 registers of forward state.)
constexpr int TBLK = 256;
constexpr int TROWS = TBLK / 2;

struct __align__(16) SmemTrain {
    SmemNet net;
    __nv_bfloat16 act[2][TROWS * LDW];   // outputs of layers 0, 1
    __nv_bfloat16 dz[3][TROWS * LDW];    // dLoss / dZ of layers 0 .. 2
    __nv_bfloat16 x[TROWS * 8];          // inputs
    float part[TBLK / 32][4 * MLP_H];    // per warp: gradients of b0, b1, b2, w3
    float part0[TBLK / 32][2];           // of b3, and the loss
};

// Column sums over a warp's 16 rows: dz[j][e] of a C fragment; lane (g, t) ends
// with the sums of columns 8 g + 2 t, + 1 (each exchange halves the columns).
__device__ __forceinline__ void column_sums(const float (&v)[8][2], float (&out)[2], int lane)
{
    float w4[4][2], w2[2][2];
    const bool u4 = lane & 16, u3 = lane & 8, u2 = lane & 4;
#pragma unroll
    for(int j = 0; j < 4; ++j) {
#pragma unroll
        for(int h = 0; h < 2; ++h) {
            const float mine = u4 ? v[j + 4][h] : v[j][h], other = u4 ? v[j][h] : v[j + 4][h];
            w4[j][h] = mine + __shfl_xor_sync(FULL_MASK, other, 16);
        }
    }
#pragma unroll
    for(int j = 0; j < 2; ++j) {
#pragma unroll
        for(int h = 0; h < 2; ++h) {
            const float mine = u3 ? w4[j + 2][h] : w4[j][h], other = u3 ? w4[j][h] : w4[j + 2][h];
            w2[j][h] = mine + __shfl_xor_sync(FULL_MASK, other, 8);
        }
    }
#pragma unroll
    for(int h = 0; h < 2; ++h) {
        const float mine = u2 ? w2[1][h] : w2[0][h], other = u2 ? w2[0][h] : w2[1][h];
        out[h] += mine + __shfl_xor_sync(FULL_MASK, other, 4);
    }
}

// Fragments of a 16 x 64 tile to rows r0 .. r0 + 15 of a shared-memory matrix.
__device__ __forceinline__ void store_frag(__nv_bfloat16* m, int r0, const unsigned (&f)[4][4], int g, int t)
{
    unsigned* lo = reinterpret_cast<unsigned*>(m + (r0 + g) * LDW) + t;
    unsigned* hi = reinterpret_cast<unsigned*>(m + (r0 + g + 8) * LDW) + t;
#pragma unroll
    for(int kk = 0; kk < 4; ++kk) {
        lo[8 * kk] = f[kk][0];
        hi[8 * kk] = f[kk][1];
        lo[8 * kk + 4] = f[kk][2];
        hi[8 * kk + 4] = f[kk][3];
    }
}

// dw[o][i] += sum_r dz[r][o] act[r][i] over the block's rows, for the warp's
// outputs o0 .. o0 + 15 and inputs i0 .. i0 + 31; each 16-row product is summed
// outside the tensor unit (round to nearest).
__device__ __forceinline__ void weight_sums(const __nv_bfloat16* dz, const __nv_bfloat16* act, int o0, int i0,
                                            float (&dw)[4][4], int lane)
{
    const int q = lane >> 3, r = lane & 7;
    const __nv_bfloat16* pa = dz + (r + (q >> 1) * 8) * LDW + o0 + (q & 1) * 8;
    const __nv_bfloat16* pb = act + (r + (q & 1) * 8) * LDW + i0 + (q >> 1) * 8;
#pragma unroll 2
    for(int k = 0; k < TROWS; k += 16) {
        unsigned a[4];
        ldsm4<true>(a, pa + k * LDW);
#pragma unroll
        for(int h = 0; h < 2; ++h) {
            unsigned b[4];
            ldsm4<true>(b, pb + k * LDW + 16 * h);
#pragma unroll
            for(int e = 0; e < 2; ++e) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma16816(d, a[0], a[1], a[2], a[3], b[2 * e], b[2 * e + 1]);
#pragma unroll
                for(int c = 0; c < 4; ++c) dw[2 * h + e][c] += d[c];
            }
        }
    }
}

// One training batch: rows r = perm(batch_base + k), k < bsize; loss = mean
// of (y - target)^2 over the batch.  Gradients are summed into grad (global).
__global__ void __launch_bounds__(TBLK, 1) k_mlp_train(MlpDev m, const uint4* __restrict__ feat,
                                                       const float* __restrict__ target, long long nrows,
                                                       long long batch_base, int bsize, unsigned long long pa,
                                                       unsigned long long pc, float* __restrict__ grad,
                                                       float* __restrict__ loss)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemTrain& s = *reinterpret_cast<SmemTrain*>(smem_raw);
    load_net<TBLK>(s.net, m);
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warp = threadIdx.x >> 5;
    const int r0 = warp * 16;                                  // the warp's rows of the tile
    const int o0 = (warp & 3) * 16, i0 = (warp >> 2) * 32;     // and its part of the weights
    const float inv_b = 1.0f / (float)bsize;
    const unsigned* x = reinterpret_cast<const unsigned*>(feat);
    float dw1[4][4] = {}, dw2[4][4] = {}, dw0[4] = {};
    float gb[4][2] = {};   // column sums for b0, b1, b2, w3
    float gb3 = 0.f, gloss = 0.f;
    for(long long base = (long long)blockIdx.x * TROWS; base < bsize; base += (long long)gridDim.x * TROWS) {
        const long long k_lo = base + r0 + g, k_hi = k_lo + 8;
        const bool v_lo = k_lo < bsize, v_hi = k_hi < bsize;
        const long long r_lo = v_lo ? (long long)((pa * (unsigned long long)(batch_base + k_lo) + pc) % nrows) : 0;
        const long long r_hi = v_hi ? (long long)((pa * (unsigned long long)(batch_base + k_hi) + pc) % nrows) : 0;
        const float t_lo = __ldg(&target[r_lo]), t_hi = __ldg(&target[r_hi]);
        const unsigned ax[2] = {v_lo ? __ldg(&x[4 * r_lo + t]) : 0u, v_hi ? __ldg(&x[4 * r_hi + t]) : 0u};
        reinterpret_cast<unsigned*>(s.x)[(r0 + g) * 4 + t] = ax[0];
        reinterpret_cast<unsigned*>(s.x)[(r0 + g + 8) * 4 + t] = ax[1];
        float c[8][4], a3[8][4], ds[3][8][4];
        unsigned act[4][4];
#pragma unroll
        for(int layer = 0; layer < 3; ++layer) {
            const __nv_bfloat16* w = layer == 1 ? s.net.w1 : s.net.w2;
            unsigned next[4][4], b0[4];
#pragma unroll
            for(int j = 0; j < 8; ++j) {
                float z[4] = {0.f, 0.f, 0.f, 0.f};
                if(layer == 0) {
                    if((j & 3) == 0) ldsm4<false>(b0, s.net.w0 + (8 * j + lane) * LDW0);
                    mma1688(z, ax[0], ax[1], b0[j & 3]);
                } else {
                    ntile_mma(w, j, act, z, lane);
                }
                const f32x2 nb = *reinterpret_cast<const f32x2*>(&s.net.nb[layer][8 * j + 2 * t]);
#pragma unroll
                for(int h = 0; h < 2; ++h) {
                    f32x2 nz, q;
                    const f32x2 a = silu2(z[2 * h], z[2 * h + 1], nb, nz, q);
                    unpack2(dsilu2(nz, q), ds[layer][j][2 * h], ds[layer][j][2 * h + 1]);
                    if(layer == 2) unpack2(a, a3[j][2 * h], a3[j][2 * h + 1]);
                    else next[j >> 1][2 * (j & 1) + h] = pack_bf16(a);
                }
            }
            if(layer == 2) break;
            store_frag(s.act[layer], r0, next, g, t);
#pragma unroll
            for(int e = 0; e < 16; ++e) act[e / 4][e % 4] = next[e / 4][e % 4];
        }
        float ylo = 0.f, yhi = 0.f;
#pragma unroll
        for(int j = 0; j < 8; ++j) {
            const float wl = s.net.w3[8 * j + 2 * t], wh = s.net.w3[8 * j + 2 * t + 1];
            ylo += a3[j][0] * wl + a3[j][1] * wh;
            yhi += a3[j][2] * wl + a3[j][3] * wh;
        }
        ylo += __shfl_xor_sync(FULL_MASK, ylo, 1);
        ylo += __shfl_xor_sync(FULL_MASK, ylo, 2);
        yhi += __shfl_xor_sync(FULL_MASK, yhi, 1);
        yhi += __shfl_xor_sync(FULL_MASK, yhi, 2);
        const float elo = v_lo ? ylo + s.net.b3 - t_lo : 0.f;
        const float ehi = v_hi ? yhi + s.net.b3 - t_hi : 0.f;
        const float dlo = 2.f * elo * inv_b, dhi = 2.f * ehi * inv_b;
        if(t == 0) {
            gloss += (elo * elo + ehi * ehi) * inv_b;
            gb3 += dlo + dhi;
        }
        // output layer: dw3, dZ of layer 2
        float v[8][2];
#pragma unroll
        for(int j = 0; j < 8; ++j) {
            v[j][0] = dlo * a3[j][0] + dhi * a3[j][2];
            v[j][1] = dlo * a3[j][1] + dhi * a3[j][3];
        }
        column_sums(v, gb[3], lane);
#pragma unroll
        for(int j = 0; j < 8; ++j) {
            const float wl = s.net.w3[8 * j + 2 * t], wh = s.net.w3[8 * j + 2 * t + 1];
            c[j][0] = dlo * wl;
            c[j][1] = dlo * wh;
            c[j][2] = dhi * wl;
            c[j][3] = dhi * wh;
        }
#pragma unroll
        for(int layer = 2; layer >= 0; --layer) {
            // c: dLoss / d(activation) of this layer -> dZ
            unsigned dzA[4][4];
#pragma unroll
            for(int j = 0; j < 8; ++j) {
#pragma unroll
                for(int e = 0; e < 4; ++e) c[j][e] *= ds[layer][j][e];
                v[j][0] = c[j][0] + c[j][2];
                v[j][1] = c[j][1] + c[j][3];
                dzA[j >> 1][2 * (j & 1)] = pack_bf16(c[j][0], c[j][1]);
                dzA[j >> 1][2 * (j & 1) + 1] = pack_bf16(c[j][2], c[j][3]);
            }
            column_sums(v, gb[layer], lane);
            store_frag(s.dz[layer], r0, dzA, g, t);
            if(layer == 0) break;
            // dA of the layer below = dZ W: W's rows are the k index
            const __nv_bfloat16* row = (layer == 2 ? s.net.w2 : s.net.w1) + lane * LDW;
#pragma unroll
            for(int j = 0; j < 8; ++j) {
                unsigned b[2][4];
                ldsm4<true>(b[0], row + 8 * j);
                ldsm4<true>(b[1], row + 32 * LDW + 8 * j);
                c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
#pragma unroll
                for(int kk = 0; kk < 4; ++kk) {
                    mma16816(c[j], dzA[kk][0], dzA[kk][1], dzA[kk][2], dzA[kk][3],
                             b[kk >> 1][2 * (kk & 1)], b[kk >> 1][2 * (kk & 1) + 1]);
                }
            }
        }
        __syncthreads();
        weight_sums(s.dz[1], s.act[0], o0, i0, dw1, lane);
        weight_sums(s.dz[2], s.act[1], o0, i0, dw2, lane);
        {   // the 5 inputs fit one n-tile: the two warps of an output strip take half the rows each
            const int q = lane >> 3, r = lane & 7, k0 = (warp >> 2) * (TROWS / 2);
            const __nv_bfloat16* pz = s.dz[0] + (k0 + r + (q >> 1) * 8) * LDW + o0 + (q & 1) * 8;
#pragma unroll
            for(int k = 0; k < TROWS / 2; k += 32) {
                unsigned a[2][4], b[4];
                ldsm4<true>(a[0], pz + k * LDW);
                ldsm4<true>(a[1], pz + (k + 16) * LDW);
                ldsm4<true>(b, s.x + (k0 + k + lane) * 8);
#pragma unroll
                for(int e = 0; e < 2; ++e) {
                    float d[4] = {0.f, 0.f, 0.f, 0.f};
                    mma16816(d, a[e][0], a[e][1], a[e][2], a[e][3], b[2 * e], b[2 * e + 1]);
#pragma unroll
                    for(int i = 0; i < 4; ++i) dw0[i] += d[i];
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for(int j = 0; j < 4; ++j) {
        const int o = o0 + g, i = i0 + 8 * j + 2 * t;
        atomicAdd(reinterpret_cast<float2*>(&grad[OFF_W1 + o * MLP_H + i]), make_float2(dw1[j][0], dw1[j][1]));
        atomicAdd(reinterpret_cast<float2*>(&grad[OFF_W1 + (o + 8) * MLP_H + i]), make_float2(dw1[j][2], dw1[j][3]));
        atomicAdd(reinterpret_cast<float2*>(&grad[OFF_W2 + o * MLP_H + i]), make_float2(dw2[j][0], dw2[j][1]));
        atomicAdd(reinterpret_cast<float2*>(&grad[OFF_W2 + (o + 8) * MLP_H + i]), make_float2(dw2[j][2], dw2[j][3]));
    }
#pragma unroll
    for(int e = 0; e < 2; ++e) {
        if(2 * t + e < MLP_IN) {
            atomicAdd(&grad[OFF_W0 + (o0 + g) * MLP_IN + 2 * t + e], dw0[e]);
            atomicAdd(&grad[OFF_W0 + (o0 + g + 8) * MLP_IN + 2 * t + e], dw0[2 + e]);
        }
    }
#pragma unroll
    for(int l = 0; l < 4; ++l) {
        s.part[warp][l * MLP_H + 8 * g + 2 * t] = gb[l][0];
        s.part[warp][l * MLP_H + 8 * g + 2 * t + 1] = gb[l][1];
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1) {
        gb3 += __shfl_xor_sync(FULL_MASK, gb3, o);
        gloss += __shfl_xor_sync(FULL_MASK, gloss, o);
    }
    if(lane == 0) {
        s.part0[warp][0] = gb3;
        s.part0[warp][1] = gloss;
    }
    __syncthreads();
    for(int k = threadIdx.x; k < 4 * MLP_H + 2; k += TBLK) {
        float v = 0.f;
        for(int w = 0; w < TBLK / 32; ++w) v += k < 4 * MLP_H ? s.part[w][k] : s.part0[w][k - 4 * MLP_H];
        const int l = k / MLP_H, e = k % MLP_H;
        if(k == 4 * MLP_H + 1) atomicAdd(loss, v);
        else atomicAdd(&grad[k == 4 * MLP_H ? OFF_B3
                                            : (l == 0 ? OFF_B0 : l == 1 ? OFF_B1 : l == 2 ? OFF_B2 : OFF_W3) + e], v);
    }
}

// Where parameter k lies in the network image: its BF16 (is16) or FP32 index.
__device__ __forceinline__ int image_index(int k, bool& is16)
{
    is16 = true;
    if(k < OFF_B0) return IMG_W0 + (k / MLP_IN) * MLP_INP + k % MLP_IN;
    if(k >= OFF_W1 && k < OFF_B1) return IMG_W1 + k - OFF_W1;
    if(k >= OFF_W2 && k < OFF_B2) return IMG_W2 + k - OFF_W2;
    is16 = false;
    if(k < OFF_W1) return IMGF_B0 + k - OFF_B0;
    if(k < OFF_W2) return IMGF_B1 + k - OFF_B1;
    if(k < OFF_W3) return IMGF_B2 + k - OFF_B2;
    return k < OFF_B3 ? IMGF_W3 + k - OFF_W3 : IMGF_B3;
}

__device__ __forceinline__ void image_put(int k, float v, __nv_bfloat16* w, float* f)
{
    bool is16;
    const int q = image_index(k, is16);
    if(is16) w[q] = __float2bfloat16(v);
    else f[q] = v;
}

// Adam update of the FP32 master parameters and their image; leaves grad and
// loss zero for the next batch (one launch between two batches instead of two
// memsets and two kernels).
__global__ void k_adam(float* __restrict__ p, float* __restrict__ grad, float* __restrict__ loss,
                       float* __restrict__ m1, float* __restrict__ m2, __nv_bfloat16* __restrict__ w,
                       float* __restrict__ f, int n, float lr, float b1, float b2, float c1, float c2, float eps)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if(k == 0) *loss = 0.f;
    if(k >= n) return;
    const float gk = grad[k];
    grad[k] = 0.f;
    const float a = b1 * m1[k] + (1.f - b1) * gk;
    const float b = b2 * m2[k] + (1.f - b2) * gk * gk;
    m1[k] = a;
    m2[k] = b;
    const float v = p[k] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[k] = v;
    image_put(k, v, w, f);
}

// The image of uploaded parameters (its padding is zeroed by the caller).
__global__ void k_make_image(const float* __restrict__ p, __nv_bfloat16* __restrict__ w, float* __restrict__ f)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if(k < MLP_NPARAM) image_put(k, p[k], w, f);
}

// Features + targets of raw Riemann states (n x 7: uL rhoL pL uR rhoR pR gamma).
__global__ void k_state_features(const double* __restrict__ st, const double* __restrict__ pstar, long long n,
                                 uint4* __restrict__ feat, float* __restrict__ target)
{
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if(r >= n) return;
    const double* s = st + 7 * r;
    const double gamma = s[6];
    const double L[4] = {s[0], s[1], s[2], sqrt(gamma * s[2] / s[1])};
    const double R[4] = {s[3], s[4], s[5], sqrt(gamma * s[5] / s[4])};
    float x[MLP_IN];
    mlp_features(L, R, gamma, x);
    uint4 v;
    v.x = pack_bf16(x[0], x[1]);
    v.y = pack_bf16(x[2], x[3]);
    v.z = pack_bf16(x[4], 0.f);
    v.w = 0u;
    feat[r] = v;
    if(target) target[r] = (float)log(pstar[r] / s[2]);
}

}  // namespace

MlpDev mlp_device(sphgpu_ctx* c)
{
    MlpDev m{};
    if(!c->d_mlp) return m;
    m.w = static_cast<const __nv_bfloat16*>(c->d_mlp);
    m.f = reinterpret_cast<const float*>(static_cast<const char*>(c->d_mlp) + IMG_F32_OFFSET);
    return m;
}

static void launch_infer(sphgpu_ctx* c, const uint4* feat, float* y, long long rows)
{
    constexpr long long per_block = (IBLK / 32) * 16;
    const long long blocks = std::min<long long>((rows + per_block - 1) / per_block, 148LL * IRES);
    k_mlp_infer<<<(unsigned)std::max<long long>(blocks, 1), IBLK, 0, c->stream>>>(mlp_device(c), feat, y, rows);
}

int mlp_infer_rows(sphgpu_ctx* c, const uint4* feat, float* y, long long rows)
{
    launch_infer(c, feat, y, rows);
    SPHGPU_LAUNCH_CHECK(c, "MLP inference");
    return SPHGPU_OK;
}

// y for device-resident states (n x 7); d_y has n floats.
int mlp_predict_states(sphgpu_ctx* c, const double* d_states, long long n, float* d_y)
{
    uint4* feat = nullptr;
    DevTemps tmp(c->stream);
    SPHGPU_CUDA(c, tmp.get(&feat, sizeof(uint4) * (size_t)n, false));
    k_state_features<<<grid_for(n, 256), 256, 0, c->stream>>>(d_states, nullptr, n, feat, nullptr);
    launch_infer(c, feat, d_y, n);
    SPHGPU_LAUNCH_CHECK(c, "MLP predict");
    SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));
    return SPHGPU_OK;
}

static int ensure_image(sphgpu_ctx* c)
{
    if(!c->d_mlp) SPHGPU_CUDA(c, cudaMalloc(&c->d_mlp, IMG_BYTES));
    return SPHGPU_OK;
}

static int upload_master(sphgpu_ctx* c)
{
    int rc = ensure_image(c);
    if(rc) return rc;
    if(!c->d_mlp_master) SPHGPU_CUDA(c, cudaMalloc(&c->d_mlp_master, sizeof(float) * 4 * MLP_NPARAM));
    SPHGPU_CUDA(c, cudaMemcpy(c->d_mlp_master, c->mlp_master.data(), sizeof(float) * MLP_NPARAM,
                              cudaMemcpyHostToDevice));
    SPHGPU_CUDA(c, cudaMemsetAsync(c->d_mlp, 0, IMG_BYTES, c->stream));
    k_make_image<<<grid_for(MLP_NPARAM, 256), 256, 0, c->stream>>>(
        c->d_mlp_master, static_cast<__nv_bfloat16*>(c->d_mlp),
        reinterpret_cast<float*>(static_cast<char*>(c->d_mlp) + IMG_F32_OFFSET));
    SPHGPU_LAUNCH_CHECK(c, "MLP image");
    SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));
    c->have_mlp = true;
    return SPHGPU_OK;
}

// The device buffer of one call on host states: the context's, kept between
// calls up to 64 MB (84 bytes a row, so some 760 K rows), one of the call's own
// beyond.  What is left is the copy from the caller's pageable memory: 500 K
// states 4.0 -> 1.85 ms for a prediction, 6.5 -> 2.7 for a loss and gradient
// (three to five cudaMalloc / cudaFree pairs a call before).  Four host threads
// filling a pinned ring gained nothing more (1.75 ms) and cost 6 ms to set up.
class MlpWork {
public:
    MlpWork() = default;
    ~MlpWork()
    {
        if(own_) cudaFree(base_);
    }
    MlpWork(const MlpWork&) = delete;
    MlpWork& operator=(const MlpWork&) = delete;
    cudaError_t take(sphgpu_ctx* c, size_t bytes)
    {
        if(bytes > KEEP) {
            own_ = true;
            return cudaMalloc(&base_, bytes);
        }
        if(c->mlp_work_bytes < bytes) {
            if(c->d_mlp_work) cudaFree(c->d_mlp_work);
            c->d_mlp_work = nullptr;
            c->mlp_work_bytes = 0;
            const cudaError_t e = cudaMalloc(&c->d_mlp_work, bytes);
            if(e != cudaSuccess) return e;
            c->mlp_work_bytes = bytes;
        }
        base_ = c->d_mlp_work;
        return cudaSuccess;
    }
    template <typename T>
    T* part(size_t count)
    {
        T* p = reinterpret_cast<T*>(static_cast<char*>(base_) + used_);
        used_ += padded(sizeof(T) * count);
        return p;
    }
    static size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }

private:
    static constexpr size_t KEEP = size_t(64) << 20;
    void* base_ = nullptr;
    bool own_ = false;
    size_t used_ = 0;
};

// device features/targets for host states, in parts of `work` (which has room
// for `extra` more bytes)
static int stage_states(sphgpu_ctx* c, MlpWork& work, const double* states, const double* pstar, int64_t n,
                        size_t extra, uint4** feat, float** target)
{
    const size_t rows = (size_t)n;
    SPHGPU_CUDA(c, work.take(c, MlpWork::padded(sizeof(double) * 7 * rows) + MlpWork::padded(sizeof(uint4) * rows) +
                                    (pstar ? MlpWork::padded(sizeof(double) * rows) + MlpWork::padded(sizeof(float) * rows)
                                           : 0) + extra));
    double* d_st = work.part<double>(7 * rows);
    double* d_ps = pstar ? work.part<double>(rows) : nullptr;
    *feat = work.part<uint4>(rows);
    *target = pstar ? work.part<float>(rows) : nullptr;
    SPHGPU_CUDA(c, cudaMemcpyAsync(d_st, states, sizeof(double) * 7 * rows, cudaMemcpyHostToDevice, c->stream));
    if(pstar) {
        SPHGPU_CUDA(c, cudaMemcpyAsync(d_ps, pstar, sizeof(double) * rows, cudaMemcpyHostToDevice, c->stream));
    }
    k_state_features<<<grid_for(n, 256), 256, 0, c->stream>>>(d_st, d_ps, n, *feat, *target);
    SPHGPU_LAUNCH_CHECK(c, "MLP features");
    return SPHGPU_OK;
}

}  // namespace sphgpu

using namespace sphgpu;

extern "C" {

int64_t sphgpu_mlp_param_count(void) { return MLP_NPARAM; }

int sphgpu_mlp_set_params(sphgpu_ctx* c, const float* params)
{
    if(!c || !params) return SPHGPU_ERR_ARG;
    if(!c->stream) return fail(c, SPHGPU_ERR_CUDA, "context has no device");
    c->mlp_master.assign(params, params + MLP_NPARAM);
    return upload_master(c);
}

int sphgpu_mlp_get_params(sphgpu_ctx* c, float* params)
{
    if(!c || !params) return SPHGPU_ERR_ARG;
    if(!c->have_mlp) return fail(c, SPHGPU_ERR_NO_MLP, "no MLP parameters loaded");
    std::memcpy(params, c->mlp_master.data(), sizeof(float) * MLP_NPARAM);
    return SPHGPU_OK;
}

// Deterministic initialisation (uniform +-sqrt(6 / (fan_in + fan_out)), zero
// biases) from a 64-bit seed.
int sphgpu_mlp_init(sphgpu_ctx* c, uint64_t seed)
{
    if(!c) return SPHGPU_ERR_ARG;
    std::vector<float> p(MLP_NPARAM, 0.f);
    uint64_t x = seed * 0x9E3779B97F4A7C15ull + 1;
    auto uni = [&]() {
        x ^= x >> 12;
        x ^= x << 25;
        x ^= x >> 27;
        return (double)((x * 0x2545F4914F6CDD1Dull) >> 11) / 9007199254740992.0;
    };
    auto fill = [&](int off, int fan_in, int fan_out, int count) {
        const double a = std::sqrt(6.0 / (fan_in + fan_out));
        for(int k = 0; k < count; ++k) p[off + k] = (float)((2.0 * uni() - 1.0) * a);
    };
    fill(OFF_W0, MLP_IN, MLP_H, MLP_H * MLP_IN);
    fill(OFF_W1, MLP_H, MLP_H, MLP_H * MLP_H);
    fill(OFF_W2, MLP_H, MLP_H, MLP_H * MLP_H);
    fill(OFF_W3, MLP_H, 1, MLP_H);
    return sphgpu_mlp_set_params(c, p.data());
}

// y = network output log(p_star / p_L) for raw states (n x 7).
int sphgpu_mlp_predict(sphgpu_ctx* c, const double* states, int64_t n, float* y)
{
    if(!c || !states || !y || n <= 0) return SPHGPU_ERR_ARG;
    if(!c->have_mlp) return fail(c, SPHGPU_ERR_NO_MLP, "no MLP parameters loaded");
    uint4* feat = nullptr;
    float* tgt = nullptr;
    MlpWork work;
    const int rc = stage_states(c, work, states, nullptr, n, MlpWork::padded(sizeof(float) * (size_t)n), &feat, &tgt);
    if(rc) return rc;
    float* d_y = work.part<float>((size_t)n);
    launch_infer(c, feat, d_y, n);
    SPHGPU_LAUNCH_CHECK(c, "MLP predict");
    SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));  // the context stream does not sync with cudaMemcpy
    SPHGPU_CUDA(c, cudaMemcpy(y, d_y, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost));
    return SPHGPU_OK;
}

// Train on labelled states with Adam (mean squared error in log(p*/p_L)).
// loss_history[e] = mean batch loss of epoch e.  With epochs == 0 only the
// full-data gradient of the current parameters is written to grad_out (for
// gradient checks) and its loss to loss_history[0].
int sphgpu_mlp_train(sphgpu_ctx* c, const double* states, const double* pstar, int64_t n, int epochs, int batch,
                     float lr, uint64_t seed, float* loss_history, float* grad_out)
{
    if(!c || !states || !pstar || n <= 0 || batch <= 0 || epochs < 0) return SPHGPU_ERR_ARG;
    if(!c->have_mlp) {
        const int rc = sphgpu_mlp_init(c, seed);
        if(rc) return rc;
    }
    uint4* feat = nullptr;
    float* tgt = nullptr;
    MlpWork work;
    const int rc = stage_states(c, work, states, pstar, n,
                                MlpWork::padded(sizeof(float) * MLP_NPARAM) + MlpWork::padded(sizeof(float)), &feat, &tgt);
    if(rc) return rc;
    float *m1 = c->d_mlp_master + MLP_NPARAM, *m2 = c->d_mlp_master + 2 * MLP_NPARAM;
    float* grad = work.part<float>(MLP_NPARAM);
    float* d_loss = work.part<float>(1);
    SPHGPU_CUDA(c, cudaMemsetAsync(m1, 0, sizeof(float) * 2 * MLP_NPARAM, c->stream));
    MlpDev md = mlp_device(c);
    auto run_batch = [&](long long base, int bsize, unsigned long long pa, unsigned long long pc) {
        const long long blocks = std::min<long long>(148, ((long long)bsize + TROWS - 1) / TROWS);
        k_mlp_train<<<(unsigned)blocks, TBLK, sizeof(SmemTrain), c->stream>>>(md, feat, tgt, n, base, bsize, pa, pc,
                                                                              grad, d_loss);
    };
    SPHGPU_CUDA(c, cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(SmemTrain)));
    SPHGPU_CUDA(c, cudaMemsetAsync(grad, 0, sizeof(float) * MLP_NPARAM, c->stream));
    SPHGPU_CUDA(c, cudaMemsetAsync(d_loss, 0, sizeof(float), c->stream));
    if(epochs == 0) {
        run_batch(0, (int)n, 1ull, 0ull);
        SPHGPU_LAUNCH_CHECK(c, "MLP gradient");
        SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));
        if(grad_out) SPHGPU_CUDA(c, cudaMemcpy(grad_out, grad, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost));
        if(loss_history) SPHGPU_CUDA(c, cudaMemcpy(loss_history, d_loss, sizeof(float), cudaMemcpyDeviceToHost));
    }
    uint64_t x = seed | 1;
    int64_t step = 0;
    for(int e = 0; e < epochs; ++e) {
        // a fresh multiplicative permutation of the rows per epoch
        x = x * 6364136223846793005ull + 1442695040888963407ull;
        unsigned long long pa = (x >> 17) % (unsigned long long)n;
        auto gcd = [](unsigned long long a, unsigned long long b) {
            while(b) {
                const unsigned long long r = a % b;
                a = b;
                b = r;
            }
            return a;
        };
        if(pa == 0) pa = 1;
        while(gcd(pa, (unsigned long long)n) != 1) pa = (pa + 1) % (unsigned long long)n;
        const unsigned long long pc = (x >> 33) % (unsigned long long)n;
        double esum = 0.0;
        int nb = 0;
        for(long long base = 0; base < n; base += batch, ++nb) {
            const int bsize = (int)std::min<long long>(batch, n - base);
            run_batch(base, bsize, pa, pc);
            if(nb % 64 == 0 || base + batch >= n) {
                float l = 0.f;
                SPHGPU_CUDA(c, cudaMemcpyAsync(&l, d_loss, sizeof(float), cudaMemcpyDeviceToHost, c->stream));
                SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));
                esum += l;
            }
            ++step;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);
            k_adam<<<grid_for(MLP_NPARAM, 256), 256, 0, c->stream>>>(
                c->d_mlp_master, grad, d_loss, m1, m2, static_cast<__nv_bfloat16*>(c->d_mlp),
                reinterpret_cast<float*>(static_cast<char*>(c->d_mlp) + IMG_F32_OFFSET), MLP_NPARAM, lr, b1, b2, c1,
                c2, 1e-8f);
        }
        SPHGPU_LAUNCH_CHECK(c, "MLP training");
        if(loss_history) loss_history[e] = (float)(esum / ((nb + 63) / 64));
    }
    SPHGPU_CUDA(c, cudaStreamSynchronize(c->stream));
    c->mlp_master.resize(MLP_NPARAM);
    SPHGPU_CUDA(c, cudaMemcpy(c->mlp_master.data(), c->d_mlp_master, sizeof(float) * MLP_NPARAM,
                              cudaMemcpyDeviceToHost));
    return SPHGPU_OK;
}

}  // extern "C"
