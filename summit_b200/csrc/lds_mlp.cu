// Surrogate network of the learned control variate: in -> 128 -> 128 -> 128 -> out,
// GELU (erf form) after each hidden layer, trained by mean squared error.
//
// Weights are kept in FP32 (Adam's master copy) and enter every product
// rounded to BF16; hidden activations are rounded to BF16 where they feed the
// next product; all sums accumulate in FP32.  Four kernels make one training
// step over a mini-batch of gathered rows:
//   mlp_forward_kernel      all four layers in shared memory, the weights loaded
//                           once per CTA, whose groups of 8 warps walk 32-row
//                           tiles; the products run on the tensor cores
//                           (mma.sync m16n8k16, BF16 x BF16 -> FP32), one
//                           16 x 32 output tile per warp; stores the
//                           pre-activations z1..z3 and the loss gradient of the
//                           outputs;
//   mlp_backward_data_kernel  dZ_l = (dZ_{l+1} W_{l+1}) * gelu'(z_l), l = 3, 2, 1,
//                           on the tensor cores too: the FP32 gradients enter as
//                           a BF16 pair hi + lo (two products), so they keep
//                           16 significant bits against the BF16 weights; keeps
//                           the activations H_l for the weight gradients;
//   mlp_backward_weight_kernel dW_l = dZ_l^T H_{l-1}, db_l = sum dZ_l over rows
//                           (row-split, FP32 atomics into the gradient), on the
//                           tensor cores with dZ as three BF16 terms, which hold
//                           all 24 bits of an FP32 value;
//   mlp_adam_kernel         Adam with bias correction on the FP32 master weights.
// Shared-memory operand rows carry 8 BF16 of padding, so the fragment loads of
// the 8 rows a quad group touches fall in distinct banks.
#include <algorithm>
#include <cuda_bf16.h>

#include <cstdint>

#include "lds_device.cuh"
#include "lds_internal.h"

namespace lds {
namespace mlp {

constexpr int kR = 32;         // rows per tile
constexpr int kThreads = 256;  // threads of a tile's group
constexpr int kMaxGroups = 4;  // groups per CTA (forward)

__device__ __forceinline__ float gelu(float z) {
    return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) +
           z * 0.39894228040143268f * expf(-0.5f * z * z);
}

constexpr int kPad = 8;              // BF16 of padding per shared-memory operand row
constexpr int kLdH = kMlpHidden + kPad;  // row stride of 128-wide operands

__host__ __device__ inline int round16(int x) { return (x + 15) & ~15; }
__host__ __device__ inline int ld_in(int in) { return round16(in) + kPad; }
__host__ __device__ inline int ld_out(int out) { return round16(out) + kPad; }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc[nt] (+)= the warp's 16 x 8 tiles (rows row0.., columns col0 + 8 nt..) of
// A B over K (a multiple of 16): A row-major BF16 [rows][lda], B stored per
// output column with K contiguous, BF16 [cols][ldb]; tiles at or beyond ncols
// are skipped.  With A2 (the low halves of a split FP32 operand) both halves
// are multiplied into the same accumulators.
__device__ __forceinline__ void warp_mma4(const __nv_bfloat16* A, const __nv_bfloat16* A2, int lda,
                                          int row0, const __nv_bfloat16* B, int ldb, int col0,
                                          int ncols, int K, float (&acc)[4][4]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
    // ldmatrix rows of this lane: A's 16 rows x two 8-column halves; B's two pairs
    // of 8-column tiles x two halves of K.
    const int ar = row0 + (lane & 15), ak = (lane >> 4) * 8;
    const int bc = col0 + (lane >> 4) * 8 + (lane & 7), bk = ((lane >> 3) & 1) * 8;
    for (int k = 0; k < K; k += 16) {
        uint32_t a[4], a2[4] = {0, 0, 0, 0};
        ldsm_x4(smem_u32(A + ar * lda + k + ak), a[0], a[1], a[2], a[3]);
        if (A2) ldsm_x4(smem_u32(A2 + ar * lda + k + ak), a2[0], a2[1], a2[2], a2[3]);
#pragma unroll
        for (int np = 0; np < 2; ++np) {
            if (col0 + 16 * np >= ncols) continue;   // (ncols is a multiple of 16)
            uint32_t b[4];
            ldsm_x4(smem_u32(B + (bc + 16 * np) * ldb + k + bk), b[0], b[1], b[2], b[3]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                mma_bf16(acc[2 * np + h], a, b[2 * h], b[2 * h + 1]);
                if (A2) mma_bf16(acc[2 * np + h], a2, b[2 * h], b[2 * h + 1]);
            }
        }
    }
}

// Element e (0..3) of the warp's fragment nt: row and column of C.
__device__ __forceinline__ int frag_row(int row0, int e) {
    return row0 + ((threadIdx.x & 31) >> 2) + 8 * (e >> 1);
}
__device__ __forceinline__ int frag_col(int col0, int nt, int e) {
    return col0 + 8 * nt + 2 * (threadIdx.x & 3) + (e & 1);
}

// A FP32 value as a BF16 pair hi + lo (hi + lo within 2^-16 relative of v).
__device__ __forceinline__ void split_bf16(float v, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// Barrier of the calling thread's group of 256 (every thread of a group runs the
// same tiles).
__device__ __forceinline__ void group_sync() {
    asm volatile("bar.sync %0, %1;" ::"r"((int)(threadIdx.x / kThreads) + 1), "r"(kThreads) : "memory");
}

// Copy `bytes` (a multiple of 16) from global to shared memory.
__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint4* d = reinterpret_cast<uint4*>(dst);
    for (int i = threadIdx.x; i < bytes / 16; i += blockDim.x) d[i] = s[i];
}

}  // namespace mlp

using namespace mlp;

// BF16 copies of the weights in the operand layouts of the products, made
// once per step (rows padded to the shared-memory strides, padding zero):
//   forward  F1 [128][ld_in] = W1, F2, F3 [128][kLdH] = W2, W3,
//            F4 [round16(out)][kLdH] = W4 (rows >= out zero);
//   backward B4 [128][ld_out] = W4^T, B3, B2 [128][kLdH] = W3^T, W2^T.
__global__ void mlp_pack_kernel(MlpArgs a, __nv_bfloat16* __restrict__ pack) {
    const MlpLayout L = mlp_layout(a.in, a.out);
    const int H = kMlpHidden, li = ld_in(a.in), lo = ld_out(a.out), o16 = round16(a.out);
    const int64_t nF1 = (int64_t)H * li, nH = (int64_t)H * kLdH, nF4 = (int64_t)o16 * kLdH;
    const int64_t nB4 = (int64_t)H * lo;
    const int64_t total = nF1 + 2 * nH + nF4 + nB4 + 2 * nH;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = i;
        float v = 0.0f;
        if (r < nF1) {
            const int c = (int)(r / li), k = (int)(r % li);
            if (k < a.in) v = a.params[L.W1 + (int64_t)c * a.in + k];
        } else if ((r -= nF1) < 2 * nH) {
            const int64_t base = r < nH ? L.W2 : L.W3;
            const int64_t q = r % nH;
            const int c = (int)(q / kLdH), k = (int)(q % kLdH);
            if (k < H) v = a.params[base + (int64_t)c * H + k];
        } else if ((r -= 2 * nH) < nF4) {
            const int c = (int)(r / kLdH), k = (int)(r % kLdH);
            if (c < a.out && k < H) v = a.params[L.W4 + (int64_t)c * H + k];
        } else if ((r -= nF4) < nB4) {
            const int n = (int)(r / lo), k = (int)(r % lo);  // B4[n][k] = W4[k][n]
            if (k < a.out) v = a.params[L.W4 + (int64_t)k * H + n];
        } else {
            r -= nB4;
            const int64_t base = r < nH ? L.W3 : L.W2;
            const int64_t q = r % nH;
            const int n = (int)(q / kLdH), k = (int)(q % kLdH);  // W^T[n][k] = W[k][n]
            if (k < H) v = a.params[base + (int64_t)k * H + n];
        }
        pack[i] = __float2bfloat16_rn(v);
    }
}

// What bounds it: erff of the 384 hidden units per row.  The weights (100 KB) are
// copied once per CTA and up to four groups of 8 warps walk the row tiles beside
// each other, so that one group's activations overlap another's products and
// loads.  100,003 rows, 68 -> 24: 270 -> 115 us (weights copied for every 32 rows,
// one group per SM).
__global__ void __launch_bounds__(kMaxGroups * kThreads)
    mlp_forward_kernel(MlpArgs a, const __nv_bfloat16* __restrict__ pack,
                       const float* __restrict__ x, const int32_t* __restrict__ rows, int64_t n,
                       const float* __restrict__ target, float* __restrict__ out,
                       float* __restrict__ zs, float* __restrict__ dout, double* __restrict__ loss,
                       float gscale) {
    extern __shared__ __align__(16) uint8_t smem[];
    const MlpLayout L = mlp_layout(a.in, a.out);
    const int op = mlp_out_pad(a.out), li = ld_in(a.in), o16 = round16(a.out);
    const int ngroups = (int)blockDim.x / kThreads, group = (int)threadIdx.x / kThreads;
    const int t = (int)threadIdx.x % kThreads;
    __nv_bfloat16* F1 = reinterpret_cast<__nv_bfloat16*>(smem);    // [128][li]
    __nv_bfloat16* F2 = F1 + kMlpHidden * li;                       // [128][kLdH]
    __nv_bfloat16* F3 = F2 + kMlpHidden * kLdH;                     // [128][kLdH]
    __nv_bfloat16* F4 = F3 + kMlpHidden * kLdH;                     // [o16][kLdH]
    __nv_bfloat16* X = F4 + o16 * kLdH + group * (kR * li + 2 * kR * kLdH);   // [kR][li]
    __nv_bfloat16* H1 = X + kR * li;                                // [kR][kLdH]
    __nv_bfloat16* H2 = H1 + kR * kLdH;                             // [kR][kLdH]
    copy16(F1, pack, (kMlpHidden * li + 2 * kMlpHidden * kLdH + o16 * kLdH) * 2);
    __syncthreads();

    const int w = t >> 5, lane = t & 31;
    const int row0 = 16 * (w & 1), col0 = 32 * (w >> 1);
    float acc[4][4];
    const float* bias[3] = {a.params + L.b1, a.params + L.b2, a.params + L.b3};
    double lsum = 0.0;
    const int64_t ntiles = (n + kR - 1) / kR;
    for (int64_t tile = (int64_t)blockIdx.x * ngroups + group; tile < ntiles;
         tile += (int64_t)gridDim.x * ngroups) {
        const int64_t r_base = tile * kR;
        group_sync();   // the previous tile's reads of X and H1
#pragma unroll
        for (int q = 0; q < kR / 8; ++q) {   // four rows per warp, lanes along the inputs
            const int r = w + 8 * q;
            const int64_t rr = r_base + r;
            const float* xr = x + (rr < n ? (int64_t)(rows ? rows[rr] : rr) : 0) * a.in;
            for (int k = lane; k < li; k += 32)
                X[r * li + k] = __float2bfloat16_rn(rr < n && k < a.in ? xr[k] : 0.0f);
        }
        group_sync();
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            const __nv_bfloat16* src = l == 0 ? X : l == 1 ? H1 : H2;
            const __nv_bfloat16* W = l == 0 ? F1 : l == 1 ? F2 : F3;
            __nv_bfloat16* dst = l == 1 ? H2 : H1;
            const int ld = l == 0 ? li : kLdH;
            warp_mma4(src, nullptr, ld, row0, W, ld, col0, kMlpHidden,
                      l == 0 ? round16(a.in) : kMlpHidden, acc);
            if (l == 2) group_sync();  // layer 3 writes H1, which layer 2 read
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const int r = frag_row(row0, e), c = frag_col(col0, nt, e);
                    const int64_t rr = r_base + r;
                    const float z0 = acc[nt][e] + bias[l][c], z1 = acc[nt][e + 1] + bias[l][c + 1];
                    if (zs && rr < n)
                        *reinterpret_cast<float2*>(zs + (rr * 3 + l) * kMlpHidden + c) =
                            make_float2(z0, z1);
                    *reinterpret_cast<__nv_bfloat162*>(dst + r * kLdH + c) =
                        __floats2bfloat162_rn(gelu(z0), gelu(z1));
                }
            group_sync();
        }
        warp_mma4(H1, nullptr, kLdH, row0, F4, kLdH, col0, o16, kMlpHidden, acc);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = frag_row(row0, e), c = frag_col(col0, nt, e);
                const int64_t rr = r_base + r;
                if (rr >= n || c >= op) continue;
                if (c >= a.out) {  // padding columns of dout read as zero in backward
                    if (dout) dout[rr * op + c] = 0.0f;
                    continue;
                }
                const float o = acc[nt][e] + a.params[L.b4 + c];
                if (out) out[rr * a.out + c] = o;
                if (target) {
                    const float d = o - target[(int64_t)(rows ? rows[rr] : rr) * a.out + c];
                    if (dout) dout[rr * op + c] = 2.0f * d * gscale;
                    lsum += (double)(d * d);
                }
            }
    }
    if (loss) {
        for (int o = 16; o; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if ((t & 31) == 0) atomicAdd(loss, lsum * (double)gscale);
    }
}

__global__ void __launch_bounds__(kThreads)
    mlp_backward_data_kernel(MlpArgs a, const __nv_bfloat16* __restrict__ pack_b, int64_t n,
                             const float* __restrict__ zs, const float* __restrict__ dout,
                             float* __restrict__ dzs, __nv_bfloat16* __restrict__ hs) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int op = mlp_out_pad(a.out), lo = ld_out(a.out);
    __nv_bfloat16* B4 = reinterpret_cast<__nv_bfloat16*>(smem);     // [128][lo] = W4^T
    __nv_bfloat16* B3 = B4 + kMlpHidden * lo;                       // [128][kLdH] = W3^T
    __nv_bfloat16* B2 = B3 + kMlpHidden * kLdH;                     // [128][kLdH] = W2^T
    __nv_bfloat16* A0 = B2 + kMlpHidden * kLdH;                     // [2][kR][kLdH] hi | lo
    __nv_bfloat16* A1 = A0 + 2 * kR * kLdH;                         // [2][kR][kLdH] hi | lo
    copy16(B4, pack_b, (kMlpHidden * lo + 2 * kMlpHidden * kLdH) * 2);
    const int64_t r_base = (int64_t)blockIdx.x * kR;
    for (int idx = threadIdx.x; idx < kR * lo; idx += blockDim.x) {
        const int r = idx / lo, k = idx - r * lo;
        const int64_t rr = r_base + r;
        const float g = (rr < n && k < op) ? dout[rr * op + k] : 0.0f;
        split_bf16(g, A0[r * lo + k], A0[kR * kLdH + r * lo + k]);
    }
    __syncthreads();
    const int t = threadIdx.x, w = t >> 5;
    const int row0 = 16 * (w & 1), col0 = 32 * (w >> 1);
    const __nv_bfloat16* Bs[3] = {B4, B3, B2};
    float acc[4][4];
    for (int s = 0; s < 3; ++s) {
        const int l = 2 - s;  // hidden layer index of z being differentiated
        __nv_bfloat16* src = (s & 1) ? A1 : A0;
        __nv_bfloat16* dst = (s & 1) ? A0 : A1;
        const int ld = s == 0 ? lo : kLdH;
        warp_mma4(src, src + kR * kLdH, ld, row0, Bs[s], ld, col0, kMlpHidden,
                  s == 0 ? round16(a.out) : kMlpHidden, acc);
        __syncthreads();
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = frag_row(row0, e), c = frag_col(col0, nt, e);
                const int64_t rr = r_base + r;
                float g = 0.0f;
                if (rr < n) {
                    const float z = zs[(rr * 3 + l) * kMlpHidden + c];
                    g = acc[nt][e] * gelu_grad(z);
                    dzs[(rr * 3 + l) * kMlpHidden + c] = g;
                    hs[(rr * 3 + l) * kMlpHidden + c] = __float2bfloat16_rn(gelu(z));
                }
                if (s < 2) split_bf16(g, dst[r * kLdH + c], dst[kR * kLdH + r * kLdH + c]);
            }
        __syncthreads();
    }
}

// Layer l = blockIdx.y (0..3), rows of split blockIdx.x: dW_l += dZ_l^T H_{l-1}
// (H_{-1} the BF16 inputs) and db_l += column sums of dZ_l.  A chunk of kWRows
// rows of dZ lies in shared memory as three BF16 terms (hi + mid + lo, 24 bits)
// beside H's; both operands are read transposed by ldmatrix (their rows are the
// product's K), warp w forming outputs 16 w..16 w + 15 against every input.
//
// Latency-bound at a mini-batch's size, so the splits are one chunk each: 4,096
// rows, 68 -> 24: 190 -> 24 us (FP32 FMAs from shared memory, GELU recomputed
// for every 16 outputs, 8 splits).
constexpr int kWRows = 64;

__host__ __device__ constexpr size_t mlp_weight_smem() {
    return (size_t)4 * kWRows * kLdH * sizeof(__nv_bfloat16);
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__global__ void __launch_bounds__(kThreads)
    mlp_backward_weight_kernel(MlpArgs a, const float* __restrict__ x,
                               const int32_t* __restrict__ rows, int64_t n,
                               const __nv_bfloat16* __restrict__ hs, const float* __restrict__ dzs,
                               const float* __restrict__ dout, float* __restrict__ grad,
                               int rows_per_split) {
    extern __shared__ __align__(16) uint8_t smem[];
    __nv_bfloat16* D = reinterpret_cast<__nv_bfloat16*>(smem);   // [3][kWRows][kLdH]
    __nv_bfloat16* H = D + 3 * kWRows * kLdH;                     // [kWRows][kLdH]
    const MlpLayout L = mlp_layout(a.in, a.out);
    const int op = mlp_out_pad(a.out), l = blockIdx.y;
    const int nout = l < 3 ? kMlpHidden : a.out, kin = l == 0 ? a.in : kMlpHidden;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int col = t & 127;                 // the unit this thread loads
    const int m0 = 16 * w, ntiles = round16(kin) / 8;
    float acc[16][4];
#pragma unroll
    for (int nt = 0; nt < 16; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.0f;
    float bsum = 0.0f;
    const int64_t r_begin = (int64_t)blockIdx.x * rows_per_split;
    const int64_t r_end = min(n, r_begin + rows_per_split);
    for (int64_t rb = r_begin; rb < r_end; rb += kWRows) {
        __syncthreads();
        for (int r = t >> 7; r < kWRows; r += kThreads / 128) {
            const int64_t rr = rb + r;
            float d = 0.0f;
            __nv_bfloat16 h = __float2bfloat16_rn(0.0f);
            if (rr < r_end) {
                if (col < nout)
                    d = l < 3 ? dzs[(rr * 3 + l) * kMlpHidden + col] : dout[rr * op + col];
                if (col < kin)
                    h = l == 0 ? __float2bfloat16_rn(x[(int64_t)(rows ? rows[rr] : rr) * a.in + col])
                               : hs[(rr * 3 + (l - 1)) * kMlpHidden + col];
            }
            bsum += d;
            // (the first term truncated, so that it is finite where d is; of an
            // infinite d there is no rest)
            const __nv_bfloat16 hi = __float2bfloat16_rz(d);
            const float r1 = isinf(d) ? 0.0f : d - __bfloat162float(hi);
            const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
            const float rest = r1 - __bfloat162float(mid);
            D[r * kLdH + col] = hi;
            D[(kWRows + r) * kLdH + col] = mid;
            D[(2 * kWRows + r) * kLdH + col] = __float2bfloat16_rn(rest);
            H[r * kLdH + col] = h;
        }
        __syncthreads();
        if (m0 < nout) {
            // ldmatrix rows of this lane: A = dZ^T (blocks: K halves x output
            // halves), B = H (blocks: two 8-input tiles x K halves)
            const int ar = (lane & 7) + (lane >> 4) * 8, ac = m0 + ((lane >> 3) & 1) * 8;
            const int br = (lane & 7) + ((lane >> 3) & 1) * 8, bc = (lane >> 4) * 8;
#pragma unroll
            for (int k = 0; k < kWRows; k += 16) {
                uint32_t a3[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    ldsm_x4_t(smem_u32(D + (p * kWRows + k + ar) * kLdH + ac), a3[p]);
#pragma unroll
                for (int np = 0; np < 8; ++np) {
                    if (2 * np >= ntiles) break;   // (ntiles is even)
                    uint32_t b[4];
                    ldsm_x4_t(smem_u32(H + (k + br) * kLdH + 16 * np + bc), b);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int p = 2; p >= 0; --p)
                            mma_bf16(acc[2 * np + h], a3[p], b[2 * h], b[2 * h + 1]);
                }
            }
        }
    }
    const int64_t wofs = l == 0 ? L.W1 : l == 1 ? L.W2 : l == 2 ? L.W3 : L.W4;
    const int64_t bofs = l == 0 ? L.b1 : l == 1 ? L.b2 : l == 2 ? L.b3 : L.b4;
    if (m0 < nout)
#pragma unroll
        for (int nt = 0; nt < 16; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = frag_row(m0, e), k = frag_col(0, nt, e);
                if (c < nout && k < kin) atomicAdd(&grad[wofs + (int64_t)c * kin + k], acc[nt][e]);
            }
    if (col < nout) atomicAdd(&grad[bofs + col], bsum);
}

__global__ void mlp_adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                                const float* __restrict__ g, int64_t P, float lr, float b1, float b2,
                                float eps, float bc1, float bc2) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

size_t mlp_forward_smem(int in, int out, int groups) {
    return (size_t)(kMlpHidden * ld_in(in) + 2 * kMlpHidden * kLdH + round16(out) * kLdH +
                    groups * (kR * ld_in(in) + 2 * kR * kLdH)) * 2;
}
size_t mlp_backward_smem(int out) {
    return (size_t)(kMlpHidden * ld_out(out) + 2 * kMlpHidden * kLdH + 4 * kR * kLdH) * 2;
}

static size_t pack_forward_elems(int in, int out) {
    return (size_t)kMlpHidden * ld_in(in) + 2 * kMlpHidden * kLdH + (size_t)round16(out) * kLdH;
}

size_t mlp_pack_elems(int in, int out) {
    return pack_forward_elems(in, out) + (size_t)kMlpHidden * ld_out(out) +
           2 * kMlpHidden * kLdH;
}

void launch_mlp_pack(const MlpArgs& a, void* pack, cudaStream_t st) {
    mlp_pack_kernel<<<148, 256, 0, st>>>(a, static_cast<__nv_bfloat16*>(pack));
    count_launch();
}

// The kernels' shared-memory limits, set once per device for the largest
// network the C ABI admits (LDS_MLP_MAX_IN inputs, LDS_MLP_MAX_OUT outputs).
static void set_smem_attrs(int, int) {
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [] {
        cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024);
        cudaFuncSetAttribute(mlp_backward_data_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)mlp_backward_smem(64));
        cudaFuncSetAttribute(mlp_backward_weight_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)mlp_weight_smem());
    });
}

void launch_mlp_forward(const MlpArgs& a, const void* pack, const float* x, const int32_t* rows,
                        int64_t n, const float* target, float* out, float* zs, float* dout,
                        double* loss, float gscale, cudaStream_t st) {
    if (n <= 0) return;
    set_smem_attrs(a.in, a.out);
    // One tile per CTA while they fit the SMs once, then up to four groups per CTA
    // (as shared memory allows) walking the rest.
    const int64_t tiles = (n + kR - 1) / kR;
    int groups = (int)std::min<int64_t>(kMaxGroups, (tiles + 147) / 148);
    while (groups > 1 && mlp_forward_smem(a.in, a.out, groups) > 227 * 1024) --groups;
    const unsigned grid = (unsigned)std::min<int64_t>(148, (tiles + groups - 1) / groups);
    mlp_forward_kernel<<<grid, groups * kThreads, mlp_forward_smem(a.in, a.out, groups), st>>>(
        a, static_cast<const __nv_bfloat16*>(pack), x, rows, n, target, out, zs, dout, loss, gscale);
    count_launch();
}

void launch_mlp_backward(const MlpArgs& a, const void* pack, const float* x, const int32_t* rows,
                         int64_t n, const float* zs, const float* dout, float* dzs, void* hs,
                         float* grad, cudaStream_t st) {
    if (n <= 0) return;
    set_smem_attrs(a.in, a.out);
    const __nv_bfloat16* pn =
        static_cast<const __nv_bfloat16*>(pack) + pack_forward_elems(a.in, a.out);
    mlp_backward_data_kernel<<<(unsigned)((n + kR - 1) / kR), kThreads, mlp_backward_smem(a.out),
                               st>>>(a, pn, n, zs, dout, dzs, static_cast<__nv_bfloat16*>(hs));
    count_launch();
    // Splits of one chunk up to eight CTAs for each SM over the four layers, longer
    // ones beyond (each split adds its sums to the gradient by atomics).
    const int64_t chunks = (n + kWRows - 1) / kWRows;
    const int per = (int)std::max<int64_t>(1, (chunks + 295) / 296);
    dim3 grid((unsigned)((chunks + per - 1) / per), 4);
    mlp_backward_weight_kernel<<<grid, kThreads, mlp_weight_smem(), st>>>(
        a, x, rows, n, static_cast<const __nv_bfloat16*>(hs), dzs, dout, grad, per * kWRows);
    count_launch();
}

void launch_mlp_adam(float* p, float* m, float* v, const float* g, int64_t P, float lr, float b1,
                     float b2, float eps, float bc1, float bc2, cudaStream_t st) {
    mlp_adam_kernel<<<(unsigned)((P + 255) / 256), 256, 0, st>>>(p, m, v, g, P, lr, b1, b2, eps,
                                                                 bc1, bc2);
    count_launch();
}

}  // namespace lds
