// SUMMIT-GxE directional LD-score products (MultiEnvironmentKernel,
// gxeldcore.cpp:10281-12557) on the B200: the elementwise and reduction
// kernels around the two tensor-core products, which reuse the phase-1 and
// phase-2 kernels.
//
// Source panel (source_block, gxeldcore.cpp:11008-11240).  Column
// c = ((e 2 + h) K + k) B + b of the panel holds
//   h = 0 (additive):     X [sqrt(a_k) o z_b o s_x,e]
//   h = 1 (interaction):  phi_e o (X [sqrt(a_k) o z_b o s_w,e])
// where X are the standardized genotypes of the block.  The product runs on
// p1_umma_kernel with one "super-bin" per (e, h, k); gxe_source_finalize
// applies phi_e and adds into the panel.
//
// Projection (project_sources, :11583-11729): P <- P - U (U^T P) with the
// common basis U, then per column the environment direction and the mean:
// P <- P - d_e (d_e^T P) - mean(P), both coefficients taken from the same
// values; the leakage onto the environment's fixed-effect basis must stay
// below 1e-9.  FP64 column reductions in a fixed order.
//
// Target (target_score_block, :11731-11936): out = X^T [P, w o P] on
// p2_umma_kernel with one "bin" per (pair half p, e, h, k) giving
// S = sum_b out^2 per SNP; gxe_target_finalize scales by s^2 / (N - rank_e)^2
// (s = s_x,e for p = 0, s_w,e for p = 1) into accum_{xx,xw,wx,ww}
// [(e total + block_start + j) K + k] (accumulator 2p + h).
//
// Probes (numpy_philox_rademacher_block, :10002-10113): NumPy's
// Philox4x64-10 stream per probe column (key from the caller), one 32-bit
// word per 4 rows, the high bit of each byte giving the sign; every row is
// independent given its counter, so the kernel is one thread per element.
#include <algorithm>
#include <cstdint>

#include "lds_internal.h"

namespace lds {

namespace {

__global__ void gxe_source_finalize_kernel(const double* __restrict__ Y, int64_t N, int64_t N_pad,
                                           int64_t C, int cols_half, const double* __restrict__ env,
                                           int64_t env_ld, int env_start, double* __restrict__ target,
                                           int64_t t_ld) {
    const int64_t n = N * C;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = t / N, i = t - c * N;
        const int64_t e = c / (2 * cols_half);
        const bool inter = ((c / cols_half) & 1) != 0;
        double v = Y[c * N_pad + i];
        if (inter) v *= env[(env_start + e) * env_ld + i];
        target[c * t_ld + i] += v;
    }
}

// out[c nb + a] = sum_i basis[a b_ld + i] panel[c p_ld + i], or with kSquares
// out[c] = sum_i panel[c p_ld + i]^2.  Columns [g group_cols, (g + 1) group_cols)
// read the basis at g group_stride, so one launch covers every environment's
// columns.  One CTA per column, fixed reduction order.
//
// Memory-bound: nb + 1 values read per nb multiply-adds, the basis from L2.
// The basis count is a template argument (32 predicated accumulators for any
// count kept each element's loads in one chain); GxE projection of 256 columns
// of 20,000 samples, 2 common columns, 4 environments: 13 launches 1,068 us ->
// 8 launches 135 us in all.
constexpr int kDotThreads = 256;
constexpr int kMaxBasis = 32;

template <int kNb, bool kSquares>
__global__ void __launch_bounds__(kDotThreads)
    col_dots_kernel(const double* __restrict__ panel, int64_t p_ld, int64_t N,
                    const double* __restrict__ basis, int64_t b_ld, int nb, int64_t group_cols,
                    int64_t group_stride, double* __restrict__ out) {
    __shared__ double red[kDotThreads / 32][kNb];
    const int64_t c = blockIdx.x;
    const double* v = panel + c * p_ld;
    const double* bs = kSquares ? nullptr : basis + c / group_cols * group_stride;
    double acc[kNb];
#pragma unroll
    for (int a = 0; a < kNb; ++a) acc[a] = 0.0;
    int64_t i = threadIdx.x;
    constexpr int kU = kNb <= 4 ? 4 : 1;
    for (; i + (kU - 1) * kDotThreads < N; i += kU * kDotThreads) {
        double x[kU], b[kU][kNb];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            x[u] = v[i + u * kDotThreads];
#pragma unroll
            for (int a = 0; a < kNb; ++a)
                b[u][a] = kSquares ? x[u] : a < nb ? bs[a * b_ld + i + u * kDotThreads] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
#pragma unroll
            for (int a = 0; a < kNb; ++a) acc[a] += b[u][a] * x[u];
    }
    for (; i < N; i += kDotThreads) {
        const double x = v[i];
#pragma unroll
        for (int a = 0; a < kNb; ++a)
            if (a < nb) acc[a] += (kSquares ? x : bs[a * b_ld + i]) * x;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < kNb; ++a) {
        double s = acc[a];
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[w][a] = s;
    }
    __syncthreads();
    if ((int)threadIdx.x < nb) {
        double s = 0.0;
        for (int q = 0; q < kDotThreads / 32; ++q) s += red[q][threadIdx.x];
        out[c * nb + threadIdx.x] = s;
    }
}

// panel[c ld + i] -= sum_a basis[a b_ld + i] coef[c nb + a] scale_a, where the
// last basis column is all ones, its coefficient scaled, when ones_last; the
// basis per column group as in col_dots_kernel.
__global__ void sub_lowrank_kernel(double* __restrict__ panel, int64_t ld, int64_t N, int64_t C,
                                   const double* __restrict__ basis, int64_t b_ld, int nb,
                                   const double* __restrict__ coef, int ones_last,
                                   double last_scale, int64_t group_cols, int64_t group_stride) {
    for (int64_t c = blockIdx.y; c < C; c += gridDim.y) {
        const double* bs = basis + c / group_cols * group_stride;
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N;
             i += (int64_t)gridDim.x * blockDim.x) {
            double s = 0.0;
            for (int a = 0; a < nb; ++a) {
                const bool ones = ones_last && a == nb - 1;
                const double b = ones ? 1.0 : bs[a * b_ld + i];
                s += b * (ones ? coef[c * nb + a] * last_scale : coef[c * nb + a]);
            }
            panel[c * ld + i] -= s;
        }
    }
}

// Ypair[c N_pad + i] = S[c s_ld + i], Ypair[(C + c) N_pad + i] = w[g(c)] o S, rows
// N..N_pad zero; g(c) = c / cols_per_group.
__global__ void gxe_pair_kernel(const double* __restrict__ S, int64_t s_ld, int64_t N,
                                int64_t N_pad, int64_t C, int64_t cols_per_group,
                                const double* __restrict__ w, int64_t w_ld, int w_first,
                                double* __restrict__ Ypair) {
    const int64_t n = N_pad * C;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = t / N_pad, i = t - c * N_pad;
        double v = 0.0, vw = 0.0;
        if (i < N) {
            v = S[c * s_ld + i];
            vw = w[(w_first + c / cols_per_group) * w_ld + i] * v;
        }
        Ypair[c * N_pad + i] = v;
        Ypair[(C + c) * N_pad + i] = vw;
    }
}

__global__ void gxe_target_finalize_kernel(const double* __restrict__ S, int64_t L, int Kp, int K,
                                           int T, const double* __restrict__ sx,
                                           const double* __restrict__ sw, int64_t s_ld,
                                           const int32_t* __restrict__ ranks, int64_t N,
                                           int env_start, int64_t total, int64_t block_start,
                                           double* a0, double* a1, double* a2, double* a3) {
    const int64_t n = L * Kp;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / Kp;
        const int g = (int)(t - j * Kp);
        // g = ((p T + e) 2 + h) K + k
        const int k = g % K;
        const int h = (g / K) & 1;
        const int pe = g / (2 * K);
        const int e = pe % T, p = pe / T;
        const double s = p == 0 ? sx[(int64_t)e * s_ld + j] : sw[(int64_t)e * s_ld + j];
        const double df = (double)(N - ranks[env_start + e]);
        const double val = S[j * Kp + g] * (s * s) * (1.0 / (df * df));
        double* acc = (p == 0) ? (h == 0 ? a0 : a1) : (h == 0 ? a2 : a3);
        acc[((int64_t)(env_start + e) * total + block_start + j) * K + k] += val;
    }
}

__global__ void scale_kernel(double* __restrict__ x, int64_t n, double s) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
        x[t] *= s;
}

// Input checks of source/target (gxeldcore.cpp:11131-11158, :11817-11829):
// flag |= 1 for a non-finite probe, 2 for a non-finite or <= 0 scale, 4 for a
// negative or non-finite annotation (when given raw).
__global__ void gxe_check_kernel(const double* __restrict__ probes, int64_t np,
                                 const double* __restrict__ sx, const double* __restrict__ sw,
                                 int64_t ns, const double* __restrict__ annot, int64_t na,
                                 unsigned* flag) {
    unsigned f = 0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < np;
         t += (int64_t)gridDim.x * blockDim.x)
        if (!isfinite(probes[t])) f |= 1u;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ns;
         t += (int64_t)gridDim.x * blockDim.x) {
        const double a = sx[t], b = sw[t];
        if (!isfinite(a) || !isfinite(b) || a <= 0.0 || b <= 0.0) f |= 2u;
    }
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < na;
         t += (int64_t)gridDim.x * blockDim.x)
        if (!isfinite(annot[t]) || annot[t] < 0.0) f |= 4u;
    if (f) atomicOr(flag, f);
}

// ---- NumPy Philox4x64-10 (the published Random123 algorithm, NumPy's
// counter/buffer conventions as gxeldcore.cpp:10011-10068 uses them) ----
__device__ __forceinline__ void philox4x64_10(uint64_t c[4], uint64_t k0, uint64_t k1) {
    const uint64_t M0 = 0xD2E7470EE14C6C93ULL, M1 = 0xCA5A826395121157ULL;
    const uint64_t W0 = 0x9E3779B97F4A7C15ULL, W1 = 0xBB67AE8584CAA73BULL;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t lo0 = M0 * c[0], hi0 = __umul64hi(M0, c[0]);
        const uint64_t lo1 = M1 * c[2], hi1 = __umul64hi(M1, c[2]);
        const uint64_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0;
        c[1] = lo1;
        c[2] = n2;
        c[3] = lo0;
        k0 += W0;
        k1 += W1;
    }
}

// Row r of column p: 32-bit word w = r / 4 of the stream (low half of 64-bit
// output w/2 first), 64-bit output q = w / 2 is word q % 4 of Philox block
// q / 4, generated from counter q / 4 + 1 (the counter is bumped before each
// block); the sign is the high bit of byte r % 4.
__global__ void philox_rademacher_kernel(const uint64_t* __restrict__ keys, int64_t P, int64_t rows,
                                         double* __restrict__ out) {
    const int64_t n = P * rows;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = t / rows, r = t - p * rows;
        const uint64_t w = (uint64_t)r >> 2, q = w >> 1, blk = q >> 2;
        uint64_t c[4] = {blk + 1, 0, 0, 0};
        if (c[0] == 0) c[1] = 1;  // 256-bit counter carry (blk + 1 overflowed)
        philox4x64_10(c, keys[2 * p], keys[2 * p + 1]);
        const int qi = (int)(q & 3);
        const uint64_t v = qi == 0 ? c[0] : qi == 1 ? c[1] : qi == 2 ? c[2] : c[3];
        const uint32_t word = (w & 1) ? (uint32_t)(v >> 32) : (uint32_t)v;
        const uint32_t byte = (word >> (8 * (r & 3))) & 0xFFu;
        out[p * rows + r] = (byte & 0x80u) ? 1.0 : -1.0;
    }
}

unsigned grid_for(int64_t n) {
    const int64_t b = (n + 255) / 256;
    return (unsigned)(b < 148 * 64 ? (b > 0 ? b : 1) : 148 * 64);
}

}  // namespace

void launch_gxe_source_finalize(const double* Y, int64_t N, int64_t N_pad, int64_t C, int cols_half,
                                const double* env, int64_t env_ld, int env_start, double* target,
                                int64_t t_ld, cudaStream_t st) {
    if (N * C == 0) return;
    gxe_source_finalize_kernel<<<grid_for(N * C), 256, 0, st>>>(Y, N, N_pad, C, cols_half, env,
                                                                 env_ld, env_start, target, t_ld);
    count_launch();
}

void launch_col_dots(const double* panel, int64_t p_ld, int64_t N, int64_t C, const double* basis,
                     int64_t b_ld, int nb, int squares, double* out, cudaStream_t st,
                     int64_t group_cols, int64_t group_stride) {
    if (C == 0) return;
    if (group_cols <= 0) group_cols = C;
    auto f = squares ? col_dots_kernel<1, true>
           : nb <= 1 ? col_dots_kernel<1, false>
           : nb <= 2 ? col_dots_kernel<2, false>
           : nb <= 4 ? col_dots_kernel<4, false>
           : nb <= 8 ? col_dots_kernel<8, false> : col_dots_kernel<kMaxBasis, false>;
    f<<<(unsigned)C, kDotThreads, 0, st>>>(panel, p_ld, N, basis, b_ld, nb, group_cols, group_stride,
                                           out);
    count_launch();
}

int col_dots_max_basis() { return kMaxBasis; }

void launch_sub_lowrank(double* panel, int64_t ld, int64_t N, int64_t C, const double* basis,
                        int64_t b_ld, int nb, const double* coef, int ones_last, double last_scale,
                        cudaStream_t st, int64_t group_cols, int64_t group_stride) {
    if (N * C == 0 || nb == 0) return;
    if (group_cols <= 0) group_cols = C;
    const dim3 grid((unsigned)std::min<int64_t>((N + 255) / 256, 64),
                    (unsigned)std::min<int64_t>(C, 65535));
    sub_lowrank_kernel<<<grid, 256, 0, st>>>(panel, ld, N, C, basis, b_ld, nb, coef, ones_last,
                                             last_scale, group_cols, group_stride);
    count_launch();
}

void launch_gxe_pair(const double* S, int64_t s_ld, int64_t N, int64_t N_pad, int64_t C,
                     int64_t cols_per_group, const double* w, int64_t w_ld, int w_first,
                     double* Ypair, cudaStream_t st) {
    if (N_pad * C == 0) return;
    gxe_pair_kernel<<<grid_for(N_pad * C), 256, 0, st>>>(S, s_ld, N, N_pad, C, cols_per_group, w,
                                                          w_ld, w_first, Ypair);
    count_launch();
}

void launch_gxe_target_finalize(const double* S, int64_t L, int Kp, int K, int T, const double* sx,
                                const double* sw, int64_t s_ld, const int32_t* ranks, int64_t N,
                                int env_start, int64_t total, int64_t block_start, double* a0,
                                double* a1, double* a2, double* a3, cudaStream_t st) {
    if (L * Kp == 0) return;
    gxe_target_finalize_kernel<<<grid_for(L * Kp), 256, 0, st>>>(
        S, L, Kp, K, T, sx, sw, s_ld, ranks, N, env_start, total, block_start, a0, a1, a2, a3);
    count_launch();
}

void launch_scale(double* x, int64_t n, double s, cudaStream_t st) {
    if (n == 0) return;
    scale_kernel<<<grid_for(n), 256, 0, st>>>(x, n, s);
    count_launch();
}

void launch_gxe_check(const double* probes, int64_t np, const double* sx, const double* sw,
                      int64_t ns, const double* annot, int64_t na, unsigned* flag, cudaStream_t st) {
    gxe_check_kernel<<<grid_for(std::max(std::max(np, ns), na)), 256, 0, st>>>(probes, np, sx, sw, ns,
                                                                              annot, na, flag);
    count_launch();
}

// Source member lists, in the SNPs' order: rows of block SNPs [a, b) whose
// annotation weight is positive, one CTA per annotation column k, to
// rows + k * cap and their number to count[k].
//
// Latency-bound (a column's chunks of 1,024 SNPs follow one another).  Lists
// built on the host from copies of the annotation and scales took 1 of the 3.6 ms
// of a reference over 20,000 samples and SNPs, 4 exposures; these two kernels take 32 us.
__device__ __forceinline__ double gxe_weight(double a, int is_sqrt) {
    return is_sqrt ? a : sqrt(a > 0.0 ? a : 0.0);
}

__global__ void gxe_members_kernel(const double* __restrict__ annot, int64_t L, int64_t a, int64_t b,
                                   int is_sqrt, int64_t cap, int32_t* __restrict__ rows,
                                   int* __restrict__ count) {
    __shared__ int warp_n[32];
    const int k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int64_t j0 = a; j0 < b; j0 += 1024) {
        const int64_t j = j0 + threadIdx.x;
        const bool in = j < b && gxe_weight(annot[k * L + j], is_sqrt) > 0.0;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) warp_n[warp] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            const int n = warp_n[w];
            if (w < warp) before += n;
            all += n;
        }
        if (in) rows[k * cap + base + before + __popc(m & ((1u << lane) - 1u))] = (int32_t)(j - a);
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) count[k] = base;
}

// Super-bin gi = (e 2 + h) K + k from off[gi] on: its rows and sqrt(a_jk) s_h,e[j],
// then padding members (row 0, scale 0) up to off[gi + 1].
__global__ void gxe_lists_kernel(const double* __restrict__ annot, const double* __restrict__ sx,
                                 const double* __restrict__ sw, int64_t L, int64_t a, int K,
                                 int is_sqrt, int64_t cap, const int32_t* __restrict__ rows,
                                 const int* __restrict__ count, const int64_t* __restrict__ off,
                                 int32_t* __restrict__ rowind, double* __restrict__ sc) {
    const int gi = blockIdx.y, k = gi % K, h = (gi / K) & 1, e = gi / (2 * K);
    const int64_t o = off[gi], p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= off[gi + 1] - o) return;
    int32_t r = 0;
    double v = 0.0;
    if (p < count[k]) {
        r = rows[k * cap + p];
        v = gxe_weight(annot[k * L + a + r], is_sqrt) * (h == 0 ? sx : sw)[e * L + a + r];
    }
    rowind[o + p] = r;
    sc[o + p] = v;
}

void launch_gxe_members(const double* annot, int64_t L, int64_t a, int64_t b, int K, int is_sqrt,
                        int64_t cap, int32_t* rows, int* count, cudaStream_t st) {
    if (K == 0) return;
    gxe_members_kernel<<<(unsigned)K, 1024, 0, st>>>(annot, L, a, b, is_sqrt, cap, rows, count);
    count_launch();
}

void launch_gxe_lists(const double* annot, const double* sx, const double* sw, int64_t L, int64_t a,
                      int K, int64_t G, int is_sqrt, int64_t cap, const int32_t* rows,
                      const int* count, const int64_t* off, int64_t longest, int32_t* rowind,
                      double* sc, cudaStream_t st) {
    if (G == 0 || longest == 0) return;
    gxe_lists_kernel<<<dim3((unsigned)((longest + 255) / 256), (unsigned)G), 256, 0, st>>>(
        annot, sx, sw, L, a, K, is_sqrt, cap, rows, count, off, rowind, sc);
    count_launch();
}

void launch_philox_rademacher(const uint64_t* keys, int64_t P, int64_t rows, double* out,
                              cudaStream_t st) {
    if (P * rows == 0) return;
    philox_rademacher_kernel<<<grid_for(P * rows), 256, 0, st>>>(keys, P, rows, out);
    count_launch();
}

}  // namespace lds
