// Device pieces of the generalized per-variant GxE two-pass estimator
// (ldscore/generalized_gxe_pass1.py, generalized_gxe_pass2.py): the global
// variant x probe Rademacher stream and the component-kernel diagonals.
// The genotype products of both passes run on the tensor-core kernels
// (lds_umma_p1.cu, lds_umma.cu) through lds_geno_source_product /
// lds_geno_target_product.
#include <algorithm>
#include <cstdint>

#include "lds_device.cuh"
#include "lds_internal.h"

namespace lds {

namespace {

// Annotations whose component sums a thread of the diagonal kernel keeps.
__host__ __device__ constexpr int diag_annots(int P) { return P >= 16 ? 1 : 16 / P; }

// splitmix64 with the increment applied first (generalized_gxe_variant.py
// _splitmix64), and the addressable sign of global_probe_sign.
__device__ __forceinline__ uint64_t splitmix64_step(uint64_t v) {
    v += 0x9E3779B97F4A7C15ULL;
    v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ULL;
    v = (v ^ (v >> 27)) * 0x94D049BB133111EBULL;
    return v ^ (v >> 31);
}

// out[b * L + j] = sign(root, variant v0 + j, probe p0 + b) (column-major L x B).
__global__ void global_probes_kernel(uint64_t root_state, int64_t v0, int64_t L, int64_t p0,
                                     int64_t B, double* __restrict__ out) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= L * B) return;
    const int64_t j = idx % L, b = idx / L;
    uint64_t s = root_state;
    s ^= splitmix64_step((uint64_t)(v0 + j) + 0xD2B74407B1CE6E93ULL);
    s ^= splitmix64_step((uint64_t)(p0 + b) + 0xCA5A826395121157ULL);
    out[idx] = (splitmix64_step(s) >> 63) ? 1.0 : -1.0;
}

constexpr int kDiagThreads = 128;   // samples per CTA
constexpr int kDiagRows = 32;       // SNPs staged at a time

// num[c * N + i] += sum_j a[j, k] kf(p) f_q(i, j) f_r(i, j) for the components
// c = k * P + p of this CTA's annotations, with the projected contextual
// features f_q(i, j) = phi_q(i) x_ij - sum_r F(i, r) coef[j, q, r] (pass-2
// feature tiles, generalized_gxe_pass2.py:528-562) and x_ij the image's
// standardized genotype (0 on a missing call); pairs p = (q, r) diagonals first,
// then lexicographic off-diagonals, kf 1 on the diagonal and 2 off it.  One
// thread per sample.
//
// Bound by FP64 issue: about Q (R + 2) + 3 P + 2 K P operations per genotype.
// The SNPs are split over blockIdx.z (a grid of sample tiles alone left most SMs
// idle), tiles of 32 SNPs' codes, statistics, coefficients and annotations go
// through shared memory, and Q is a template argument so that the features and
// their products stay in registers.  A split's sums go to part[z][c][i], added
// in order by component_diag_reduce_kernel; a single part adds to num itself.
// N = 4,000, M = 6,000, Q = R = K = 2: 10.2 ms -> 99 us.
template <int Q, int RM>
__global__ void __launch_bounds__(kDiagThreads)
    component_diag_kernel(const uint8_t* __restrict__ codes, int64_t nbp,
                          const double* __restrict__ mean, const double* __restrict__ sdinv,
                          int64_t j0, int64_t L, int64_t N, const double* __restrict__ annot,
                          int K, const double* __restrict__ basis,
                          const double* __restrict__ fixed, int R,
                          const double* __restrict__ coef, int64_t rows_per_part,
                          double* __restrict__ part, double* __restrict__ num) {
    constexpr int P = Q * (Q + 1) / 2;
    constexpr int KC = diag_annots(P);   // annotations per CTA
    __shared__ uint4 s_codes[kDiagRows * 2];
    __shared__ double s_mean[kDiagRows], s_sd[kDiagRows];
    __shared__ double s_annot[kDiagRows * KC];
    __shared__ double s_coef[RM > 0 ? kDiagRows * Q * RM : 1];
    const int64_t i0 = (int64_t)blockIdx.x * kDiagThreads, i = i0 + threadIdx.x;
    const int k0 = blockIdx.y * KC, nk = min(KC, K - k0);
    const bool live = i < N;
    double phi[Q], frow[RM > 0 ? RM : 1], acc[KC * P];
#pragma unroll
    for (int q = 0; q < Q; ++q) phi[q] = live ? basis[(int64_t)q * N + i] : 0.0;
#pragma unroll
    for (int r = 0; r < RM; ++r) frow[r] = live && r < R ? fixed[(int64_t)r * N + i] : 0.0;
#pragma unroll
    for (int t = 0; t < KC * P; ++t) acc[t] = 0.0;
    const int64_t r0 = (int64_t)blockIdx.z * rows_per_part, r1 = min(L, r0 + rows_per_part);
    const int shift = 2 * (int)(threadIdx.x & 3);
    const uint8_t* row_codes = reinterpret_cast<const uint8_t*>(s_codes) + (threadIdx.x >> 2);
    for (int64_t jb = r0; jb < r1; jb += kDiagRows) {
        const int rows = (int)min((int64_t)kDiagRows, r1 - jb);
        __syncthreads();
        {
            // 32 bytes of every row: this CTA's 128 samples (rows are padded to
            // a multiple of 64 bytes, so both halves are inside the image)
            const int r = threadIdx.x >> 1, c = threadIdx.x & 1;
            if (r < rows)
                s_codes[threadIdx.x] = *reinterpret_cast<const uint4*>(
                    codes + (j0 + jb + r) * nbp + (i0 >> 2) + 16 * c);
        }
        if (threadIdx.x < rows) {
            s_mean[threadIdx.x] = mean[j0 + jb + threadIdx.x];
            s_sd[threadIdx.x] = sdinv[j0 + jb + threadIdx.x];
        }
        for (int t = threadIdx.x; t < rows * KC; t += kDiagThreads) {
            const int r = t / KC, k = t - r * KC;
            s_annot[t] = k < nk ? annot[(jb + r) * K + k0 + k] : 0.0;
        }
        if (RM > 0)
            for (int t = threadIdx.x; t < rows * Q * RM; t += kDiagThreads) {
                const int rq = t / RM, r = t - rq * RM;
                s_coef[t] = r < R ? coef[(jb * Q + rq) * R + r] : 0.0;
            }
        __syncthreads();
        for (int jl = 0; jl < rows; ++jl) {
            const uint32_t code = ((uint32_t)row_codes[jl * 32] >> shift) & 3u;
            const double g = (double)((code >> 1) + (code == 3u));
            const double x = code == 1u ? 0.0 : s_sd[jl] * (g - s_mean[jl]);
            double f[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                double v = phi[q] * x;
                const double* cj = s_coef + (jl * Q + q) * RM;
#pragma unroll
                for (int r = 0; r < RM; ++r) v -= frow[r] * cj[r];
                f[q] = v;
            }
            double prod[P];
#pragma unroll
            for (int q = 0; q < Q; ++q) prod[q] = f[q] * f[q];
            int p = Q;
#pragma unroll
            for (int q = 0; q < Q - 1; ++q)
#pragma unroll
                for (int r = q + 1; r < Q; ++r) prod[p++] = 2.0 * f[q] * f[r];
#pragma unroll
            for (int k = 0; k < KC; ++k) {
                const double a = s_annot[jl * KC + k];
                if (a == 0.0) continue;   // (the same for every sample)
#pragma unroll
                for (int t = 0; t < P; ++t) acc[k * P + t] += a * prod[t];
            }
        }
    }
    if (!live) return;
#pragma unroll
    for (int k = 0; k < KC; ++k)
        if (k < nk)
#pragma unroll
            for (int t = 0; t < P; ++t) {
                const int64_t o = (int64_t)((k0 + k) * P + t) * N + i;
                if (gridDim.z > 1) part[(int64_t)blockIdx.z * K * P * N + o] = acc[k * P + t];
                else num[o] += acc[k * P + t];
            }
}

// num[o] += the parts' sums in order.
__global__ void component_diag_reduce_kernel(const double* __restrict__ part, int nparts, int64_t n,
                                             double* __restrict__ num) {
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    double s = 0.0;
    for (int z = 0; z < nparts; ++z) s += part[(int64_t)z * n + o];
    num[o] += s;
}

// Pass-2 scores of one variant block, one CTA per variant row jl: the row's
// cross sketches cross[c] = s_j cs[c] (G^T y_c - mu_j O^T y_c) / rr from the
// exact raw digit products (column c = (k * B + b) * F + f of the
// right-hand side, raw row stride raw_ld), then
//   out[jl][tp][k * P + sp] = (1 / B) sum over the orientation terms (f1, f2)
//   of (tp, sp) of sum_b cross[(k B + b) F + f1] cross[(k B + b) F + f2]
// (generalized_gxe_pass2.py:600-676).
__global__ void gen_rows_kernel(const long long* __restrict__ raw_g,
                                const long long* __restrict__ raw_o, int64_t raw_ld,
                                const double* __restrict__ cs, const double* __restrict__ mean,
                                const double* __restrict__ sdinv, int64_t j0, double inv_rr, int K,
                                int B, int F, int P, const int* __restrict__ term_off,
                                const int* __restrict__ term_f1, const int* __restrict__ term_f2,
                                double* __restrict__ out) {
    extern __shared__ double cross[];
    const int64_t jl = blockIdx.x, j = j0 + jl;
    const int cols = K * B * F, C = K * P, nout = P * C;
    const double mu = mean[j], sd = sdinv[j];
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
        const int64_t q = jl * raw_ld + c;
        cross[c] = sd * cs[c] * ((double)raw_g[q] - mu * (double)raw_o[q]) * inv_rr;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < nout; o += blockDim.x) {
        const int tp = o / C, c = o - tp * C, k = c / P, sp = c - k * P;
        double acc = 0.0;
        for (int t = term_off[tp * P + sp]; t < term_off[tp * P + sp + 1]; ++t) {
            const double* x1 = cross + (int64_t)k * B * F + term_f1[t];
            const double* x2 = cross + (int64_t)k * B * F + term_f2[t];
            double s = 0.0;
            for (int b = 0; b < B; ++b) s += x1[b * F] * x2[b * F];
            acc += s;
        }
        out[jl * nout + o] = acc / (double)B;
    }
}

// directed[c1][c2] += sum_jl a[j0 + jl][k1] rows[jl][p1][c2], c1 = k1 P + p1,
// in two steps: sums over chunks of variants, then one warp per entry over the
// chunks, both in a fixed order.  A CTA takes 256 entries of a chunk; the chunks are
// of at least kDirRows variants, and as many as give kDirCtas CTAs, which also bounds
// their sums (one CTA for all entries of a chunk left C = 291 with 94 CTAs).
// 6,000 variants, C = 6: 786 -> 25 us (one thread per entry over all variants);
// C = 291: 883 us (1,298; with one CTA per chunk 3,597).
constexpr int kDirRows = 64, kDirThreads = 256, kDirCtas = 8 * 148;

// Chunks of L variants for n entries.
static int64_t gen_directed_chunks(int64_t L, int64_t n) {
    const int64_t groups = (n + kDirThreads - 1) / kDirThreads;
    return std::max<int64_t>(1, std::min((L + kDirRows - 1) / kDirRows,
                                         (kDirCtas + groups - 1) / groups));
}

__global__ void __launch_bounds__(kDirThreads)
    gen_directed_kernel(const double* __restrict__ rows, int64_t L, int64_t rows_per_chunk,
                        const double* __restrict__ annot, int64_t j0, int K, int P,
                        double* __restrict__ part) {
    const int C = K * P, idx = (int)(blockIdx.x * kDirThreads + threadIdx.x);
    if (idx >= C * C) return;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_chunk, r1 = min(L, r0 + rows_per_chunk);
    const int c1 = idx / C, c2 = idx - c1 * C, k1 = c1 / P, p1 = c1 - k1 * P;
    double s = 0.0;
#pragma unroll 8
    for (int64_t jl = r0; jl < r1; ++jl)
        s += annot[(j0 + jl) * K + k1] * rows[(jl * P + p1) * C + c2];
    part[(int64_t)blockIdx.y * C * C + idx] = s;
}

__global__ void gen_directed_reduce_kernel(const double* __restrict__ part, int64_t nchunks, int n,
                                           double* __restrict__ directed) {
    const int idx = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (idx >= n) return;
    double s = 0.0;
    for (int64_t z = lane; z < nchunks; z += 32) s += part[z * n + idx];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) directed[idx] += s;
}

// Pass 2's right-hand side from the contextual sources
// (GeneralizedGxEPass2Executor's family columns, generalized_gxe_pass2.py):
// column (k B + b) F + f = phi_t o sources[k, s][:, b] for family f = (t, s).
// S holds the sources as K Q B rows of N_pad samples, basis is N x Q
// row-major; Y gets one column of N_pad samples per (k, b, f), rows N and
// beyond left as they are (zero).
__global__ void gen_assemble_rhs_kernel(const double* __restrict__ S, int64_t Np,
                                        const double* __restrict__ basis, int Q,
                                        const int* __restrict__ fam_t,
                                        const int* __restrict__ fam_s, int B, int F, int64_t N,
                                        double* __restrict__ Y) {
    const int col = blockIdx.y;
    const int f = col % F, kb = col / F;
    const int b = kb % B, k = kb / B;
    const int t = fam_t[f], s = fam_s[f];
    const double* src = S + ((int64_t)(k * Q + s) * B + b) * Np;
    double* dst = Y + (int64_t)col * Np;
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < N;
         n += (int64_t)gridDim.x * blockDim.x)
        dst[n] = src[n] * basis[n * Q + t];
}

// Pass 1's projection of the contextual sources off the fixed effects
// (GeneralizedGxEPass1Executor, generalized_gxe_pass1.py:718-757), one CTA per
// (annotation k, basis coordinate q, probe b): with w = basis[:, q] o
// base[k, b], coef = fixed^T w, the row is p = w - fixed coef, written to out;
// leak = fixed^T p (R values) and p^T p are reduced in a fixed order for the
// host's leakage check.  base is K B rows of N samples, basis N x Q and fixed
// N x R row-major.
constexpr int kProjThreads = 256;

// Sums v[0..n) over the CTA (warp trees, then warps in order); the totals
// land in tot[0..n) for every thread.
template <int kMax>
__device__ __forceinline__ void block_sum(double (&v)[kMax], int n, double (*red)[kMax],
                                          double* tot) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int r = 0; r < kMax; ++r) {
        if (r >= n) break;
        double x = v[r];
        for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[w][r] = x;
    }
    __syncthreads();
    if (threadIdx.x < n) {
        double t = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i][threadIdx.x];
        tot[threadIdx.x] = t;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kProjThreads)
    gen_project_kernel(const double* __restrict__ base, const double* __restrict__ basis, int Q,
                       const double* __restrict__ fixed, int R, int B, int64_t N,
                       double* __restrict__ out, double* __restrict__ leak,
                       double* __restrict__ pn2) {
    constexpr int kM = kGenMaxR + 1;
    __shared__ double red[kProjThreads / 32][kM];
    __shared__ double coef[kM];
    const int row = blockIdx.x;  // (k Q + q) B + b
    const int b = row % B, kq = row / B, q = kq % Q, k = kq / Q;
    const double* src = base + ((int64_t)k * B + b) * N;
    double* dst = out + (int64_t)row * N;
    double acc[kM];
#pragma unroll
    for (int r = 0; r < kM; ++r) acc[r] = 0.0;
    for (int64_t n = threadIdx.x; n < N; n += blockDim.x) {
        const double w = src[n] * basis[n * Q + q];
#pragma unroll
        for (int r = 0; r < kGenMaxR; ++r)
            if (r < R) acc[r] += w * fixed[n * R + r];
    }
    block_sum<kM>(acc, R, red, coef);
#pragma unroll
    for (int r = 0; r < kM; ++r) acc[r] = 0.0;  // leak[0..R), p^T p at R
    for (int64_t n = threadIdx.x; n < N; n += blockDim.x) {
        const double w = src[n] * basis[n * Q + q];
        double fc = 0.0;
#pragma unroll
        for (int r = 0; r < kGenMaxR; ++r)
            if (r < R) fc += fixed[n * R + r] * coef[r];
        const double p = w - fc;
        dst[n] = p;
#pragma unroll
        for (int r = 0; r < kGenMaxR; ++r)
            if (r < R) acc[r] += p * fixed[n * R + r];
        acc[R < kGenMaxR ? R : kGenMaxR] += p * p;
    }
    block_sum<kM>(acc, R + 1, red, coef);
    if (threadIdx.x < R) leak[(int64_t)row * R + threadIdx.x] = coef[threadIdx.x];
    if (threadIdx.x == 0) pn2[row] = coef[R];
}

}  // namespace

void launch_gen_project(const double* base, const double* basis, int Q, const double* fixed,
                        int R, int K, int B, int64_t N, double* out, double* leak, double* pn2,
                        cudaStream_t st) {
    const int rows = K * Q * B;
    if (rows <= 0 || N <= 0) return;
    gen_project_kernel<<<(unsigned)rows, kProjThreads, 0, st>>>(base, basis, Q, fixed, R, B, N, out,
                                                               leak, pn2);
    count_launch();
}

void launch_gen_assemble_rhs(const double* S, int64_t Np, const double* basis, int Q,
                             const int* fam_t, const int* fam_s, int K, int B, int F, int64_t N,
                             double* Y, cudaStream_t st) {
    const int cols = K * B * F;
    if (cols <= 0 || N <= 0) return;
    const unsigned bx = (unsigned)std::min<int64_t>((N + 255) / 256, 64);
    gen_assemble_rhs_kernel<<<dim3(bx, (unsigned)cols), 256, 0, st>>>(S, Np, basis, Q, fam_t, fam_s,
                                                                     B, F, N, Y);
    count_launch();
}

size_t gen_rows_smem_bytes(int cols) { return (size_t)cols * sizeof(double); }

void launch_gen_rows(const long long* raw_g, const long long* raw_o, int64_t raw_ld,
                     const double* cs, const double* mean, const double* sdinv, int64_t j0,
                     int64_t L, double inv_rr, int K, int B, int F, int P, const int* term_off,
                     const int* term_f1, const int* term_f2, double* out, cudaStream_t st) {
    if (L <= 0) return;
    const size_t smem = gen_rows_smem_bytes(K * B * F);
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        cudaFuncSetAttribute(gen_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kGenRowsMaxSmem);
    });
    gen_rows_kernel<<<(unsigned)L, 256, smem, st>>>(raw_g, raw_o, raw_ld, cs, mean, sdinv, j0,
                                                     inv_rr, K, B, F, P, term_off, term_f1,
                                                     term_f2, out);
    count_launch();
}

int64_t gen_directed_part_elems(int64_t L, int K, int P) {
    const int64_t n = (int64_t)K * P * K * P;
    return gen_directed_chunks(L, n) * n;
}

void launch_gen_directed(const double* rows, int64_t L, const double* annot, int64_t j0, int K,
                         int P, double* part, double* directed, cudaStream_t st) {
    const int C = K * P, n = C * C;
    if (L <= 0 || C <= 0) return;
    const int64_t chunks = gen_directed_chunks(L, n), per = (L + chunks - 1) / chunks;
    const int64_t used = (L + per - 1) / per;
    gen_directed_kernel<<<dim3((unsigned)((n + kDirThreads - 1) / kDirThreads), (unsigned)used),
                          kDirThreads, 0, st>>>(rows, L, per, annot, j0, K, P, part);
    count_launch();
    gen_directed_reduce_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(part, used, n, directed);
    count_launch();
}

void launch_global_probes(uint64_t root_state, int64_t v0, int64_t L, int64_t p0, int64_t B,
                          double* out, cudaStream_t st) {
    const int64_t n = L * B;
    if (n <= 0) return;
    global_probes_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(root_state, v0, L, p0, B,
                                                                      out);
    count_launch();
}

// SNP parts of a component-diagonal launch: enough CTAs for six per SM, at
// least one staged tile each, and at most 256 MB of partial sums.
int component_diag_parts(int64_t N, int64_t L, int K, int Q) {
    const int P = Q * (Q + 1) / 2;
    const int64_t ctas = (N + kDiagThreads - 1) / kDiagThreads *
                         ((K + diag_annots(P) - 1) / diag_annots(P));
    const int64_t want = (148 * 6 + ctas - 1) / std::max<int64_t>(ctas, 1);
    const int64_t fit = ((int64_t)256 << 20) / (8 * N * K * P);
    const int64_t parts = std::min(std::min(want, (L + kDiagRows - 1) / kDiagRows), fit);
    return (int)std::max<int64_t>(parts, 1);
}

template <int Q, int RM>
static void diag_launch(const uint8_t* codes, int64_t nbp, const double* mean, const double* sdinv,
                        int64_t j0, int64_t L, int64_t N, const double* annot, int K,
                        const double* basis, const double* fixed, int R, const double* coef,
                        double* part, double* num, cudaStream_t st) {
    constexpr int P = Q * (Q + 1) / 2;
    const int parts = component_diag_parts(N, L, K, Q);
    const int64_t per = ((L + parts - 1) / parts + kDiagRows - 1) / kDiagRows * kDiagRows;
    const int used = (int)((L + per - 1) / per);
    dim3 grid((unsigned)((N + kDiagThreads - 1) / kDiagThreads),
              (unsigned)((K + diag_annots(P) - 1) / diag_annots(P)), (unsigned)used);
    component_diag_kernel<Q, RM><<<grid, kDiagThreads, 0, st>>>(
        codes, nbp, mean, sdinv, j0, L, N, annot, K, basis, fixed, R, coef, per, part, num);
    count_launch();
    if (used > 1) {
        const int64_t n = (int64_t)K * P * N;
        component_diag_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(part, used, n, num);
        count_launch();
    }
}

template <int Q>
static void diag_launch_r(const uint8_t* codes, int64_t nbp, const double* mean,
                          const double* sdinv, int64_t j0, int64_t L, int64_t N,
                          const double* annot, int K, const double* basis, const double* fixed,
                          int R, const double* coef, double* part, double* num, cudaStream_t st) {
    static_assert(kGenMaxR == 16, "the widest instance holds every fixed effect");
    auto f = R == 0 ? diag_launch<Q, 0> : R <= 4 ? diag_launch<Q, 4> : diag_launch<Q, 16>;
    f(codes, nbp, mean, sdinv, j0, L, N, annot, K, basis, fixed, R, coef, part, num, st);
}

void launch_component_diag(const uint8_t* codes, int64_t nbp, const double* mean,
                           const double* sdinv, int64_t j0, int64_t L, int64_t N,
                           const double* annot, int K, const double* basis, int Q,
                           const double* fixed, int R, const double* coef, double* part,
                           double* num, cudaStream_t st) {
    if (N <= 0 || L <= 0 || K <= 0) return;
    static_assert(kGenMaxQ == 6, "one instance per basis count");
    auto f = Q == 1 ? diag_launch_r<1> : Q == 2 ? diag_launch_r<2> : Q == 3 ? diag_launch_r<3>
           : Q == 4 ? diag_launch_r<4> : Q == 5 ? diag_launch_r<5> : diag_launch_r<6>;
    f(codes, nbp, mean, sdinv, j0, L, N, annot, K, basis, fixed, R, coef, part, num, st);
}

}  // namespace lds
