// Exact windowed LD scores on tcgen05 tensor cores (the deterministic
// estimator of compute_windowed_ld_chr_impl, winldcore.cpp:783-931).
//
// For SNPs j, i of one window the reference forms r_ij = x~_j . x~_i / N from
// restandardized columns (winldcore.cpp:215-267, :480-594).  Mathematically
// r_ij = c_ji / sqrt(c_jj c_ii) with
//   c_ji = sum_n o_jn o_in (g_jn - mu_j)(g_in - mu_i)
//        = GG - mu_i GO - mu_j OG + mu_j mu_i OO,
// where GG = sum g_j g_i, GO = sum g_j o_i, OG = sum o_j g_i, OO = sum o_j o_i
// are exact integer Gram sums of the decoded planes (g in {0,1,2}, o in {0,1}).
// One CTA owns a tile J of 128 SNPs and walks a run of partner tiles I: per
// K-step of 128 samples it decodes the packed codes of both tiles into
// SWIZZLE_128B int8 operands (A = G_J and O_J, B = [G_I | O_I], 256 rows) and
// issues two tcgen05.mma.kind::i8 (M=128, N=256, K=32) x 4 into TMEM:
//   columns   0..255: G_J [G_I | O_I]^T  -> GG | GO
//   columns 256..511: O_J [G_I | O_I]^T  -> OG | OO
// exact in int32 (|sums| <= 4N).  r is symmetric, so each unordered pair of
// tiles is formed once: the epilogue turns the sums into f(r) = r^2 or the
// unbiased r^2 - (1 - r^2)/(corr_dim - 1) in FP64 (winldcore.cpp:409-432),
// zeroes pairs outside each SNP's partner interval (:434-478), and adds f(r)
// annot[i, :] for the rows j of J and, off the diagonal, f(r) annot[j, :] for
// the columns i of I (transposed through a few KB of shared memory per warp).
// The sums go to units of 128 SNPs x K doubles of their own; a second kernel
// adds a tile's units in a fixed order, so results are deterministic.
//
// Bound by shared-memory bandwidth: per K-step 96 KB of MMA operand reads, 64 KB
// of decoded operands and 16 KB of packed rows are 1,375 cycles at 128 bytes each
// (MMA 1,024); it takes about 1,650.  N = 50,000, 12,000 SNPs with partners 2,000
// to each side: 7.54 -> 3.6 ms (before: both orders of every pair, and four
// decoding warps for 256 operand rows).
//
// Roles (576 threads): warp 0 TMEM allocation and MMA issue (the warp walks the
// loop uniformly, one elected thread issues); warps 1-16 decode, two groups of
// eight that take alternate K-steps, four warps for tile J's rows and four for
// tile I's; after each partner tile every four of them read out a quarter of its
// columns; warp 17 is the TMA producer of packed-code tiles (loads of 32-byte row
// pieces by the decoding threads themselves kept the load-store pipe as busy as
// their operand stores: 2,300 cycles per K-step).  Every mbarrier wait is
// bounded; on timeout the kernel records a code in `status`, stops issuing work,
// drains its copies and MMAs, and releases TMEM.
#include <algorithm>
#include <cstdint>

#include "lds_internal.h"
#include "lds_tc.cuh"

namespace lds {
namespace gram {

using namespace umma;

constexpr int kBM = kGramTile;     // SNPs per tile
constexpr int kBK = 128;           // samples per K-step
constexpr int kTile = kBM * kBK;   // 16 KB int8 operand tile
constexpr int kStages = 3;         // decoded operand stages: G_J, O_J, G_I, O_I (64 KB)
constexpr int kDecGroups = 2;      // group d decodes the K-steps it with it % 2 == d
constexpr int kDecWarps = 8;       // warps of a group: tile J's rows, tile I's rows
constexpr int kPk = kDecGroups;    // packed-code slots, one per group (J + I rows)
constexpr int kPkBytes = 2 * kBM * 32;
constexpr int kThreads = 64 + 32 * kDecGroups * kDecWarps;
constexpr int kColSets = kDecGroups * kDecWarps / 4;   // epilogue: warps by quarter of the columns
constexpr int kSetCols = kBM / kColSets;
constexpr uint32_t kTmemCols = 512;
constexpr int kCB = 4;             // columns transposed at a time
constexpr int kCLd = 33;           // row stride of a transposed column (doubles)
static_assert(kColSets == kGramRowUnits, "one row unit per set of columns");

__host__ __device__ constexpr uint32_t stage_off(int s) { return (uint32_t)s * 4 * kTile; }
__host__ __device__ constexpr uint32_t pk_off(int s) {
    return stage_off(kStages) + (uint32_t)s * kPkBytes;
}
__host__ __device__ constexpr uint32_t bar_off() { return pk_off(kPk); }
__host__ __device__ constexpr uint32_t col_off() { return bar_off() + 256; }
constexpr size_t kSmemBytes =
    (size_t)col_off() + (size_t)kDecGroups * kDecWarps * kCB * kCLd * 8 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

// KC: annotation columns per epilogue pass.
template <int KC>
__global__ void __launch_bounds__(kThreads, 1)
    gram_ld_kernel(const __grid_constant__ CUtensorMap tmC, GramArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (a plain offset keeps shared-space accesses)
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + bar_off());
    uint64_t* pk_full = bars;                    // [kPk] packed rows landed (TMA)
    uint64_t* pk_empty = pk_full + kPk;          // [kPk] packed rows used by the decoders
    uint64_t* full = pk_empty + kPk;             // [kStages] operands decoded
    uint64_t* empty = full + kStages;            // [kStages] operands consumed by the MMAs
    uint64_t* acc_full = empty + kStages;        // accumulators hold a finished tile pair
    uint64_t* acc_empty = acc_full + 1;          // accumulators read out
    uint64_t* mma_done = acc_empty + 1;          // drain of the issuer's MMAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const GramItem item = a.items[blockIdx.x];
    const int64_t jrow0 = item.jrow0, irow0 = item.irow0;
    const int nI = item.tiles;

    if (tid == 0) {
        for (int s = 0; s < kPk; ++s) {
            mbar_init(&pk_full[s], 1);
            mbar_init(&pk_empty[s], kDecWarps);
        }
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], kDecWarps);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kDecGroups * kDecWarps);
        mbar_init(mma_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto fail = [&](int code) {
        atomicCAS(a.status, 0u, (unsigned)code);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ---------------- MMA issuer ----------------
        const uint32_t idesc = idesc_i8(kBM, 256);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = 0; t < nI && ok; ++t) {
            if (t > 0 && !warp_wait(acc_empty, (uint32_t)(t - 1) & 1u, abort_flag)) {
                fail(32);
                break;
            }
            tc_fence_after();
            for (int kt = 0; kt < a.nkt; ++kt) {
                if (!warp_wait(&full[s], ph, abort_flag)) {
                    fail(33);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t dGJ = sw128_desc(smem + stage_off(s));
                const uint64_t dOJ = dGJ + (kTile >> 4), dB = dGJ + (2 * kTile >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kBK / 32; ++kk) {
                        const uint32_t acc = (kt | kk) ? 1u : 0u;
                        umma_i8(tmem, dGJ + 2 * kk, dB + 2 * kk, idesc, acc);
                        umma_i8(tmem + 256, dOJ + 2 * kk, dB + 2 * kk, idesc, acc);
                    }
                    umma_commit(&empty[s]);
                }
                __syncwarp();
                if (++s == kStages) { s = 0; ph ^= 1u; }
            }
            if (ok && elect_one()) umma_commit(acc_full);
            __syncwarp();
        }
        // Drain: every MMA issued here completes before TMEM is released.
        if (elect_one()) umma_commit(mma_done);
        __syncwarp();
        mbar_wait(mma_done, 0u);
    } else if (warp == kThreads / 32 - 1) {
        // ---------------- packed-code producer ----------------
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int t = 0; t < nI && ok; ++t)
                for (int kt = 0; kt < a.nkt; ++kt, ++it) {
                    const int s = it % kPk;
                    if (it >= kPk && !mbar_wait(&pk_empty[s], ((uint32_t)(it / kPk) & 1u) ^ 1u,
                                                abort_flag)) {
                        fail(31);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&pk_full[s], (uint32_t)kPkBytes);
                    tma_load_2d(smem + pk_off(s), &tmC, kt * 32, (int)jrow0, &pk_full[s]);
                    tma_load_2d(smem + pk_off(s) + kBM * 32, &tmC, kt * 32,
                                (int)(irow0 + (int64_t)kBM * t), &pk_full[s]);
                }
            // Drain: no copy may still be landing when the CTA exits.
            for (int j = max(0, it - kPk); j < it; ++j)
                mbar_wait(&pk_full[j % kPk], (uint32_t)(j / kPk) & 1u);
        }
    } else {
        // ---------------- decoders (warps 1..16) + epilogue ----------------
        const int dw = warp - 1, group = dw / kDecWarps;
        const int which = (dw >> 2) & 1;        // 0: tile J's rows, 1: tile I's
        const int r = (dw & 3) * 32 + lane;     // operand row this thread decodes
        const int cset = dw >> 2;               // columns this warp reads out
        const int q = warp & 3;                 // TMEM lane quadrant of this warp
        const int jl = q * 32 + lane;           // accumulator row (SNP of tile J)
        const int64_t j = jrow0 + jl;
        const bool jvalid = j < a.row1;
        const int64_t lo = jvalid ? (int64_t)a.lo[j - a.row0] : 0;
        const int64_t hi = jvalid ? (int64_t)a.hi[j - a.row0] : 0;
        const double mu_j = jvalid ? a.mean[j] : 0.0;
        const double rs_j = jvalid ? a.rs[j] : 0.0;
        const uint32_t rowoff = (uint32_t)(which * 2 * kTile + (r >> 3) * 1024 + (r & 7) * 128);
        double* const cols = reinterpret_cast<double*>(smem + col_off()) + dw * kCB * kCLd;
        const uint4* const pk = reinterpret_cast<const uint4*>(
            smem + pk_off(group) + which * kBM * 32 + r * 32);
        int it = 0, s = 0;
        uint32_t ph = 0, php = 0;
        for (int t = 0; t < nI; ++t) {
            for (int kt = 0; kt < a.nkt; ++kt, ++it) {
                if (it % kDecGroups == group) {
                    if (!warp_wait(&pk_full[group], php, abort_flag)) { fail(34); break; }
                    php ^= 1u;
                    const uint4 p0 = pk[0], p1 = pk[1];
                    // The slot goes back as soon as the rows are in registers: the
                    // arrival depends on the words that were read (a copy of them
                    // that the compiler cannot know to be equal), so no read of the
                    // slot can still be on its way.
                    const uint32_t words = p0.x ^ p0.y ^ p0.z ^ p0.w ^ p1.x ^ p1.y ^ p1.z ^ p1.w;
                    uint32_t same;
                    asm volatile("shfl.sync.bfly.b32 %0, %1, 0, 31, 0xffffffff;"
                                 : "=r"(same)
                                 : "r"(words));
                    __syncwarp();
                    if (lane == 0 && same == words) mbar_arrive(&pk_empty[group]);
                    if (it >= kStages && !warp_wait(&empty[s], ph ^ 1u, abort_flag)) {
                        fail(35);
                        break;
                    }
                    uint8_t* row = smem + stage_off(s) + rowoff;
                    decode_row_sw128(p0, p1, row, row + kTile, r);
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[s]);
                }
                if (++s == kStages) { s = 0; ph ^= 1u; }
            }
            if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
            // ---- epilogue of partner tile t: this warp's quarter of the columns ----
            if (!warp_wait(acc_full, (uint32_t)t & 1u, abort_flag)) { fail(36); break; }
            tc_fence_after();
            const int64_t ib = irow0 + (int64_t)kBM * t;
            const bool diag = ib == jrow0;
            // this item's column units of tile I: one per quadrant of J's rows
            const int64_t cu = item.col_unit + 4 * (t - (irow0 == jrow0 ? 1 : 0)) + q;
            const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16);
            for (int kc = 0; kc < a.K; kc += KC) {
                double acc[KC];
#pragma unroll
                for (int b = 0; b < KC; ++b) acc[b] = 0.0;
                for (int c0 = kSetCols * cset; c0 < kSetCols * (cset + 1); c0 += 16) {
                    if (ib + c0 >= a.row1) break;  // warp-uniform
                    double f[16];
                    {
                        int gg[16], go[16], og[16], oo[16];
                        __syncwarp();
                        tmem_ld16(tb + (uint32_t)c0, gg);
                        tmem_ld16(tb + 128u + (uint32_t)c0, go);
                        tmem_ld16(tb + 256u + (uint32_t)c0, og);
                        tmem_ld16(tb + 384u + (uint32_t)c0, oo);
                        tmem_wait_ld(gg);
                        tmem_wait_ld(go);
                        tmem_wait_ld(og);
                        tmem_wait_ld(oo);
#pragma unroll
                        for (int u = 0; u < 16; ++u) {
                            const int64_t i = min(ib + c0 + u, a.row1 - 1);  // warp-uniform
                            const double mu_i = __ldg(a.mean + i), rs_i = __ldg(a.rs + i);
                            const double c = (double)gg[u] - mu_i * (double)go[u] -
                                             mu_j * (double)og[u] + mu_j * mu_i * (double)oo[u];
                            const double rr = c * rs_j * rs_i;
                            f[u] = rr * rr;
                            if (a.corr_den > 0.0) f[u] -= (1.0 - f[u]) * a.corr_den;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const int64_t i = ib + c0 + u;
                        if (!(i >= lo && i < hi) || i >= a.row1) continue;
                        const double* an = a.annot + (i - a.row0) * a.K + kc;
#pragma unroll
                        for (int b = 0; b < KC; ++b)
                            if (kc + b < a.K) acc[b] += f[u] * __ldg(an + b);
                    }
                    if (diag) continue;
                    // Columns: the warp's 32 rows of four columns at a time through
                    // shared memory; eight lanes per column add four rows each.
                    const int cu_i = lane >> 3, part = lane & 7;
#pragma unroll
                    for (int sub = 0; sub < 16 / kCB; ++sub) {
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < kCB; ++u) cols[u * kCLd + lane] = f[kCB * sub + u];
                        __syncwarp();
                        const int il = c0 + kCB * sub + cu_i;
                        const int64_t i = ib + il;
                        const bool ivalid = i < a.row1;
                        const int64_t lo_i = ivalid ? (int64_t)a.lo[i - a.row0] : 0;
                        const int64_t hi_i = ivalid ? min((int64_t)a.hi[i - a.row0], a.row1) : 0;
                        double ca[KC];
#pragma unroll
                        for (int b = 0; b < KC; ++b) ca[b] = 0.0;
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            const int64_t jj = jrow0 + q * 32 + part * 4 + m;
                            if (!(jj >= lo_i && jj < hi_i)) continue;
                            const double fv = cols[cu_i * kCLd + part * 4 + m];
                            const double* an = a.annot + (jj - a.row0) * a.K + kc;
#pragma unroll
                            for (int b = 0; b < KC; ++b)
                                if (kc + b < a.K) ca[b] += fv * __ldg(an + b);
                        }
                        __syncwarp();
#pragma unroll
                        for (int b = 0; b < KC; ++b)
                            for (int o = 1; o < 8; o <<= 1)
                                ca[b] += __shfl_xor_sync(0xffffffffu, ca[b], o);
                        if (part == 0 && ivalid) {
                            double* out = a.units + (cu * kBM + il) * a.K + kc;
#pragma unroll
                            for (int b = 0; b < KC; ++b)
                                if (kc + b < a.K) out[b] = ca[b];
                        }
                    }
                }
                if (jvalid) {
                    // row unit of this quarter of the columns, summed over the run
                    double* out = a.units + ((int64_t)(item.row_unit + cset) * kBM + jl) * a.K + kc;
#pragma unroll
                    for (int b = 0; b < KC; ++b)
                        if (kc + b < a.K) out[b] = t > 0 ? out[b] + acc[b] : acc[b];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemCols));
    }
}

// out[(j - row0) K + b] += the sum over the units of j's tile, in list order.
__global__ void gram_reduce_kernel(const double* __restrict__ units,
                                   const int32_t* __restrict__ beg, const int32_t* __restrict__ list,
                                   int64_t row0, int64_t row1, int K, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = (row1 - row0) * K;
    if (t >= n) return;
    const int64_t jr = t / K;
    const int b = (int)(t - jr * K);
    const int64_t T = jr / kBM;
    const int jl = (int)(jr - T * kBM);
    double s = 0.0;
    for (int32_t u = beg[T]; u < beg[T + 1]; ++u)
        s += units[((int64_t)list[u] * kBM + jl) * K + b];
    out[t] += s;
}

}  // namespace gram

void launch_gram_ld(const CUtensorMap& tmC, const GramArgs& a, int n_items, cudaStream_t st) {
    if (n_items <= 0) return;
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        for (auto f : {gram::gram_ld_kernel<1>, gram::gram_ld_kernel<4>, gram::gram_ld_kernel<8>})
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)gram::kSmemBytes);
    });
    auto f = a.K == 1 ? gram::gram_ld_kernel<1>
           : a.K <= 4 ? gram::gram_ld_kernel<4> : gram::gram_ld_kernel<8>;
    f<<<(unsigned)n_items, gram::kThreads, gram::kSmemBytes, st>>>(tmC, a);
    count_launch();
}

void launch_gram_reduce(const double* units, const int32_t* beg, const int32_t* list, int64_t row0,
                        int64_t row1, int K, double* out, cudaStream_t st) {
    const int64_t n = (row1 - row0) * K;
    if (n <= 0) return;
    gram::gram_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(units, beg, list, row0,
                                                                          row1, K, out);
    count_launch();
}

}  // namespace lds
