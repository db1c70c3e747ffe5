// Phase 2 on 5th-generation tensor cores (tcgen05, sm_100a).
//
// Work[j, c] = x_j^T Y[:, c] for a tile of 128 SNPs and the CTA's annotation
// bins, with the LD-score epilogue, as in p2_kernel (lds_kernels.cu) but with:
//   * a TMA tile copy (cp.async.bulk.tensor into the CTA's own shared memory)
//     bringing the packed 2-bit genotype tile (128 SNPs x 128 samples = 4 KB),
//     and one bulk copy (cp.async.bulk) of the sketch digit tile (up to 256
//     columns x 128 samples), stored contiguous and pre-swizzled
//     (digit_offset), into shared-memory rings;
//   * two sets of 4 decoder warps expanding packed codes into the G (value)
//     and O (observed) int8 operand tiles in the canonical K-major
//     SWIZZLE_128B layout the UMMA descriptors expect;
//   * a warp issuing tcgen05.mma.kind::i8 (M=128, N<=256, K=32) from one elected
//     thread into two TMEM accumulators (G at column 0, O at column 256; on tiles
//     without a missing call, the column groups' G products in turn);
//   * the first decoder set reading the accumulators back with tcgen05.ld for
//     the exact digit recombination and the squared-sum epilogue.
// The CTA's bins' columns are walked in MMA groups of up to 256, a bin
// possibly straddling two groups: the issuing warp's time per K-step is nearly
// the same at N = 64 and N = 256, so full groups do the most work for it.
//
// What bounds it: the int8 tensor pipe (1,076 cycles per K-step of 256 columns,
// 1,024 of them MMA, at the power-capped clock).  Before the issuing loop was
// made warp-uniform with one wait and one commit per K-step it took 1,316, and a
// group's epilogue 38,000 cycles (now 12,000; the reads of its probe table were
// chained behind the outputs).  N = 50,000, M = 40,000, K = 24, B = 50: 12.6 ->
// 11.1 ms; windowed, M = 60,000: 19.8 -> 17.5 ms; N = 200,003, K = 1: 1.04 -> 0.84
// ms; N = 10,007, HWE, K = 6, B = 10: 180 -> 141 us; N = 5,000, M = 20,000,
// B = 20: 72 -> 53 us.
// Digits of each probe column sit next to each other (column = 4 v + t), so
// one 32-column TMEM load holds 8 probes x 4 digits.
//
// Every wait on an mbarrier is bounded; on timeout the kernel records an
// error code in `status`, stops issuing work and releases its TMEM.
#include <cfloat>
#include <cooperative_groups.h>
#include <cstdint>
#include <cstdio>
#include <cuda.h>
#include <cuda_runtime.h>

#include "lds_device.cuh"
#include "lds_internal.h"
#include "lds_tc.cuh"
#include "lds_umma.h"

namespace lds {
namespace umma {

constexpr int kBM = 128;              // SNP rows per CTA (UMMA M)
constexpr int kBK = 128;              // samples per stage (bytes per operand row)
constexpr int kPkBytes = kBM * 32;    // packed tile: 128 rows x 32 bytes
constexpr int kATile = kBM * kBK;     // 16 KB
constexpr int kPkStages = 6;          // packed-code ring (HBM latency)
// Operand ring: a stage holds a K-step's decoded G and O tiles and its sketch
// tile.  The issuing warp waits on one barrier per K-step and commits to one:
// the first decoder warp of a step waits for the sketch tile before it arrives.
constexpr int kStages = 3;
// Decoder sets: set d decodes the K-steps it with it % kDecSets == d, so two
// sets keep two operand tiles in flight while the first set also runs the
// epilogue.
constexpr int kDecSets = 2;
constexpr int kThreads = 96 + 128 * kDecSets;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kOCol = 256;       // TMEM column of the O accumulator

// What an epilogue thread needs of one probe column group (4 digit columns).
struct __align__(16) ProbeSlot {
    double scale;          // the sketch column's scale
    long long colsum;      // recombined digit column sums (tiles without a missing call)
    int bin;               // bin offset within the CTA's bins, -1: no output uses the columns
    int v;                 // probe
};

struct Layout {
    uint32_t b_slot;                  // bytes of one sketch tile (box_rows x 128, 1 KB multiple)
    __host__ __device__ explicit Layout(int box_rows)
        : b_slot((uint32_t)(((box_rows * kBK) + 1023) / 1024 * 1024)) {}
    __host__ __device__ uint32_t a_off(int s) const { return (uint32_t)s * (2 * kATile + b_slot); }
    __host__ __device__ uint32_t b_off(int s) const { return a_off(s) + 2 * kATile; }
    __host__ __device__ uint32_t pk_off(int s) const { return a_off(kStages) + s * kPkBytes; }
    __host__ __device__ uint32_t bar_off() const { return pk_off(kPkStages); }
    // 64 probe slots for each of the four epilogue warps
    __host__ __device__ uint32_t slot_off() const { return bar_off() + 256; }
    __host__ __device__ uint32_t bytes() const { return slot_off() + 4 * 64 * sizeof(ProbeSlot); }
};

__global__ void __launch_bounds__(kThreads, 1)
    p2_umma_kernel(const __grid_constant__ CUtensorMap tmA, P2UArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (a plain offset keeps shared-space accesses)
    const Layout lay(a.box_rows);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + lay.bar_off());
    uint64_t* pk_full = bars;                          // [kPkStages]
    uint64_t* pk_empty = pk_full + kPkStages;          // [kPkStages]
    uint64_t* b_full = pk_empty + kPkStages;           // [kStages] sketch tile landed
    uint64_t* full = b_full + kStages;                 // [kStages] operands decoded and landed
    uint64_t* empty = full + kStages;                  // [kStages] operands consumed
    uint64_t* acc_full = empty + kStages;              // [2] accumulator holds a finished group
    uint64_t* acc_empty = acc_full + 2;                // [2] accumulator read out
    uint64_t* mma_done = acc_empty + 2;                // drain of the issuer's MMAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    // This CTA's bins: k0 .. k0 + nbk - 1, sharing each decoded genotype tile;
    // their sketch columns are consecutive (bin-major), one TMA box for all.
    // (tile, bin group) of this CTA: the grid's (x, y), or entry x of the work
    // order when one is given.
    const int2 wk = a.work ? a.work[blockIdx.x] : make_int2((int)blockIdx.x, (int)blockIdx.y);
    const int k0 = wk.y * a.bins_per_cta;
    const int nbk = min(a.bins_per_cta, a.K - k0);
    const int cols = a.bins_per_cta * a.ncolp;
    int64_t jt0, jend;
    int sb = 0;  // super-bin base of this tile's window
    if (a.tiles) {
        const int4 t = a.tiles[wk.x];
        jt0 = t.x;
        jend = t.y;
        sb = t.z;
    } else {
        jt0 = a.j0 + (int64_t)wk.x * kBM;
        jend = a.j1;
    }
    const int kb = sb + k0;  // first super-bin of this CTA
    // Bounds-checked build: this CTA's tile, bins and sketch columns, before
    // any barrier or tensor memory is touched (a failing CTA only returns).
    if (!in_range(!a.tiles || (wk.x >= 0 && (int64_t)wk.x < a.j1), 0x2001u) ||
        !in_range(wk.y >= 0 && k0 < a.K, 0x2002u) ||
        !in_range(jt0 >= 0 && jend <= a.M, 0x2003u) ||
        !in_range(a.yq_cols == 0 || ((int64_t)kb + nbk) * a.ncolp <= a.yq_cols, 0x2004u))
        return;

    if (tid == 0) {
        for (int s = 0; s < kPkStages; ++s) {
            mbar_init(&pk_full[s], 1);
            mbar_init(&pk_empty[s], 4);   // one arrival per decoder warp
        }
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&b_full[s], 1);
            mbar_init(&full[s], 4);       // one arrival per decoder warp
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);  // one arrival per epilogue warp
        }
        mbar_init(mma_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // A tile whose output rows have no missing call needs no O plane: its groups
    // take the two accumulators in turn, so that one is read out while the next
    // group's MMAs fill the other.
    int no_missing = (a.snp_missing && a.colsum) ? 1 : 0;
    if (no_missing && tid < kBM) {
        const int64_t j = jt0 + tid;
        if (j < jend && j < a.M && a.snp_missing[j]) no_missing = 0;
    }
    const bool complete = __syncthreads_and(no_missing) != 0;

    auto fail = [&](int code) {
        atomicCAS(a.status, 0u, (unsigned)code);
        *abort_flag = 1;
    };

    // Column groups of this CTA's bins (the last CTA of a tile may hold fewer
    // bins than bins_per_cta).
    const int ngroups = min(a.ngroups, (nbk * a.ncolp + 255) / 256);
    const int total = ngroups * a.nkt;
    if (warp == 0) {
        // ---------------- packed-code producer (runs up to kPkStages ahead) ----------------
        if (lane == 0) {
            int it = 0, s = 0;
            uint32_t ph = 0;
            for (; it < total; ++it) {
                if (it >= kPkStages && !mbar_wait(&pk_empty[s], ph ^ 1u, abort_flag)) { fail(1); break; }
                mbar_expect_tx(&pk_full[s], (uint32_t)kPkBytes);
                tma_load_2d(smem + lay.pk_off(s), &tmA, (it % a.nkt) * 32, (int)jt0, &pk_full[s]);
                if (++s == kPkStages) { s = 0; ph ^= 1u; }
            }
            // Drain: no tile copy may still be landing when the CTA exits (only
            // reachable with copies outstanding after an abort).  Each slot's
            // latest copy is among the last kPkStages issued.
            for (int j = max(0, it - kPkStages); j < it; ++j)
                mbar_wait(&pk_full[j % kPkStages], (uint32_t)(j / kPkStages) & 1u);
        }
    } else if (warp == 2) {
        // ---------------- sketch-digit producer ----------------
        if (lane == 0) {
            int it = 0, s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int g = 0; g < ngroups && ok; ++g) {
                // The group's columns that exist (this CTA's bins); MMA columns
                // past them read stale rows whose results no output uses.
                const int live = min(min(256, cols - g * 256), nbk * a.ncolp - g * 256);
                const uint32_t bytes = (uint32_t)live * (uint32_t)kBK;
                const uint32_t first = (uint32_t)(live / 32) * 16u * (uint32_t)kBK;
                const int8_t* src = a.yq + ((int64_t)kb * a.ncolp + g * 256) * kBK;
                for (int kt = 0; kt < a.nkt; ++kt, ++it, src += a.yq_cols * kBK) {
                    if (it >= kStages && !mbar_wait(&empty[s], ph ^ 1u, abort_flag)) {
                        fail(2);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&b_full[s], bytes);
                    // two copies of whole 16-row pieces (2 KB multiples): phase 2
                    // measured ~2 % faster than with one copy of up to 32 KB
                    if (first) bulk_load(smem + lay.b_off(s), src, first, &b_full[s]);
                    bulk_load(smem + lay.b_off(s) + first, src + first, bytes - first, &b_full[s]);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
            for (int j = max(0, it - kStages); j < it; ++j)
                mbar_wait(&b_full[j % kStages], (uint32_t)(j / kStages) & 1u);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop, so that addresses, phases and descriptors
        // stay in uniform registers, and one elected thread issues: the loop of a
        // single diverged thread took 1,316 cycles per K-step with its operands
        // always ready (MMAs 1,024).
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int g = 0; g < ngroups && ok; ++g) {
            const int b = complete ? g & 1 : 0, u = complete ? g >> 1 : g;
            const int ncols = min(256, cols - g * 256);
            const uint32_t idesc = idesc_i8(kBM, ncols);
            const uint32_t acc = tmem + (uint32_t)b * kOCol;
            if (u > 0 && !warp_wait(&acc_empty[b], (uint32_t)(u - 1) & 1u, abort_flag)) {
                fail(3);
                break;
            }
            tc_fence_after();
            for (int kt = 0; kt < a.nkt; ++kt) {
                if (!warp_wait(&full[s], ph, abort_flag)) {
                    fail(4);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t dG = sw128_desc(smem + lay.a_off(s));
                const uint64_t dO = dG + (kATile >> 4);
                const uint64_t dB = sw128_desc(smem + lay.b_off(s));
                if (elect_one()) {
                    if (complete) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 32; ++kk)
                            umma_i8(acc, dG + 2 * kk, dB + 2 * kk, idesc, (kt | kk) ? 1u : 0u);
                    } else {
#pragma unroll
                        for (int kk = 0; kk < kBK / 32; ++kk) {
                            const uint32_t go = (kt | kk) ? 1u : 0u;
                            umma_i8(tmem, dG + 2 * kk, dB + 2 * kk, idesc, go);
                            umma_i8(tmem + kOCol, dO + 2 * kk, dB + 2 * kk, idesc, go);
                        }
                    }
                    umma_commit(&empty[s]);
                }
                __syncwarp();
                if (++s == kStages) { s = 0; ph ^= 1u; }
            }
            if (ok && elect_one()) umma_commit(&acc_full[b]);
            __syncwarp();
        }
        // Drain: every MMA issued here completes before TMEM is released.
        if (elect_one()) umma_commit(mma_done);
        __syncwarp();
        mbar_wait(mma_done, 0u);
    } else {
        // ---------------- decoders (warps 3..) + epilogue (warps 3..6) ----------------
        const int dset = (warp - 3) >> 2;    // decoder set of this warp
        const int r = (tid - 96) & 127;      // operand row this thread decodes
        const int q = warp & 3;              // TMEM lane quadrant this warp may access
        const int row = q * 32 + lane;       // accumulator row (SNP) of this thread
        const int64_t j = jt0 + row;
        const bool stats = (j < a.M) && a.mean && a.sdinv;
        const double mu = stats ? a.mean[j] : 0.0;
        const double sd = stats ? a.sdinv[j] : 0.0;
        double run2 = 0.0, run4 = 0.0, run2b = 0.0;
        unsigned long long chk_g = 0ULL, chk_o = 0ULL;  // product checksums (a.chk)
        int cur = 0;  // bin offset (within this CTA's bins) that run2/run4 belong to
        ProbeSlot* const slots =
            reinterpret_cast<ProbeSlot*>(smem + lay.slot_off()) + ((warp - 3) & 3) * 64;
        // Add the running sums of bin k0 + cur to the outputs, with the
        // reference's guards, and restart them.
        auto flush = [&]() {
            if (!*abort_flag && j < jend && !a.raw_g && cur < nbk) {
                const double ls = a.left_scale[j];
                double upd = (run2 + run2b) * ls;
                const double seg = (double)a.V;
                const bool nonfinite = !isfinite(upd);
                const bool extreme = !nonfinite && isfinite(a.extreme_warn) && seg > 0.0 &&
                                     upd > a.extreme_warn * seg;
                if (a.guard_counts) {
                    if (nonfinite) atomicAdd(&a.guard_counts[0], 1ULL);
                    else if (extreme) atomicAdd(&a.guard_counts[1], 1ULL);
                }
                if (!(nonfinite || (extreme && a.drop_extreme))) {
                    if (upd < 0.0) upd = 0.0;
                    const int64_t o = (j - a.out_row0) * a.K + k0 + cur;
                    if (!in_range(a.accum_elems == 0 || (o >= 0 && o < a.accum_elems), 0x2005u))
                        return;
                    if (a.accum2) {
                        a.accum[o] += run2 * ls;
                        a.accum2[o] += run2b * ls;
                    } else {
                        a.accum[o] += upd;
                    }
                    if (a.mc) a.mc[o] += run4 * ls * ls;
                }
            }
            run2 = run4 = run2b = 0.0;
        };
        int it = 0, sp = 0, s = 0;
        uint32_t php = 0, ph = 0;
        for (int g = 0; g < ngroups; ++g) {
            for (int kt = 0; kt < a.nkt; ++kt, ++it) {
                if (it % kDecSets == dset) {
                    // Warp-uniform waits and one arrival per warp (after __syncwarp,
                    // which orders the warp's shared-memory accesses before it):
                    // 4 arrivals per stage instead of 128.
                    if (!warp_wait(&pk_full[sp], php, abort_flag)) {
                        fail(5);
                        break;
                    }
                    const uint4* pk = reinterpret_cast<const uint4*>(smem + lay.pk_off(sp) + r * 32);
                    const uint4 p0 = pk[0], p1 = pk[1];
                    if (it >= kStages && !warp_wait(&empty[s], ph ^ 1u, abort_flag)) {
                        fail(6);
                        break;
                    }
                    uint8_t* gRow = smem + lay.a_off(s) + (r >> 3) * 1024 + (r & 7) * 128;
                    if (complete) decode_row_sw128_g(p0, p1, gRow, r);
                    else decode_row_sw128(p0, p1, gRow, gRow + kATile, r);
                    // The packed rows go back only now: the decode has used what was
                    // read, so no read of the slot can still be on its way.
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&pk_empty[sp]);
                    fence_async_smem();
                    if (((warp - 3) & 3) == 0 && !warp_wait(&b_full[s], ph, abort_flag)) {
                        fail(8);
                        break;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[s]);
                }
                if (++sp == kPkStages) { sp = 0; php ^= 1u; }
                if (++s == kStages) { s = 0; ph ^= 1u; }
            }
            if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
            if (dset != 0) continue;
            // Epilogue of column group g: this warp's table of the group's 64 probe
            // slots first, while the last MMAs run.
            const int ncols = min(256, cols - g * 256);
            __syncwarp();
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int gc = g * 256 + 4 * (lane + 32 * x);   // column within this CTA's bins
                const int bo = gc / a.ncolp, v = (gc - bo * a.ncolp) >> 2;
                ProbeSlot ps{0.0, 0LL, -1, v};
                if (gc < cols && bo < nbk && v < a.V) {
                    ps.bin = bo;
                    if (a.colscale) ps.scale = a.colscale[(int64_t)(kb + bo) * a.V + v];
                    if (complete) {
                        const int* cs = a.colsum + (int64_t)kb * a.ncolp + gc;
                        ps.colsum = (((long long)cs[0] * 128 + cs[1]) * 128 + cs[2]) * 128 + cs[3];
                    }
                }
                slots[lane + 32 * x] = ps;
            }
            __syncwarp();
            const int b = complete ? g & 1 : 0, u = complete ? g >> 1 : g;
            if (!warp_wait(&acc_full[b], (uint32_t)u & 1u, abort_flag)) {
                fail(7);
                break;
            }
            tc_fence_after();
            const uint32_t tbase = tmem + (uint32_t)b * kOCol + ((uint32_t)(q * 32) << 16);
            for (int c0 = 0; c0 < ncols; c0 += 32) {
                int rg[32], ro[32];
                __syncwarp();
                tmem_ld32(tbase + (uint32_t)c0, rg);
                if (!complete) {
                    tmem_ld32(tbase + kOCol + (uint32_t)c0, ro);
                    tmem_wait_ld(ro);
                }
                tmem_wait_ld(rg);
                // All eight probes' products and scaled values before any sum or
                // output: a bin's flush in between would chain the probes' table
                // reads and FP64 work one after another (38,000 cycles per group).
                const ProbeSlot* const sl = slots + (c0 >> 2);
                long long TG[8], TO[8];
                double wv[8];
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    TG[p] = (((long long)rg[4 * p] * 128 + rg[4 * p + 1]) * 128 + rg[4 * p + 2]) * 128 +
                            rg[4 * p + 3];
                    // without a missing call, O^T y = the digit columns' sums
                    TO[p] = complete ? sl[p].colsum
                                     : (((long long)ro[4 * p] * 128 + ro[4 * p + 1]) * 128 +
                                        ro[4 * p + 2]) * 128 + ro[4 * p + 3];
                    wv[p] = sd * sl[p].scale * ((double)TG[p] - mu * (double)TO[p]);
                }
                if (a.raw_g || a.chk) {
                    // Checksum weights of the chunk's 8 probes: lane p hashes
                    // probe p's, the loop below broadcasts them.
                    unsigned long long hl = 0ULL;
                    if (a.chk)
                        hl = check_weight(k0 + max(sl[lane & 7].bin, 0), a.chk_v0 + sl[lane & 7].v);
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const unsigned long long h = a.chk ? __shfl_sync(0xffffffffu, hl, p) : 0ULL;
                        if (sl[p].bin < 0) continue;
                        chk_g += h * (unsigned long long)TG[p];
                        chk_o += h * (unsigned long long)TO[p];
                        if (a.raw_g && j < jend) {
                            const int64_t o =
                                ((j - a.out_row0) * a.K + k0 + sl[p].bin) * a.V + sl[p].v;
                            a.raw_g[o] = TG[p];
                            a.raw_o[o] = TO[p];
                        }
                    }
                    if (a.raw_g) continue;
                }
                // The sums, in probe order.  One bin without the half split is the
                // common chunk; a bin's end inside the chunk flushes.
                const int b0 = sl[0].bin;
                if (b0 >= 0 && b0 == sl[7].bin && !a.accum2) {
                    if (b0 != cur) {
                        flush();
                        cur = b0;
                    }
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const double w2 = wv[p] * wv[p];
                        run2 += w2;
                        run4 += w2 * w2;
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        const int bo = sl[p].bin;   // (warp-uniform)
                        if (bo < 0) continue;
                        if (bo != cur) {
                            flush();
                            cur = bo;
                        }
                        const double w2 = wv[p] * wv[p];
                        if (a.accum2 && sl[p].v >= a.split_v) run2b += w2;
                        else run2 += w2;
                        run4 += w2 * w2;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
        }
        if (dset == 0) {
            flush();
            if (a.chk && j < jend && !*abort_flag) {
                atomicAdd(&a.chk[2 * j], chk_g);
                atomicAdd(&a.chk[2 * j + 1], chk_o);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemCols));
    }
}

// ---------------------------------------------------------------------------
// Sketch digits in the layout of this kernel: per bin, column 4 v + t holds
// digit t of probe v; ncolp columns per bin (padding columns zero).
//
// Bound by HBM: 8 bytes read and 4 written per sketch value.  A column's scale
// needs its maximum first, so a thread-block cluster owns a column, each CTA a
// slice of its samples: the slice's maximum, the cluster's through distributed
// shared memory, then the digits.  A slice of at most kQCacheBytes stays in
// shared memory between the two passes; the cluster is as wide as that asks
// for (8 at most) and as a grid of few columns needs to fill the chip.  A warp
// takes 128 samples of the column, 4 per lane: 32-byte loads, and after a
// 4 x 4 byte transpose one full 128-byte digit row per digit.  The value's
// 28 bits are rounded once (FP64 -> int32) and split by digits_word.
// N = 200,003, K V = 50: 569 -> 43 us; N = 50,000, K V = 1,200: 434 -> 203 us
// (one CTA per column, two passes over HBM, byte stores).
// ---------------------------------------------------------------------------
constexpr int kQThreads = 512;
constexpr int kQWarps = kQThreads / 32;
constexpr int kQCacheBytes = 104 * 1024;   // two CTAs per SM

template <bool kVec>
__global__ void __launch_bounds__(kQThreads, 2)
    quantize_y4_kernel(const double* __restrict__ Y, int64_t N, int64_t N_pad, int K, int V,
                       int ncolp, int8_t* __restrict__ Yq, double* __restrict__ colscale,
                       int* __restrict__ colsum, int chunks_per_cta, int cached) {
    extern __shared__ __align__(16) double cache[];   // the slice's samples when `cached`
    __shared__ double s_max[kQWarps];
    __shared__ int s_sum[kQWarps][4];
    __shared__ double c_max;        // read by the other CTAs of the cluster
    __shared__ int c_sum[4];
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int nranks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int64_t kv = (int64_t)(blockIdx.x / nranks);
    const int k = (int)(kv / V), v = (int)(kv - (int64_t)k * V);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* y = Y + kv * N_pad;
    const int64_t nch = N_pad >> 7;
    const int64_t ch0 = (int64_t)rank * chunks_per_cta;
    const int64_t ch1 = min(nch, ch0 + chunks_per_cta);
    auto load4 = [&](int64_t i, double (&x)[4]) {
        if (kVec && i + 4 <= N) {
            const double2 a = *reinterpret_cast<const double2*>(y + i);
            const double2 b = *reinterpret_cast<const double2*>(y + i + 2);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = i + q < N ? y[i + q] : 0.0;
        }
    };
    double amax = 0.0;
    int bad = 0;
    for (int64_t ch = ch0 + warp; ch < ch1; ch += kQWarps) {
        double x[4];
        load4(ch * 128 + lane * 4, x);
        if (cached) {
            double2* cw = reinterpret_cast<double2*>(cache + (ch - ch0) * 128);
            cw[lane] = make_double2(x[0], x[1]);
            cw[32 + lane] = make_double2(x[2], x[3]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double av = fabs(x[q]);
            bad |= !(av <= DBL_MAX);  // NaN or infinite
            amax = fmax(amax, av);
        }
    }
    // A non-finite sketch value makes every product with this column
    // non-finite in the reference's GEMM; a NaN column scale does the same
    // here, so the phase-2 guards drop those updates as the reference does.
    // A non-finite value anywhere marks the slice's maximum as infinite.
    for (int o = 16; o; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) s_max[warp] = amax;
    bad = __syncthreads_or(bad);
    if (warp == 0) {
        double x = lane < kQWarps ? s_max[lane] : 0.0;
        for (int o = 16; o; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
        if (lane == 0) c_max = bad ? (double)INFINITY : x;
    }
    cl.sync();
    amax = 0.0;
    for (int r = 0; r < nranks; ++r) amax = fmax(amax, *cl.map_shared_rank(&c_max, r));
    bad = !(amax <= DBL_MAX);
    int e = 0;
    if (amax > 0.0 && !bad) {
        e = ilogb(amax) + 1;
        if (ldexp(amax, 7 - e) > 127.0) e += 1;
    }
    // 2^(28 - e) as two factors: it overflows for columns of tiny values.
    const int e1 = min(28 - e, 1000);
    const double f1 = bad ? 0.0 : ldexp(1.0, e1), f2 = ldexp(1.0, 28 - e - e1);
    const int64_t col0 = (int64_t)k * ncolp + 4 * v, cols = (int64_t)K * ncolp;
    const int npad = v == V - 1 ? ncolp - 4 * V : 0;   // zero columns after the last probe
    int dsum[4] = {0, 0, 0, 0};
    for (int64_t ch = ch0 + warp; ch < ch1; ch += kQWarps) {
        double x[4];
        if (cached) {
            const double2* cw = reinterpret_cast<const double2*>(cache + (ch - ch0) * 128);
            const double2 a = cw[lane], b = cw[32 + lane];
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        } else {
            load4(ch * 128 + lane * 4, x);
        }
        uint32_t w[4], d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = digits_word(bad ? 0 : __double2int_rn(x[q] * f1 * f2));
        // word byte b holds digit 3 - b
        transpose4x4(w[0], w[1], w[2], w[3], d[3], d[2], d[1], d[0]);
        int8_t* blk = Yq + (ch * cols + col0) * 128;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int sw = (lane >> 2) ^ (int)((col0 + t) & 7);
            *reinterpret_cast<uint32_t*>(blk + t * 128 + (sw << 4) + (lane & 3) * 4) = d[t];
            dsum[t] = __dp4a((int)d[t], 0x01010101, dsum[t]);
        }
        for (int t = 4; t < 4 + npad; ++t)
            *reinterpret_cast<uint32_t*>(blk + t * 128 + lane * 4) = 0u;
    }
    if (rank == 0 && threadIdx.x == 0)
        colscale[kv] = bad ? (double)NAN : ldexp(1.0, e - 7 - 21);
    if (colsum) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            for (int o = 16; o; o >>= 1) dsum[t] += __shfl_xor_sync(0xffffffffu, dsum[t], o);
            if (lane == 0) s_sum[warp][t] = dsum[t];
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            int tot = 0;
            for (int q = 0; q < kQWarps; ++q) tot += s_sum[q][threadIdx.x];
            c_sum[threadIdx.x] = tot;
        }
    }
    // No CTA leaves while another may still read its shared memory.
    cl.sync();
    if (colsum && rank == 0 && (int)threadIdx.x < 4 + npad) {
        int tot = 0;
        if (threadIdx.x < 4)
            for (int r = 0; r < nranks; ++r) tot += *cl.map_shared_rank(&c_sum[threadIdx.x], r);
        colsum[col0 + threadIdx.x] = tot;
    }
    if (colsum) cl.sync();
}

// colsum[c] = sum of digit column c over its N_pad samples (one CTA per column;
// a column's 128-byte rows, one per sample chunk, in any swizzled order).
__global__ void digit_colsum_kernel(const int8_t* __restrict__ Yq, int64_t cols, int64_t N_pad,
                                    int* __restrict__ colsum) {
    __shared__ int part[32];
    const int8_t* col = Yq + (int64_t)blockIdx.x * 128;
    int s = 0;
    for (int64_t u = threadIdx.x; u < (N_pad >> 7) * 8; u += blockDim.x) {
        const int4 v = *reinterpret_cast<const int4*>(col + (u >> 3) * cols * 128 + (u & 7) * 16);
        const int w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
            s += (int)(int8_t)(w[q]) + (int)(int8_t)(w[q] >> 8) + (int)(int8_t)(w[q] >> 16) +
                 (int)(int8_t)(w[q] >> 24);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += part[w];
        colsum[blockIdx.x] = tot;
    }
}

void launch_quantize_y4(const double* Y, int64_t N, int64_t N_pad, int K, int V, int ncolp,
                        int8_t* Yq, double* colscale, cudaStream_t st, int* colsum) {
    const int64_t kv = (int64_t)K * V, nch = N_pad / 128;
    if (kv <= 0 || nch <= 0) return;
    // Cluster width: slices that fit the cache, and 2 CTAs for each SM as long
    // as a warp still has a 128-sample chunk of its own.
    int width = 1;
    while (width < 8 && ((nch + width - 1) / width * 1024 > kQCacheBytes ||
                         (kv * width < 2 * 148 && nch >= 2 * kQWarps * width)))
        width *= 2;
    const int per = (int)((nch + width - 1) / width);
    const int cached = (int64_t)per * 1024 <= kQCacheBytes;
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] {
        cudaFuncSetAttribute(quantize_y4_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kQCacheBytes);
        cudaFuncSetAttribute(quantize_y4_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kQCacheBytes);
    });
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(kv * width));
    cfg.blockDim = dim3(kQThreads);
    cfg.dynamicSmemBytes = cached ? (size_t)per * 1024 : 0;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)width;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // 16-byte loads need the caller's sketch on a 16-byte boundary (N_pad is a
    // multiple of 128, so every column then is).
    const bool vec = (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
    cudaLaunchKernelEx(&cfg, vec ? quantize_y4_kernel<true> : quantize_y4_kernel<false>, Y, N, N_pad,
                       K, V, ncolp, Yq, colscale, colsum, per, cached);
    count_launch();
}

void launch_digit_colsum(const int8_t* Yq, int64_t ncols, int64_t N_pad, int* colsum,
                         cudaStream_t st) {
    if (ncols <= 0) return;
    digit_colsum_kernel<<<(unsigned)ncols, 256, 0, st>>>(Yq, ncols, N_pad, colsum);
    count_launch();
}

// Self-test of the bounded wait: one thread initializes an mbarrier that
// expects one arrival and waits for its first phase.  Nothing arrives, so the
// wait must give up after the configured number of tries and the kernel
// reports 1 (a completed wait would report 2).  No copy or MMA is in flight,
// so the CTA exits cleanly either way.
__global__ void wait_timeout_probe_kernel(unsigned* status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *status = mbar_wait(&bar, 0u) ? 2u : 1u;
    }
}

}  // namespace umma

void launch_wait_timeout_probe(unsigned* status_dev, cudaStream_t st) {
    umma::wait_timeout_probe_kernel<<<1, 32, 0, st>>>(status_dev);
    count_launch();
}

namespace umma {

size_t p2_umma_smem_bytes(int box_rows) { return (size_t)Layout(box_rows).bytes() + 1024; }

void prepare_p2_umma() {
    cudaFuncSetAttribute(p2_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)p2_umma_smem_bytes(256));
}

void launch_p2_umma(const CUtensorMap& tmA, const P2UArgs& a, cudaStream_t st) {
    const int64_t rows = a.j1 - a.j0;
    if ((!a.tiles && rows <= 0) || a.K <= 0) return;
    const size_t smem = p2_umma_smem_bytes(a.box_rows);
    // The attribute is set for the largest tile (256 sketch rows), which
    // covers every launch; function attributes are per device.
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] { prepare_p2_umma(); });
    // With a tile table, j0 is unused and j1 - j0 carries the number of tiles.
    const int nb = a.bins_per_cta > 0 ? a.bins_per_cta : 1;
    dim3 grid((unsigned)(a.tiles ? rows : (rows + kBM - 1) / kBM), (unsigned)((a.K + nb - 1) / nb));
    if (a.work) grid = dim3((unsigned)a.n_work, 1);
    p2_umma_kernel<<<grid, kThreads, smem, st>>>(tmA, a);
    count_launch();
}

}  // namespace umma
}  // namespace lds
