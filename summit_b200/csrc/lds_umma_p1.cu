// Phase 1 on tcgen05 tensor cores: Y[:, (k, v)] = sum_{j in bin k} x_j w_{j,(k,v)}.
//
// UMMA shape per CTA: M = 128 samples, N = the bin's digit columns (4 per
// probe, <= 256 per pass), K = 64 member SNPs per stage.  The A operand is
// the decoded genotype tile in MN-major SWIZZLE_128B layout: a packed SNP row
// already lists samples contiguously, so decoder thread t expands member SNP t
// of the stage into row t of the tile with no transpose.  G and O tiles are
// multiplied by the digits of W1 = s_j sc z and of -W2 = -mu_j W1 (side by side
// in 128-byte rows, SWIZZLE_128B, K-major, laid out contiguous by the weight
// kernel, w_digit_offset, so that one bulk copy brings a K-step's tile) into ONE
// accumulator, so TMEM holds G.W1 - O.W2 = sum_j (g - mu_j o) s_j sc z directly.
//
// Roles (832 threads): warp 0 TMA producer for the digit tiles; warp 1 TMEM
// allocation and MMA issue (one elected thread); warps 2-9, four decoder sets of
// two (set d takes the K-steps it with it % 4 == d), gather the member SNPs' packed
// bytes from global memory (one row each, kept several steps ahead by
// cp.async) and decode them into the operand tiles; warps 10-25, eight per TMEM
// accumulator, read it out and split it into digits.  Two TMEM accumulators let
// the MMAs of the next job (super-bin, column group) run while the epilogue of
// the previous one drains, which matters for windowed estimates, whose super-bins
// are a few K-steps long.
//
// What bounds it: with many K-steps per super-bin the weight tiles' L2 reads
// (26.6 KB per 64 members and sample tile at N = 208, about 10 TB/s over the
// chip); with few, the digit epilogue and the latency from a stage's release to
// its next tiles.  Stages of 64 members and not 128 give four and not two of
// them in 227 KB, and short lists less padding; the issuing warp's loop is
// warp-uniform with one wait per K-step (a single diverged thread with two waits
// took 640 cycles per K-step beside 416 of MMA).  Windowed, N = 50,000,
// M = 60,000, K = 24, B = 50: 8.7 -> 8.2 ms; N = 10,007, K = 6, B = 10: 137 ->
// 115 us; N = 200,003, K = 1, B = 50: 1.19 -> 1.07 ms.
#include <algorithm>
#include <cooperative_groups.h>
#include <cstdint>
#include <cstdio>

#include "lds_internal.h"
#include "lds_p1_drain.h"
#include "lds_tc.cuh"
#include "lds_umma.h"

namespace lds {
namespace umma {

namespace p1 {
constexpr int kMaxStages = 8;
constexpr int kBM = 128;          // samples per CTA
constexpr int kBK = kP1Step;      // member SNPs per stage (64)
constexpr int kATile = kBM * kBK; // 8 KB
constexpr int kDecSets = 4;
constexpr int kSetWarps = kBK / 32;      // a decoder thread per member row
constexpr int kDecWarp0 = 2;
constexpr int kEpiWarp0 = kDecWarp0 + kSetWarps * kDecSets;
constexpr int kEpiWarps = 8;             // per accumulator: two per TMEM lane quadrant
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kThreads = 32 * (kEpiWarp0 + 2 * kEpiWarps);
constexpr int kAccCols = 256;            // one accumulator: <= 256 digit columns
constexpr uint32_t kTmemCols = 512;      // two accumulators (MMA of job j+1 || epilogue of j)
constexpr int kDepth = 3;                // gathered K-steps in flight per decoder set
constexpr int kRing = kDepth * kDecSets; // ring slots
constexpr int kRingSlot = kBK * 32;      // a K-step's member rows x 32 bytes
constexpr int kMaxSb = 256;              // super-bins per CTA (their offsets in shared memory)
constexpr int kShiftBytes = 2 * kEpiWarps * 32 * 16;  // digit shifts of 32 probes per epilogue warp
constexpr int kSmemLimit = 227 * 1024;
// Longest list whose |128 t2 + t3| stays below 2^31: the low digits' products
// are at most 3 * 64 per member.
constexpr int kMaxNarrowSteps = 86000 / kBK;

// Shared memory: the stages (G and O tiles, then the weight-digit tile of
// tile_rows columns), the gather ring, the barriers, the super-bin table, and
// each epilogue warp's digit-shift table.
struct Layout {
    uint32_t stage;
    int stages;
    __host__ __device__ explicit Layout(int tile_rows)
        : stage(2 * kATile + (uint32_t)((tile_rows * 2 * kBK + 1023) / 1024 * 1024)),
          stages(0) {
        const int fit = (int)((kSmemLimit - 1024 - tail()) / stage);
        stages = fit < kMaxStages ? fit : kMaxStages;
    }
    __host__ __device__ static constexpr uint32_t tail() {
        return kRing * kRingSlot + 256 + (kMaxSb + 4) * 4 + kShiftBytes;
    }
    __host__ __device__ uint32_t ring_off() const { return (uint32_t)stages * stage; }
    __host__ __device__ uint32_t bar_off() const { return ring_off() + kRing * kRingSlot; }
    __host__ __device__ uint32_t shift_off() const { return bar_off() + 256; }
    __host__ __device__ uint32_t table_off() const { return shift_off() + kShiftBytes; }
    __host__ __device__ uint32_t bytes() const { return ring_off() + tail(); }
};
static_assert(4 * (2 * kATile + 2 * 256 * kBK) + Layout::tail() + 1024 <= kSmemLimit,
              "four stages of 256 digit columns fit");
constexpr int kDecWarps = kSetWarps * kDecSets;
static_assert((2 * kMaxStages + 5) * 8 + 8 + kDecWarps * 4 <= 256,
              "the barriers, the abort flag and the decoders' positions fit");

// (out of line: it is for the error path only)
__device__ __noinline__ void settle(uint64_t* full, const volatile int* dec_next, int issued,
                                    int nst) {
    for (int w = 0; w < kDecWarps; ++w)
        for (long long i = 0; dec_next[w] < 0 && i < wait_limit(); ++i) {
        }
    __threadfence_block();
    p1_settle(issued, nst, kDecSets, kSetWarps,
              [&](int w) { return dec_next[w] < 0 ? INT_MAX : dec_next[w]; },
              [&](int st) { mbar_arrive(&full[st]); });
}
}  // namespace p1

__global__ void __launch_bounds__(p1::kThreads, 1)
    p1_umma_kernel(P1UArgs a) {
    using namespace p1;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);  // (a plain offset keeps shared-space accesses)
    const Layout lay(p1_tile_rows(a));
    const int nst = lay.stages;
    uint8_t* ring = smem + lay.ring_off();
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + lay.bar_off());
    uint64_t* full = bars;                      // [nst] genotype tiles decoded, weight tile landed
    uint64_t* empty = bars + kMaxStages;        // [nst] stage consumed by the MMAs
    uint64_t* acc_full = bars + 2 * kMaxStages; // [2] accumulator b holds a finished job
    uint64_t* acc_empty = acc_full + 2;         // [2] accumulator b read out
    uint64_t* mma_done = acc_empty + 2;         // drain of the issuer's MMAs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* dec_next = abort_flag + 1;    // [kDecWarps] first step not arrived for, once left
    int4* shift_tab = reinterpret_cast<int4*>(smem + lay.shift_off());
    int* ktab = reinterpret_cast<int*>(smem + lay.table_off());

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int64_t i0 = (int64_t)blockIdx.x * kBM;
    // This CTA's super-bins: kb0 .. kb0 + nsb; a job is one (super-bin, column
    // group), or with share > 1 that many super-bins with one member list, their
    // digit columns side by side, so that a decoded tile serves them all.  ktab holds their list offsets in K-steps.  With nsplit > 1 the CTA
    // takes part blockIdx.z of every super-bin's K-steps.
    const int kb0 = blockIdx.y * a.sb_per_cta;
    const int nsb = min(a.K - kb0, a.sb_per_cta);

    for (int q = tid; q <= nsb; q += kThreads) ktab[q] = (int)(a.bin_off[kb0 + q] / kBK);
    if (tid == 0) {
        for (int s = 0; s < nst; ++s) {
            // the step's decoder warps, and the weight producer with its copies' bytes
            mbar_init(&full[s], kSetWarps + 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kEpiWarps);   // one arrival per epilogue warp
        }
        mbar_init(mma_done, 1);
        *abort_flag = 0;
        for (int w = 0; w < kDecWarps; ++w) dec_next[w] = -1;
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
    auto fail = [&](int code) {
        atomicCAS(a.status, 0u, (unsigned)code);
        *abort_flag = 1;
    };
    // K-steps [k0, k0 + n) of super-bin kb0 + q that this CTA takes.
    auto steps_of = [&](int q, int& k0) {
        const int n = ktab[q + 1] - ktab[q];
        if (a.nsplit <= 1) {
            k0 = 0;
            return n;
        }
        const int per = (n + a.nsplit - 1) / a.nsplit;
        k0 = min(n, (int)blockIdx.z * per);
        return min(n, k0 + per) - k0;
    };

    if (warp == 0) {
        // ---------------- TMA producer of weight-digit tiles ----------------
        if (lane == 0) {
            int it = 0, s = 0;
            uint32_t ph = 0;
            for (int q = 0; q < nsb && !*abort_flag; q += a.share) {
                int k0;
                const int nkt = steps_of(q, k0), nbin = min(a.share, nsb - q);
                for (int g = 0; g < a.ngroups && !*abort_flag; ++g) {
                    for (int kt = 0; kt < nkt; ++kt, ++it) {
                        if (it >= nst && !mbar_wait(&empty[s], ph ^ 1u, abort_flag)) { fail(11); break; }
                        uint8_t* w = smem + s * lay.stage + 2 * kATile;
                        // the group's columns, for each bin of the job
                        const uint32_t bytes = (uint32_t)min(256, a.ncolp - g * 256) * 2 * kBK;
                        mbar_expect_tx(&full[s], (uint32_t)nbin * bytes);
                        for (int u = 0; u < nbin; ++u, w += a.ncolp * 2 * kBK)
                            bulk_load(w, a.wq + ((int64_t)(ktab[q + u] + k0 + kt) * a.ncolp + g * 256) *
                                                    2 * kBK,
                                      bytes, &full[s]);
                        if (++s == nst) { s = 0; ph ^= 1u; }
                    }
                }
            }
            // Drain: no tile copy may still be landing when the CTA exits
            // (only reachable with copies outstanding after an abort).
            bool settled = false;
            for (int j = max(0, it - nst); j < it; ++j) {
                const uint32_t par = (uint32_t)(j / nst) & 1u;
                if (mbar_wait(&full[j % nst], par, abort_flag)) continue;
                if (!settled) {
                    settle(full, dec_next, it, nst);
                    settled = true;
                }
                mbar_wait(&full[j % nst], par);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop (so that addresses, phases and
        // descriptors stay in uniform registers); one elected thread issues.
        int s = 0, au = 0;  // stage, jobs (accumulator uses)
        uint32_t ph = 0;
        bool ok = true;
        for (int q = 0; q < nsb && ok; q += a.share) {
            int k0;
            const int nkt = steps_of(q, k0);
            const int width = min(a.share, nsb - q) * a.ncolp;   // the job's digit columns
            if (nkt == 0) continue;
            for (int g = 0; g < a.ngroups && ok; ++g, ++au) {
                const int b = au & 1, u = au >> 1;
                const int ncols = min(kAccCols, width - g * 256);
                const uint32_t idesc = idesc_i8_amn(kBM, ncols);
                const uint32_t acc = tmem + (uint32_t)(b * kAccCols);
                if (u > 0 && !warp_wait(&acc_empty[b], (uint32_t)(u - 1) & 1u, abort_flag)) {
                    fail(12);
                    ok = false;
                    break;
                }
                tc_fence_after();
                for (int kt = 0; kt < nkt; ++kt) {
                    if (!warp_wait(&full[s], ph, abort_flag)) {
                        fail(13);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint8_t* st = smem + s * lay.stage;
                    const uint64_t dG = sw128_desc_mn(st);
                    const uint64_t dO = sw128_desc_mn(st + kATile);
                    const uint64_t dW1 = sw128_desc(st + 2 * kATile);
                    const uint64_t dW2 = dW1 + kBK / 16;
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kBK / 32; ++kk) {
                            // A advances 32 K-rows = 4 swizzle atoms (4 KB); B advances 32 bytes.
                            umma_i8(acc, dG + 256 * kk, dW1 + 2 * kk, idesc, (kt | kk) ? 1u : 0u);
                            umma_i8(acc, dO + 256 * kk, dW2 + 2 * kk, idesc, 1u);
                        }
                        umma_commit(&empty[s]);
                    }
                    __syncwarp();
                    if (++s == nst) { s = 0; ph ^= 1u; }
                }
                if (ok && elect_one()) umma_commit(&acc_full[b]);
                __syncwarp();
            }
        }
        // Drain: every MMA issued here completes before TMEM is released.
        if (elect_one()) umma_commit(mma_done);
        __syncwarp();
        mbar_wait(mma_done, 0u);
    } else if (warp < kEpiWarp0) {
        // ---------------- gather + decode (four sets of two warps) ----------------
        const int dset = (warp - kDecWarp0) / kSetWarps;
        const int t = (tid - 32 * kDecWarp0) % kBK;
        const uint8_t* codes = a.codes + i0 / 4;
        // Gather prefetcher: walks the same (super-bin, group, K-step) sequence
        // ahead of the decode, copying this thread's member row of the set's
        // steps into ring slots.  The member row of the step being fetched is
        // read from rowind one step earlier (row_next), so that load's latency
        // overlaps a step of work instead of stalling the cp.async that needs
        // the address.
        int pq = -a.share, pg = a.ngroups - 1, pkt = 0, pn = 0, pit = 0;
        const int32_t* prow = nullptr;
        bool pend = false;
        auto advance = [&]() {   // cursor to the next K-step, or pend past the last one
            if (pend || pkt < pn) {
                return;
            }
            pkt = 0;
            if (pn > 0 && ++pg < a.ngroups) return;
            pg = 0;
            int k0 = 0;
            do {
                if ((pq += a.share) >= nsb) {
                    pend = true;
                    return;
                }
                pn = steps_of(pq, k0);
            } while (pn == 0);
            prow = a.rowind + ((int64_t)(ktab[pq] + k0) * kBK + t);
        };
        auto cursor_row = [&]() -> int32_t {  // member row of the set's next step, or -1
            advance();
            if (pend) return -1;
            while (pit % kDecSets != dset) {  // the other sets' steps
                ++pkt;
                ++pit;
                advance();
                if (pend) return -1;
            }
            const int32_t row = prow[(int64_t)pkt * kBK];
            ++pkt;
            ++pit;
            return row;
        };
        int pslot = dset;                     // ring slot of the step being fetched
        // (kept as loaded: anything computed from it here would wait for the load)
        int32_t row_next = cursor_row();
        auto prefetch_one = [&]() {
            const int32_t row = row_next;
            row_next = cursor_row();
            // bounds-checked build: a member row outside the image is not gathered
            if (row >= 0 && in_range(a.m_pad == 0 || row < a.m_pad, 0x1001u)) {
                const uint8_t* src = codes + (int64_t)row * a.nbp;
                uint8_t* dst = ring + pslot * kRingSlot + t * 32;
                cp_async16(dst, src);
                cp_async16(dst + 16, src + 16);
            }
            cp_async_commit();
            pslot = pslot + kDecSets < kRing ? pslot + kDecSets : dset;
        };
        for (int d = 0; d < kDepth - 1; ++d) prefetch_one();
        int it = 0, s = 0, slot = 0;
        uint32_t ph = 0;
        for (int q = 0; q < nsb && !__any_sync(0xffffffffu, *abort_flag != 0); q += a.share) {
            int k0;
            const int nkt = steps_of(q, k0) * a.ngroups;
            for (int kt = 0; kt < nkt; ++kt, ++it) {
                if (it % kDecSets == dset) {
                    prefetch_one();
                    asm volatile("cp.async.wait_group %0;\n" ::"n"(kDepth - 1));
                    const uint4* src =
                        reinterpret_cast<const uint4*>(ring + slot * kRingSlot + t * 32);
                    const uint4 c0 = src[0], c1 = src[1];
                    if (it >= nst && !warp_wait(&empty[s], ph ^ 1u, abort_flag)) {
                        fail(14);
                        break;
                    }
                    uint8_t* gRow = smem + s * lay.stage + (t >> 3) * 1024 + (t & 7) * 128;
                    decode_row_sw128(c0, c1, gRow, gRow + kATile, t);
                    fence_async_smem();
                    __syncwarp();  // orders the warp's operand stores before its one arrival
                    if (lane == 0) mbar_arrive(&full[s]);
                }
                if (++s == nst) { s = 0; ph ^= 1u; }
                if (++slot == kRing) slot = 0;
            }
        }
        cp_async_wait_all();  // no gather copy may outlive the CTA (abort path)
        __threadfence_block();
        __syncwarp();
        if (lane == 0) dec_next[warp - kDecWarp0] = it;
    } else {
        // ---------------- epilogue (eight warps per accumulator) ----------------
        // Each half of the warps answers for one accumulator, so that the waits,
        // loads and shuffles of one job overlap the arithmetic of the next.
        const int half = (warp - kEpiWarp0) / kEpiWarps;
        const int e = (tid - 32 * kEpiWarp0) % kEpiThreads;
        const int q = warp & 3;                  // TMEM lane quadrant of this warp
        const int h = ((warp - kEpiWarp0) >> 2) & 1;  // which of every two column chunks
        const int64_t i = i0 + q * 32 + lane;    // sample row of this thread's accumulator lane
        int4* const tab = shift_tab + (warp - kEpiWarp0) * 32;   // this warp's digit shifts
        // Sketch column, counted from the job's first bin, of digit-column group
        // `slot` (4 columns each): -1 past a bin's probes or the job's bins.
        auto probe_of = [&](int slot, int nbin) -> int64_t {
            if (a.share == 1) return slot < a.V ? slot : -1;
            const int per = a.ncolp / 4, u = slot / per, v = slot - u * per;
            return u < nbin && v < a.V ? (int64_t)u * a.V + v : -1;
        };
        int au = 0;
        for (int kq = 0; kq < nsb && !__any_sync(0xffffffffu, *abort_flag != 0); kq += a.share) {
            const int k = kb0 + kq;
            int k0;
            const int nkt = steps_of(kq, k0), nbin = min(a.share, nsb - kq);
            if (nkt == 0 ? (au & 1) != half : a.ngroups == 1 && (au & 1) != half) {
                if (nkt > 0) ++au;
                continue;
            }
            // This sample tile's block of super-bin k in phase 2's digit layout
            // (digit_offset): ncolp rows of 128 bytes.
            int8_t* const yblk =
                a.yq ? a.yq + ((int64_t)blockIdx.x * a.K * a.ncolp + (int64_t)k * a.ncolp) * 128
                     : nullptr;
            if (a.yq && (nkt == 0 || ((au + a.ngroups - 1) & 1) == half)) {
                // Digit padding rows 4V..ncolp of this tile read as zero in phase 2.
                for (int idx = e; idx < (a.ncolp - 4 * a.V) * 8; idx += kEpiThreads)
                    *reinterpret_cast<uint4*>(yblk + (4 * a.V + (idx >> 3)) * 128 + (idx & 7) * 16) =
                        make_uint4(0, 0, 0, 0);
            }
            if (nkt == 0) {
                // Bin without members: its sketch columns are zero (the
                // reference's untouched-bin zeroing, gw_ldscore.py:2017-2019;
                // a split's columns start at zero).
                if (a.yq) {
                    for (int idx = e; idx < 4 * a.V * 8; idx += kEpiThreads)
                        *reinterpret_cast<uint4*>(yblk + (idx >> 3) * 128 + (idx & 7) * 16) =
                            make_uint4(0, 0, 0, 0);
                } else if (a.nsplit <= 1) {
                    for (int idx = e; idx < nbin * a.V * 64; idx += kEpiThreads)
                        *reinterpret_cast<uint4*>(a.Y + ((int64_t)k * a.V + (idx >> 6)) * a.N_pad +
                                                  i0 + (idx & 63) * 2) = make_uint4(0, 0, 0, 0);
                }
                continue;
            }
            // (nkt is this super-bin's whole list: the digit form is never split)
            const bool small_sums = nkt <= kMaxNarrowSteps;
            for (int g = 0; g < a.ngroups && !__any_sync(0xffffffffu, *abort_flag != 0); ++g, ++au) {
                const int b = au & 1, u = au >> 1;
                if (b != half) continue;
                // Loaded before the accumulator wait so the loads overlap the MMAs:
                // the digit shifts of this warp's (at most four) chunks of 8 probes,
                // or the group's 64 per-probe scales, two per lane.
                bool narrow = false;
                double scA = 0.0, scB = 0.0;
                if (a.yq) {
                    const int v = g * 64 + 8 * (h + 2 * (lane >> 3)) + (lane & 7);
                    const int r = v < a.V ? -a.yshift[(int64_t)k * a.V + v] : 0;
                    narrow = small_sums && __all_sync(0xffffffffu, r >= 0 && r <= 14);
                    const NarrowShift sh = narrow_shift(r);
                    tab[lane] = make_int4(sh.r, sh.up, sh.half, sh.odd);
                    __syncwarp();
                } else {
                    const int64_t oa = probe_of(g * 64 + lane, nbin), ob = probe_of(g * 64 + lane + 32, nbin);
                    if (oa >= 0) scA = a.colscale[(int64_t)k * a.V + oa];
                    if (ob >= 0) scB = a.colscale[(int64_t)k * a.V + ob];
                }
                if (!warp_wait(&acc_full[b], (uint32_t)u & 1u, abort_flag)) {
                    fail(15);
                    break;
                }
                tc_fence_after();
                const int ncols = min(kAccCols, nbin * a.ncolp - g * 256);
                const uint32_t tbase = tmem + (uint32_t)(b * kAccCols) + ((uint32_t)(q * 32) << 16);
                if (a.yq) {
                    // Digits straight into phase 2's operand layout, 8 probes (32
                    // digit columns) per TMEM load; the quadrant's two warps take
                    // every second chunk.  With y = T 2^(eW-28) and the column
                    // exponent eY fixed in advance by a bound on |y|, the sketch's
                    // 28-bit value is R = rint(T 2^-r), r = eY - eW (round half to
                    // even), and digits_word splits it.  A 4 x 4 byte transpose
                    // within each lane quad turns the lanes' digit words (4 digits
                    // of one sample) into words of one digit for 4 consecutive
                    // samples, stored straight to global memory (a warp writes 4
                    // digit rows x 32 samples per probe).  Lane 4a + t stores digit
                    // row 4v + t, samples s = 32 q + 4a of the block: 16-byte chunk
                    // s / 16 = 2q + a / 4, swizzled with the row's low three bits,
                    // (4 v + t) & 7 = 4 (v & 1) + t.
                    //
                    // R in 32 bits (`narrow`) where 0 <= r <= 14 and the low digits' part
                    // stays below 2^31 (up to kMaxNarrowSteps K-steps): narrow_round.
                    const int qd = lane & 3;
                    // word byte b holds digit 3 - b: lane t of a quad keeps byte 3 - t
                    const uint32_t selA = qd < 2 ? 0x7632u : 0x1054u;
                    const uint32_t selB = (qd & 1) ? 0x2604u : 0x7351u;
                    const int chunk = 2 * q + (lane >> 4);
                    int8_t* const ylane = yblk + qd * 128 + 4 * ((lane >> 2) & 3);
                    int8_t* const ydst[2] = {ylane + ((chunk ^ qd) << 4),
                                             ylane + ((chunk ^ (4 + qd)) << 4)};
                    for (int c0 = 32 * h, cc = 0; c0 < ncols; c0 += 64, cc += 8) {
                        int rr[32];
                        tmem_ld32(tbase + (uint32_t)c0, rr);
                        tmem_wait_ld(rr);
                        const int v0 = g * 64 + (c0 >> 2);          // first probe of the chunk (even)
                        const int nv = a.V - v0;                    // probes left (warp-uniform)
                        // All roundings before the first store: a store in between
                        // would order the next probe's shift-table read behind it
                        // (they could alias) and with it the probes one by one
                        // (about 2,400 cycles per chunk).
                        int R[8];
                        if (narrow) {
#pragma unroll
                            for (int p = 0; p < 8; ++p) {
                                const int4 sh = tab[cc + p];
                                R[p] = narrow_round(rr[4 * p], rr[4 * p + 1], rr[4 * p + 2],
                                                    rr[4 * p + 3],
                                                    NarrowShift{sh.x, sh.y, sh.z, sh.w});
                            }
                        } else {
#pragma unroll
                            for (int p = 0; p < 8; ++p) {
                                const int r = tab[cc + p].x;
                                const long long T =
                                    (((long long)rr[4 * p] * 128 + rr[4 * p + 1]) * 128 +
                                     rr[4 * p + 2]) * 128 + rr[4 * p + 3];
                                if (r <= 0) R[p] = (int)(T << -r);
                                else R[p] = (int)((T + ((1LL << (r - 1)) - 1) + ((T >> r) & 1)) >> r);
                            }
                        }
                        uint32_t w[8];
#pragma unroll
                        for (int p = 0; p < 8; ++p) w[p] = digits_word(R[p]);
#pragma unroll
                        for (int p = 0; p < 8; ++p)
                            w[p] = __byte_perm(w[p], __shfl_xor_sync(0xffffffffu, w[p], 2), selA);
#pragma unroll
                        for (int p = 0; p < 8; ++p)
                            w[p] = __byte_perm(w[p], __shfl_xor_sync(0xffffffffu, w[p], 1), selB);
#pragma unroll
                        for (int p = 0; p < 8; ++p)
                            if (p < nv)
                                *reinterpret_cast<uint32_t*>(ydst[p & 1] + (int64_t)(v0 + p) * 512) =
                                    w[p];
                    }
                } else {
                for (int c0c = 16 * h; c0c < ncols; c0c += 32) {
                    int rr[16];
                    tmem_ld16(tbase + (uint32_t)c0c, rr);
                    tmem_wait_ld(rr);
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const int vl = c0c / 4 + p;  // probe within the group (warp-uniform)
                        const int64_t o = probe_of(g * 64 + vl, nbin);
                        if (o < 0) continue;
                        const long long T =
                            (((long long)rr[4 * p] * 128 + rr[4 * p + 1]) * 128 + rr[4 * p + 2]) *
                                128 + rr[4 * p + 3];
                        const double sc = __shfl_sync(0xffffffffu, vl < 32 ? scA : scB, vl & 31);
                        double* const y = a.Y + ((int64_t)k * a.V + o) * a.N_pad + i;
                        if (a.nsplit > 1) atomicAdd(y, sc * (double)T);
                        else *y = sc * (double)T;
                    }
                }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
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

// Weight digits in the layout of p1_umma_kernel (w_digit_offset): part 0 = W1,
// 1 = -W2, column 4 v + t = digit t of probe v.  The padding columns
// 4V..ncolp are left as they are: their accumulator columns are never read.
//
// Latency-bound gathers (rowind -> sdinv, mean, Z) followed by 8 bytes written
// per (member, probe).  A cluster of CTAs owns a (bin, probe) column: each CTA
// a slice of the members, 4 consecutive members per thread (one 4-byte store
// per digit after a byte transpose), the column's maximum and bound through
// distributed shared memory.  A thread's first four weights stay in registers
// between the two passes, which covers lists of up to 4 threads-widths without
// a second gather.  The value's 28 bits are rounded once and split by
// digits_word.  K = 1, V = 20, 20,000 members: 95 -> 15 us; V = 50, 16,001
// members: 112 -> 25 us (one 256-thread CTA per column, byte stores, FP64
// digit splitting).
// Short lists (windowed super-bins) take a warp per column instead, 8 columns
// per CTA, so that an SM has 24 and not 5 of their gather chains in flight
// (966 super-bins x 50 probes of 128 to 640 members: 326 -> 123 us).
constexpr int kWMaxThreads = 512;
constexpr int kWShort = 1024;     // longest list of the warp form
constexpr int kWWarps = 8;        // its columns per CTA

template <bool kWarp>
__global__ void __launch_bounds__(kWarp ? 32 * kWWarps : kWMaxThreads)
    p1_weights4_kernel(P1UWeights w, const double* __restrict__ mean,
                       const double* __restrict__ sdinv, const double* __restrict__ Z,
                       int64_t z_ld) {
    __shared__ double red[2][kWMaxThreads / 32];
    __shared__ double c_red[2];   // slice maximum and bound, read by the cluster
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
    const int nranks = kWarp ? 1 : (int)cl.num_blocks(), rank = kWarp ? 0 : (int)cl.block_rank();
    const int64_t kv = kWarp ? (int64_t)blockIdx.x * kWWarps + warp : (int64_t)(blockIdx.x / nranks);
    if (kWarp && kv >= (int64_t)w.K * w.V) return;
    const int gtid = kWarp ? lane : (int)threadIdx.x;       // thread of this column's group
    const int gsize = kWarp ? 32 : (int)blockDim.x;
    const int k = (int)(kv / w.V), v = (int)(kv - (int64_t)k * w.V);
    const int64_t r0 = w.bin_off[k], nnzp = w.bin_off[k + 1] - r0;
    const int64_t stride = (int64_t)nranks * gsize * 4;
    const int64_t rbeg = ((int64_t)rank * gsize + gtid) * 4;
    // Members r .. r + 3 (lists are padded to a multiple of kP1Step): w1 and mu w1.
    auto load4 = [&](int64_t r, double (&a)[4], double (&m)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double sc = w.sc[r0 + r + q];
            a[q] = m[q] = 0.0;
            if (sc != 0.0) {
                const int64_t j = w.rowind[r0 + r + q];
                a[q] = sdinv[j] * (sc * Z[(int64_t)v * z_ld + j]);
                m[q] = mean[j] * a[q];
            }
        }
    };
    double a0[4] = {0, 0, 0, 0}, m0[4] = {0, 0, 0, 0};
    double amax = 0.0, bsum = 0.0;
    for (int64_t r = rbeg; r < nnzp; r += stride) {
        double a[4], m[4];
        load4(r, a, m);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            amax = fmax(amax, fmax(fabs(a[q]), fabs(m[q])));
            bsum += 2.0 * fabs(a[q]) + fabs(m[q]);
            if (r == rbeg) {
                a0[q] = a[q];
                m0[q] = m[q];
            }
        }
    }
    for (int o = 16; o; o >>= 1) {
        amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
    }
    if (!kWarp) {
        if (lane == 0) {
            red[0][warp] = amax;
            red[1][warp] = bsum;
        }
        __syncthreads();
        if (warp == 0) {
            double x = lane < nwarps ? red[0][lane] : 0.0, y = lane < nwarps ? red[1][lane] : 0.0;
            for (int o = 16; o; o >>= 1) {
                x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
                y += __shfl_xor_sync(0xffffffffu, y, o);
            }
            if (lane == 0) {
                c_red[0] = x;
                c_red[1] = y;
            }
        }
        if (nranks == 1) {
            __syncthreads();
            amax = c_red[0];
            bsum = c_red[1];
        } else {
            cl.sync();
            amax = bsum = 0.0;
            for (int q = 0; q < nranks; ++q) {
                amax = fmax(amax, *cl.map_shared_rank(&c_red[0], q));
                bsum += *cl.map_shared_rank(&c_red[1], q);
            }
        }
    }
    int e = 0;
    if (amax > 0.0 && isfinite(amax)) {
        e = ilogb(amax) + 1;
        if (ldexp(amax, 7 - e) > 127.0) e += 1;
    }
    // 2^(28 - e) as two factors: it overflows for columns of tiny weights.
    const int e1 = min(28 - e, 1000);
    const double f1 = ldexp(1.0, e1), f2 = ldexp(1.0, 28 - e - e1);
    for (int64_t r = rbeg; r < nnzp; r += stride) {
        double a[4], m[4];
        if (r == rbeg) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                a[q] = a0[q];
                m[q] = m0[q];
            }
        } else {
            load4(r, a, m);
        }
        uint32_t x[4], d[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = digits_word(__double2int_rn(a[q] * f1 * f2));
        transpose4x4(x[0], x[1], x[2], x[3], d[3], d[2], d[1], d[0]);  // byte b: digit 3 - b
        const int64_t step = (r0 + r) / kP1Step;
        const int rs = (int)(r % kP1Step);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            *reinterpret_cast<uint32_t*>(w.wq + w_digit_offset(step, 0, 4 * v + t, rs, w.ncolp)) = d[t];
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] = digits_word(__double2int_rn(-(m[q] * f1 * f2)));
        transpose4x4(x[0], x[1], x[2], x[3], d[3], d[2], d[1], d[0]);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            *reinterpret_cast<uint32_t*>(w.wq + w_digit_offset(step, 1, 4 * v + t, rs, w.ncolp)) = d[t];
    }
    if (rank == 0 && gtid == 0) {
        w.colscale[kv] = ldexp(1.0, e - 7 - 21);
        if (w.ycolscale) {
            // Rigorous bound on |y_i| = |sum_j g_ij w1_j - o_ij w2_j| <= sum_j 2|w1_j| + |w2_j|,
            // fixing the sketch's digit exponent before phase 1 runs.  The weights enter as
            // 4-digit values, each within 2^(e-29) of w1 and of mu*w1: add that slack for
            // every member, then the FP64 rounding of the sum.
            const double tot = (bsum + (double)nnzp * 3.0 * ldexp(1.0, e - 29)) * (1.0 + 1e-9);
            int ey = 0;
            if (tot > 0.0 && isfinite(tot)) {
                ey = ilogb(tot) + 1;
                if (ldexp(tot, 7 - ey) > 127.0) ey += 1;
            }
            w.ycolscale[kv] = ldexp(1.0, ey - 28);
            // digit shift for the phase-1 epilogue: R = rint(T 2^(eW - eY))
            w.yshift[kv] = e - ey;
        }
    }
    if (nranks > 1) cl.sync();   // no CTA leaves while another may still read its shared memory
}

void launch_p1_weights4(const P1UWeights& w, const double* mean, const double* sdinv,
                        const double* Z, int64_t z_ld, cudaStream_t st) {
    const int64_t kv = (int64_t)w.K * w.V;
    if (kv == 0) return;
    if (w.lmax <= kWShort && kv >= 148 * kWWarps) {
        p1_weights4_kernel<true><<<(unsigned)((kv + kWWarps - 1) / kWWarps), 32 * kWWarps, 0, st>>>(
            w, mean, sdinv, Z, z_ld);
        count_launch();
        return;
    }
    // As many threads as the longest list has groups of 4 members, and a
    // cluster where that is more than a CTA's and the columns alone leave SMs
    // without a CTA.
    const int64_t quads = (w.lmax + 3) / 4;
    const int threads =
        (int)std::max<int64_t>(32, std::min<int64_t>(kWMaxThreads, (quads + 31) / 32 * 32));
    int width = 1;
    while (width < 8 && kv * width < 2 * 148 && quads > (int64_t)threads * width) width *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(kv * width));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)width;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, p1_weights4_kernel<false>, w, mean, sdinv, Z, z_ld);
    count_launch();
}

size_t p1_umma_smem_bytes(int tile_rows) { return (size_t)p1::Layout(tile_rows).bytes() + 1024; }

void prepare_p1_umma() {
    cudaFuncSetAttribute(p1_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         p1::kSmemLimit);
}

void launch_p1_umma(const P1UArgs& a, int64_t N_pad, cudaStream_t st) {
    static std::atomic<unsigned long long> attr{0};
    once_per_device(attr, [] { prepare_p1_umma(); });
    P1UArgs b = a;
    b.share = std::max(a.share, 1);   // (whole groups per CTA)
    b.sb_per_cta = std::max(std::min(a.sb_per_cta, p1::kMaxSb) / b.share, 1) * b.share;
    dim3 grid((unsigned)(N_pad / p1::kBM), (unsigned)((a.K + b.sb_per_cta - 1) / b.sb_per_cta));
    // Few sample tiles leave SMs idle while each CTA walks its whole list: as
    // many CTAs as fill the chip once then share a list's K-steps (16 at least
    // each).  Their contributions are integers times the column's power-of-two
    // scale, all below 2^53 in total, so the FP64 additions into the zeroed
    // sketch are exact in any order.  N = 5,000 (40 tiles), K = 1, 20,000
    // members: 118 -> 48 us with 3 CTAs per list.
    const int64_t ctas = (int64_t)grid.x * grid.y, steps = a.lmax / p1::kBK;
    b.nsplit = 1;
    if (!a.yq && ctas > 0 && a.lmax <= ((int64_t)1 << 22))
        b.nsplit = (int)std::max<int64_t>(1, std::min<int64_t>(148 / ctas, steps / 16));
    grid.z = (unsigned)b.nsplit;
    if (b.nsplit > 1)
        cudaMemsetAsync(a.Y, 0, sizeof(double) * (size_t)(a.K * a.V) * (size_t)N_pad, st);
    p1_umma_kernel<<<grid, p1::kThreads, p1_umma_smem_bytes(p1_tile_rows(b)), st>>>(b);
    count_launch();
}

}  // namespace umma
}  // namespace lds
