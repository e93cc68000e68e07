// rounds.cu -- the greedy round loop on the device, plain and batched.
//
// Plain form: one representative per round, as the reference's clustering()
// (cuda-version/func.cu:1001-1066) and clusteringDrop() (func.cu:1068-1097).
// A round is a fixed sequence of kernels that read their sizes from a
// RoundState in device memory, so rounds run back to back (and inside a CUDA
// graph) with no host round trip:
//   k_filter      kernel_preFilter + kernel_makeTable/kernel_filter
//                 (func.cu:712-754, 803-826): one warp per candidate; the
//                 composition bound first, then the candidate's (k-mer, count)
//                 entries streamed with 16-byte loads against the
//                 representative's table staged in shared memory.  Survivors
//                 are queued for alignment by the size of their window.
//   k_seg         kernel_align (func.cu:828-999): bit-parallel LCS on the text
//                 rows a long enough common subsequence can still use
//                 (lcs_seg.cuh); k_align (lcs_sys.cuh) takes the pairs whose
//                 window is wider than that kernel holds.
//   k_compact     updataRemain (func.cu:689-699): drops clustered reads from
//                 the remain list and finds the smallest unclustered index;
//                 its last block advances the round state
//                 (updateRepresentative, func.cu:677-687).
//
// Batched form: every decision is a pure function of (representative,
// candidate), so a pass takes the next R unclustered reads r_1 < ... < r_R as
// tentative representatives, computes accept(i, j) for every tentative i and
// every unclustered j > r_i at once, and then replays the reference's order:
// r_i survives iff no surviving r_h (h < i) accepted it, and each candidate
// joins the first surviving tentative that accepted it.  That is exactly what
// R consecutive reference rounds produce.
//   k_bselect     next R unclustered indices from a forward cursor
//   k_bfilter_tab / k_bfilter_idx / k_bfilter_bits / k_bfilter_hash /
//   k_bfilter_mask (+ k_bexact_t, k_bexact_d)
//                 prefilter + word filter of (tentative group, candidate):
//                 transposed per-tentative tables, an inverted k-mer index,
//                 k-mer count bitmaps, hashed k-mer counts or per-k-mer
//                 tentative masks (the last three with exact sums for the pairs
//                 their bounds leave open);
//                 k_bprefilter in drop mode
//   k_band, k_seg, k_align  as above, accepted pairs listed instead of applied
//                 (k_band: a lane per pair, short reads with narrow bands)
//   k_bclaim      survival of the tentatives in order, then the first
//                 surviving tentative per candidate (keyed atomicMax)
//   k_compact     as above, and writes the winners into cluster[]
// R adapts per pass: it halves after a pass in which representatives absorbed
// many reads (tentatives there mostly repeat each other's work) and doubles
// otherwise (8x after a pass too small to fill the device), up to the
// caller's maximum.  The result does not depend on R.
#include <cuda_runtime.h>

#include "gsdr_device.cuh"
#include "lcs_band.cuh"
#include "lcs_seg.cuh"
#include "lcs_sys.cuh"
#include "tc05.cuh"

namespace gsdr {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// A pass is a chain of short kernels.  Those launched with launch_next may be
// set up while the kernel before them drains (programmatic dependent launch),
// so each begins with chain_wait, which returns when that kernel has finished
// and its writes are visible.  Every path through such a kernel passes it: a
// kernel that ended without it would let the next one run beside the one
// before it.  (One representative per round 147 -> 132 ms a call of 7,097
// rounds; 14 passes of 10k reads 3.04 -> 2.96 ms.  Letting the next kernel's
// blocks in at this kernel's start instead of its end took 10% longer on a
// burst of served jobs: they wait in places other streams could use.)
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
constexpr int kFilterThreads = 256;
constexpr int kAlignThreads = 256;  // 8 warps: 8/G groups of G warps
constexpr int kAbsorbHigh = 64;     // absorbed reads per representative that shrink R
// Remaining reads from which a pass of the hashed filter takes only full groups
// of tentatives (hash_even_r): the passes of 1M reads of 100-150 bp, t = 0.90,
// 133 -> 123.5 ms with 960 instead of 1,024 tentatives (the filter 117 -> 108,
// 27 more passes).  On 200k reads at t = 0.95, where the filter is a smaller
// part of a pass, 960 throughout took 1% longer.
constexpr int kEvenRemain = 200000;
// Shorter bitmaps of k_bfilter_bits: 1 one level, 2 folded to half, 3 to a quarter.
constexpr int kMaxDepth = 3;
// Open pairs of a pass, one in so many, above which the next passes take longer
// bitmaps than the estimate asks for.
constexpr int kOpenLimit = 128;
constexpr int kFewPairs = 16384;    // queued pairs below which R grows 8x, not 2x
// Widest band window (words) sent to the lane-banded kernel: batched passes,
// plain rounds.  A plain round waits for its slowest pair, and a lane works
// through its pair alone, so the plain form keeps to the segment kernel.
constexpr int kBandMaxW = kBandMaxWords;
constexpr int kPlainBandMaxW = 0;

__device__ __forceinline__ bool prefilter_pass(const int4 a, const int4 b, int cut) {
    const int s = min(a.x, b.x) + min(a.y, b.y) + min(a.z, b.z) + min(a.w, b.w);
    return !(s < cut);
}

// Alignment class of a pattern of `words` 32-base words; the classes hold the
// same word counts in both forms, as warps x words per lane:
//   class            0       1       2        3        4        5        6
//   words          <=32    <=64   <=128    <=256    <=512   <=1024   <=2048
//   plain form      1x1     1x2     2x2      4x2      8x2      8x4      8x8
//   batched form    1x1     1x2     1x4      1x8      2x8      4x8      8x8
// The plain form waits for every round's longest pair, so it spreads a pattern
// over more warps (shorter per-base chain); the batched form has many pairs in
// flight and packs each pattern into as few warps as it can (fewer
// instructions per DP cell, no hand-offs between warps).
__device__ __forceinline__ int align_class(int words) {
    return words <= 32 ? 0 : words <= 64 ? 1 : words <= 128 ? 2 : words <= 256 ? 3
                         : words <= 512 ? 4 : words <= 1024 ? 5
                         : words <= kMaxPatternWords ? 6 : kLongClass;
}

// Queue of a pair whose full window takes `words` words: the segment kernel's
// class, its wide form's, or the systolic length class of the pattern.
__device__ __forceinline__ int full_class(int words, int q, int seg_max_w) {
    if (words <= seg_max_w) return seg_class(words);
    if (seg_max_w == kSegMaxWords && words <= kSegWideWords) return kWideClass;
    return align_class((q + 31) >> 5);
}

// Queue of a pair: a band class (windows of 4 and 8 words) when its band fits
// and its serial work (text bases x window words: a lane works through its
// pair alone, and a longer one would hold up its pass) stays below
// band_serial; else the segment kernel's class of its widest window; else the
// systolic length class of its pattern.  Pairs decided without alignment
// (trivial_decision) go to whichever of the last two the job launches.
__device__ __forceinline__ int pair_class(int T, int q, int c, int band_max_w,
                                          long long band_serial, int seg_max_w) {
    if (T > 0 && c > 0 && q >= c && T >= c) {
        const int bw = band_words(T, q, c);
        if (bw <= band_max_w) {
            const int w = bw <= 4 ? 4 : 8;
            if ((long long)T * w <= band_serial) return kSysClasses + (w == 4 ? 0 : 1);
        }
        const int sw = seg_words(T, q, c, kSegSteps32);
        if (seg_max_w > 0 && seg_narrow(T, q, c, sw, seg_max_w)) return kNarrowClass;
        return full_class(sw, q, seg_max_w);
    } else if (seg_max_w > 0) {
        return seg_class(1);
    }
    return align_class((q + 31) >> 5);
}

__device__ __forceinline__ void queue_align(RoundState* st, Pair* pairs, int seg_cap,
                                            const DevReads& R, int rep, int q, int band_max_w) {
    const int cls =
        pair_class(R.len_gf[rep], R.len_gf[q], R.cut_base[q], band_max_w, R.band_serial,
                   R.group_max_w);
    const int slot = atomicAdd(&st->n_pairs[cls], 1);
    if (slot < seg_cap) pairs[(size_t)cls * seg_cap + slot] = Pair{rep, q};
    else st->pair_overflow = 1;
}

// A pair that passed the composition bound and the word filter: to the
// alignment queues, or with the pigeon filter on (p 1) to its queue first.
// The reference applies the pigeon filter between the two (func.cu:1030-1044);
// all three are pure functions of the pair, so the order does not change
// which pairs reach the alignment.
__device__ __forceinline__ void push_pair(RoundState* st, Pair* pairs, int seg_cap,
                                          const DevReads& R, int rep, int q, int band_max_w) {
    if (R.pig_q) {
        const int slot = atomicAdd(&st->n_pig, 1);
        if (slot < R.pig_cap) R.pig_q[slot] = Pair{rep, q};
        else st->pair_overflow = 1;
        return;
    }
    queue_align(st, pairs, seg_cap, R, rep, q, band_max_w);
}

// Input bytes of the filter stage (filter_bytes), per launch for every
// remaining candidate: its composition, cutoffs and index (28 bytes) and its
// (k-mer, count) list, or its k-mer bitmap in the bitmap form -- in the plain
// form only what the filter reads (no list behind a failed composition
// bound), in the batched forms once per launch.  Re-reads of the same bytes
// by other tentative groups are not counted.
constexpr unsigned long long kCandFixedBytes = 16 + 8 + 4;
__device__ __forceinline__ unsigned long long cand_bytes(const DevReads& R, int q, bool drop) {
    // (k >= 8: 4-byte k-mer ids and 2-byte counts)
    return kCandFixedBytes + (drop ? 0ull : (R.kcnt ? 6ull : 4ull) * (unsigned)R.n_kmer[q]);
}

// Adds a kernel's counts to the round state, once per block.  Every thread of
// the block calls it; the values are per warp, in lane 0.
__device__ __forceinline__ void add_counts(RoundState* st, int lane, unsigned long long n_pf,
                                           unsigned long long n_wf, unsigned long long n_al,
                                           unsigned long long bytes) {
    __shared__ unsigned long long s_cnt[4];
    if (threadIdx.x < 4) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    if (lane == 0) {
        if (n_pf) atomicAdd(&s_cnt[0], n_pf);
        if (n_wf) atomicAdd(&s_cnt[1], n_wf);
        if (n_al) atomicAdd(&s_cnt[2], n_al);
        if (bytes) atomicAdd(&s_cnt[3], bytes);
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_cnt[threadIdx.x])
        atomicAdd(threadIdx.x == 0   ? &st->cnt_prefilter
                  : threadIdx.x == 1 ? &st->cnt_word
                  : threadIdx.x == 2 ? &st->cnt_aligned
                                     : &st->filter_bytes,
                  s_cnt[threadIdx.x]);
}

// ---------------------------------------------------------------- plain form

// tent: null in the plain form.  In the batched form (table filter) this
// kernel takes the passes with a single tentative: that tentative is the
// smallest unclustered read, so every other remaining read is its candidate
// and the pass is a plain round; k_bfilter_tab takes the passes with more.
// LATE (plain rounds): the representative's table may wait (below); the
// batched form's passes with one tentative stream every candidate, and the
// queue of open candidates would cost them registers.
template <int K, bool DROP, bool LATE>
__global__ void __launch_bounds__(kFilterThreads, 6) k_filter(DevReads R, RoundState* st,
                                                           const int32_t* __restrict__ remain,
                                                           Pair* pairs, int seg_cap,
                                                           const int32_t* __restrict__ tent) {
    extern __shared__ __align__(16) uint16_t table[];
    constexpr bool BITS = !DROP && K <= kMaxBitsK;
    constexpr int NBW = BITS ? (1 << (2 * K)) / 32 : 4;
    __shared__ __align__(16) uint32_t rbits[NBW];
    chain_wait();
    if (st->done) return;
    if (tent && st->n_tent != 1) return;
    const int rep = tent ? tent[0] : st->rep;
    const int band_w = tent ? kBandMaxW : kPlainBandMaxW;
    const int n = st->n_remain;
    if (n <= 0) return;
    // a block with no candidate skips its copy of the representative's tables
    if ((long long)blockIdx.x * (kFilterThreads / 32) >= n) return;
    const int lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (kFilterThreads / 32);
    const int idx0 = blockIdx.x * (kFilterThreads / 32) + (threadIdx.x >> 5);
    unsigned n_pf = 0, n_wf = 0, n_al = 0;
    unsigned long long bytes = 0;
    const int4 crep = R.comp[rep];
    // kernel_filter (func.cu:803-826): S = sum over distinct k-mers of
    // min(count in representative, count in candidate) against the candidate's
    // word cutoff, from the candidate's list and the representative's table
    auto make_table = [&]() {
        constexpr int NB = 1 << (2 * K);
        uint32_t* t32 = reinterpret_cast<uint32_t*>(table);
        for (int i = threadIdx.x; i < NB / 2; i += blockDim.x) t32[i] = 0u;
        __syncthreads();
        const uint32_t* e = R.kmer + R.kmer_off[rep];
        const int ne = R.n_kmer[rep];
        for (int i = threadIdx.x; i < ne; i += blockDim.x) {
            const uint32_t v = __ldg(e + i);
            const uint32_t c = v & 0xffffu;
            if (c) table[v >> 16] = (uint16_t)c;  // kernel_makeTable: only order > 0
        }
        __syncthreads();
    };
    auto word_sum = [&](int q) {
        const int ne4 = (R.n_kmer[q] + 3) >> 2;
        const uint4* e4 = reinterpret_cast<const uint4*>(R.kmer + R.kmer_off[q]);
        bytes += 16ull * ne4;
        int sum = 0;
#pragma unroll 4
        for (int i = lane; i < ne4; i += 32) {
            const uint4 v = __ldcs(e4 + i);
            sum += min((uint32_t)table[v.x >> 16], v.x & 0xffffu);
            sum += min((uint32_t)table[v.y >> 16], v.y & 0xffffu);
            sum += min((uint32_t)table[v.z >> 16], v.z & 0xffffu);
            sum += min((uint32_t)table[v.w >> 16], v.w & 0xffffu);
        }
        return warp_sum_i(sum);
    };
    // With a few candidates per warp (the later rounds) the bitmaps decide
    // nearly all of them, so the table waits until some warp of the block
    // needs it; with more it is made at once.
    const bool late = LATE && BITS && n <= 4 * nwarps;
    constexpr int kLate = 4;  // a late block has at most this many candidates per warp
    int open[kLate], n_open = 0;
    if (BITS) {
        for (int i = threadIdx.x; i < NBW; i += blockDim.x) rbits[i] = R.kbits[(size_t)rep * NBW + i];
        if (late) __syncthreads();
    }
    if (!DROP && !late) make_table();
    const int rep_extra = BITS ? R.kextra[rep] : 0;
    // Software pipeline over this warp's candidates: while candidate i is
    // decided, the composition and cutoff of candidate i+1 are already in
    // flight and the index of candidate i+2 too, so part of the chain of
    // dependent loads (remain -> scalars -> list) overlaps the previous
    // candidate's list stream.  (Prefetching the bitmap as well needs 48
    // registers, five CTAs per SM instead of six, and measured slower.)
    int idx = idx0;
    int q_nx = idx < n ? __ldg(remain + idx) : -1;
    int q_af = idx + nwarps < n ? __ldg(remain + idx + nwarps) : -1;
    int4 comp_nx = make_int4(0, 0, 0, 0);
    int cb_nx = 0;
    if (q_nx >= 0) {
        comp_nx = R.comp[q_nx];
        cb_nx = R.cut_base[q_nx];
    }
    for (; idx < n; idx += nwarps) {
        const int q = q_nx;
        const int4 comp_q = comp_nx;
        const int cb_q = cb_nx;
        // issue the next candidate's loads before this one's work
        q_nx = q_af;
        q_af = idx + 2 * nwarps < n ? __ldg(remain + idx + 2 * nwarps) : -1;
        if (q_nx >= 0) {
            comp_nx = R.comp[q_nx];
            cb_nx = R.cut_base[q_nx];
        }
        if (q == rep) continue;
        n_pf++;
        bytes += kCandFixedBytes;  // composition, cutoffs, index
        // kernel_preFilter (func.cu:738-754); lossless, so also used in drop mode.
        if (!prefilter_pass(crep, comp_q, cb_q - R.strict)) continue;
        if (!DROP) {
            n_wf++;
            const int cw = R.cut_word[q];
            bool decided = false, pass = false;
            if (BITS) {
                // D = shared k-mers (non-zero counts) bounds S: D <= S <= D + min(excesses)
                bytes += 4ull * NBW;
                const int q_extra = R.kextra[q];
                const uint4 cb = __ldcs(
                    reinterpret_cast<const uint4*>(R.kbits + (size_t)q * NBW) + lane % (NBW / 4));
                int d = 0;
                if (lane < NBW / 4) {
                    const uint4 rb = reinterpret_cast<const uint4*>(rbits)[lane];
                    d = __popc(cb.x & rb.x) + __popc(cb.y & rb.y) + __popc(cb.z & rb.z) +
                        __popc(cb.w & rb.w);
                }
                d = warp_sum_i(d);
                if (d >= cw) decided = pass = true;
                else if (d + min(q_extra, rep_extra) < cw) decided = true;
            }
            if (!decided) {
                if (LATE && late) {
#pragma unroll
                    for (int u = 0; u < kLate; u++)
                        if (u == n_open) open[u] = q;
                    n_open++;
                    continue;
                }
                pass = !(word_sum(q) < cw);
            }
            if (!pass) continue;
        }
        n_al++;
        if (lane == 0) push_pair(st, pairs, seg_cap, R, rep, q, band_w);
    }
    if (LATE && BITS && late && __syncthreads_or(n_open)) {
        make_table();
#pragma unroll
        for (int u = 0; u < kLate; u++) {
            if (u >= n_open) break;
            const int q = open[u];
            if (word_sum(q) < R.cut_word[q]) continue;
            n_al++;
            if (lane == 0) push_pair(st, pairs, seg_cap, R, rep, q, band_w);
        }
    }
    // one addition per block and counter: the counters share a cache line, and
    // one per warp (7,296 warps) took most of a 10k-candidate launch's 21.9 us
    add_counts(st, lane, n_pf, n_wf, n_al, bytes);
}

// kernel_pigeon (cuda-version/func.cu:756-801) on the queued pairs, one warp
// per pair, lane = 8 of the 256 buckets: within a bucket the two position
// lists (descending) are walked together; a pair of positions at least
// `gap` apart counts and both lists advance, otherwise the larger position
// advances.  gap = raw length of the representative - ceil(raw length of
// the candidate * t), in float as the reference computes it; the pair passes
// when the count reaches the candidate's pigeon cutoff.
template <bool BATCH>
__global__ void __launch_bounds__(256) k_pigeon(DevReads R, RoundState* st, Pair* pairs,
                                                int seg_cap) {
    if (st->done) return;
    if (BATCH && st->n_tent == 0) return;
    const int np = min(st->n_pig, R.pig_cap);
    const int lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    unsigned rejected = 0;
    for (int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < np; k += nwarps) {
        const Pair p = R.pig_q[k];
        const float prod = ceilf(__fmul_rn((float)R.len[p.cand], R.threshold));
        const int gap = (int)__fsub_rn((float)R.len[p.rep], prod);
        const uint16_t* pr = R.pig + (size_t)p.rep * 256;
        const uint16_t* pc = R.pig + (size_t)p.cand * 256;
        const uint16_t* ir = R.pidx + R.off[p.rep];
        const uint16_t* ic = R.pidx + R.off[p.cand];
        int sum = 0;
        for (int t = lane; t < 256; t += 32) {
            int s1 = t > 0 ? pr[t - 1] : 0, s2 = t > 0 ? pc[t - 1] : 0;
            const int e1 = pr[t], e2 = pc[t];
            while (s1 < e1 && s2 < e2) {
                const int one = ir[s1], two = ic[s2];
                if (abs(one - two) >= gap) {
                    s1++;
                    s2++;
                    sum++;
                } else if (one > two) {
                    s1++;
                } else {
                    s2++;
                }
            }
        }
        sum = warp_sum_i(sum);
        if (!(sum < R.cut_pig[p.cand])) {
            if (lane == 0)
                queue_align(st, pairs, seg_cap, R, p.rep, p.cand,
                            BATCH ? kBandMaxW : kPlainBandMaxW);
        } else {
            rejected++;
        }
    }
    if (lane == 0 && rejected) atomicAdd(&st->cnt_pig_reject, (unsigned long long)rejected);
}

// ---- word lengths 8..12, plain form: the reference's global table ----------
//
// kernel_makeTable / kernel_filter / kernel_cleanTable (func.cu:712-736,
// 803-826): the representative's counts go into a 4^k-entry table in global
// memory (set before the filter, cleared after it), and one warp per
// candidate sums min(table[k-mer], count) over the candidate's entries.

__global__ void k_gtab(DevReads R, RoundState* st, int clear) {
    if (st->done) return;
    const int rep = st->rep;
    const uint32_t* e = R.kmer + R.kmer_off[rep];
    const uint16_t* c = R.kcnt + R.kmer_off[rep];
    const int ne = R.n_kmer[rep];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += gridDim.x * blockDim.x) {
        if (clear) R.gtab[e[i]] = 0;
        else if (c[i]) R.gtab[e[i]] = c[i];  // only order > 0
    }
}

__global__ void __launch_bounds__(kFilterThreads) k_filter_g(DevReads R, RoundState* st,
                                                             const int32_t* __restrict__ remain,
                                                             Pair* pairs, int seg_cap) {
    if (st->done) return;
    const int rep = st->rep;
    const int n = st->n_remain;
    if (n <= 0) return;
    const int lane = threadIdx.x & 31;
    const int4 crep = R.comp[rep];
    unsigned n_pf = 0, n_wf = 0, n_al = 0;
    unsigned long long bytes = 0;
    const int nwarps = gridDim.x * (kFilterThreads / 32);
    for (int idx = blockIdx.x * (kFilterThreads / 32) + (threadIdx.x >> 5); idx < n;
         idx += nwarps) {
        const int q = remain[idx];
        if (q == rep) continue;
        n_pf++;
        bytes += kCandFixedBytes;
        if (!prefilter_pass(crep, R.comp[q], R.cut_base[q] - R.strict)) continue;
        n_wf++;
        bytes += 6ull * (unsigned)R.n_kmer[q];  // k-mer ids and counts
        const uint32_t* e = R.kmer + R.kmer_off[q];
        const uint16_t* c = R.kcnt + R.kmer_off[q];
        const int ne = R.n_kmer[q];
        int sum = 0;
        for (int i = lane; i < ne; i += 32)
            sum += min((uint32_t)__ldg(R.gtab + __ldg(e + i)), (uint32_t)__ldg(c + i));
        sum = warp_sum_i(sum);
        if (sum < R.cut_word[q]) continue;
        n_al++;
        if (lane == 0) push_pair(st, pairs, seg_cap, R, rep, q, kPlainBandMaxW);
    }
    add_counts(st, lane, n_pf, n_wf, n_al, bytes);
}

// Decisions that need no alignment; -1 when the LCS must be computed.
__device__ __forceinline__ int trivial_decision(int T, int q, int c) {
    if (T == 0) return 0;  // the reference's kernel_align never decides such a pair
    if (c <= 0) return 1;  // LCS >= 0 >= cutoff
    if (q < c || T < c) return 0;
    return -1;
}

struct AlignArgs {
    const Pair* pairs;
    int seg_cap;
    int32_t* cluster;
    int* work;
    // batched form
    const uint32_t* tidx;
    uint32_t* tt;
    uint32_t* ttrow;
    Pair* acc;
    int acc_cap;
};

// An accepted pair: the plain form absorbs the candidate at once; the batched
// form lists the pair for the greedy-order resolution and records when a
// tentative accepted another tentative.
template <bool BATCH>
__device__ __forceinline__ void on_accept(RoundState* st, const AlignArgs& A, const Pair p,
                                          int pass) {
    if (!BATCH) {
        A.cluster[p.cand] = p.rep;
        return;
    }
    const int slot = atomicAdd(&st->n_acc, 1);
    if (slot < A.acc_cap) A.acc[slot] = p;
    else st->acc_overflow = 1;
    const uint32_t kc = A.tidx[p.cand];
    if ((int)(kc >> 12) == pass) {
        const int h = A.tidx[p.rep] & 0xfff, ci = kc & 0xfff;
        atomicOr(&A.tt[ci * kTTWords + (h >> 5)], 1u << (h & 31));
        atomicOr(&A.ttrow[ci >> 5], 1u << (ci & 31));
    }
}

template <int G, int W, bool BATCH>
__global__ void __launch_bounds__(kAlignThreads, 3) k_align(DevReads R, RoundState* st, AlignArgs A,
                                                         int cls) {
    constexpr int NG = (kAlignThreads / 32) / G;
    __shared__ SysGroupT<G> groups[NG];
    extern __shared__ __align__(16) uint32_t peq_all[];  // sys_peq_words(W) per warp
    if (st->done) return;
    if (BATCH && (st->pair_overflow || st->n_tent == 0)) return;
    const int np = min(st->n_pairs[cls], A.seg_cap);
    if (np <= 0) return;
    const int pass = BATCH ? st->pass : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = warp / G, gw = warp % G;
    SysGroupT<G>& S = groups[g];
    const int bar_id = 1 + g, bar_n = G * 32;
    const Pair* list = A.pairs + (size_t)cls * A.seg_cap;
    if (gw == 0 && lane == 0) {
        for (int b = 0; b < G; b++) {
            S.ready[b] = 0;
            S.consumed[b] = 0;
        }
        S.stop = 0;
        S.result = 0;
        S.error = 0;
    }
    unsigned long long acc = 0, cells = 0, done = 0;
    while (true) {
        if (gw == 0 && lane == 0) S.idx = atomicAdd(A.work + cls, 1);
        group_bar(bar_id, bar_n);
        const int i = *(volatile int*)&S.idx;
        if (i >= np) break;
        const Pair p = list[i];
        const int T = R.len_gf[p.rep], q = R.len_gf[p.cand], c = R.cut_base[p.cand];
        const int trivial = trivial_decision(T, q, c);
        if (trivial < 0) {
            const int words = (q + 31) >> 5;
            const int B = (words + 32 * W - 1) / (32 * W);
            if (gw < B)
                done += (unsigned long long)lcs_sys_pair<W>(
                            S, peq_all + warp * sys_peq_words(W), R.packed + R.pack_off[p.cand],
                            q, R.packed + R.pack_off[p.rep], T, c, B, gw, lane, &st->error) *
                        (32ull * 32 * 32 * W);
        }
        group_bar(bar_id, bar_n);
        if (gw == 0 && lane == 0) {
            const int ok = trivial >= 0 ? trivial : (S.error ? 0 : *(volatile int*)&S.result);
            cells += (unsigned long long)T * (unsigned long long)q;
            if (ok) {
                acc++;
                on_accept<BATCH>(st, A, p, pass);
            }
            for (int b = 0; b < G; b++) {
                S.ready[b] = 0;
                S.consumed[b] = 0;
            }
            S.stop = 0;
            S.result = 0;
            S.error = 0;
        }
        group_bar(bar_id, bar_n);
    }
    if (gw == 0 && lane == 0 && cells) {
        if (!BATCH) atomicAdd(&st->cnt_accepted, acc);
        atomicAdd(&st->cells, cells);
    }
    if (lane == 0 && done) atomicAdd(&st->cells_done, done);
}

// The four single-warp classes of the batched grouping (1x1, 1x2, 1x4, 1x8)
// in one launch: a warp takes pairs from one queue that runs through classes
// 3, 2, 1, 0 in that order, so the longest pairs start first and the short
// ones fill in behind them (one kernel tail per pass instead of four).
__global__ void __launch_bounds__(kAlignThreads, 3) k_align_single(DevReads R, RoundState* st,
                                                                   AlignArgs A, int* work) {
    __shared__ SysGroupT<1> groups[kAlignThreads / 32];  // one single-warp group per warp
    extern __shared__ __align__(16) uint32_t peq_all[];  // sys_peq_words(8) per warp
    if (st->done) return;
    if (st->pair_overflow || st->n_tent == 0) return;
    int cnt[4], total = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        cnt[c] = min(st->n_pairs[3 - c], A.seg_cap);
        total += cnt[c];
    }
    if (total <= 0) return;
    const int pass = st->pass;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    SysGroupT<1>& S = groups[warp];
    unsigned long long cells = 0;
    unsigned done = 0;  // blocks of 32 steps x words per lane this warp ran
    while (true) {
        int i = 0;
        if (lane == 0) i = atomicAdd(work, 1);
        i = __shfl_sync(kFull, i, 0);
        if (i >= total) break;
        int q4 = 0;
        while (i >= cnt[q4]) i -= cnt[q4++];
        const int cls = 3 - q4;
        const Pair p = A.pairs[(size_t)cls * A.seg_cap + i];
        const int T = R.len_gf[p.rep], q = R.len_gf[p.cand], c = R.cut_base[p.cand];
        int ok = trivial_decision(T, q, c);
        if (ok < 0) {
            if (lane == 0) {
                S.ready[0] = 0;
                S.consumed[0] = 0;
                S.stop = 0;
                S.result = 0;
                S.error = 0;
            }
            __syncwarp();
            const uint32_t* pq = R.packed + R.pack_off[p.cand];
            const uint32_t* pt = R.packed + R.pack_off[p.rep];
            uint32_t* peq = peq_all + warp * sys_peq_words(8);
            // words per lane: the fewest that hold the pattern (1024 bases
            // each over the warp), not the class's power of two -- a step
            // costs about three integer ops per word plus three
            const int wl = (q + 1023) >> 10;  // 1..8 in these classes (q <= 8192)
            int blocks = 0;
            switch (wl) {
                case 1: blocks = lcs_sys_pair<1>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 2: blocks = lcs_sys_pair<2>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 3: blocks = lcs_sys_pair<3>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 4: blocks = lcs_sys_pair<4>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 5: blocks = lcs_sys_pair<5>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 6: blocks = lcs_sys_pair<6>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                case 7: blocks = lcs_sys_pair<7>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
                default: blocks = lcs_sys_pair<8>(S, peq, pq, q, pt, T, c, 1, 0, lane, &st->error); break;
            }
            done += (unsigned)blocks * (unsigned)(wl > 8 ? 8 : wl);
            __syncwarp();
            ok = *(volatile int*)&S.error ? 0 : *(volatile int*)&S.result;
        }
        if (lane == 0) {
            cells += (unsigned long long)T * (unsigned long long)q;
            if (ok) on_accept<true>(st, A, p, pass);
        }
    }
    if (lane == 0 && cells) atomicAdd(&st->cells, cells);
    // cells: 32 steps x 32 lanes x words per lane x 32 bits per block
    if (lane == 0 && done) atomicAdd(&st->cells_done, (unsigned long long)done * (32ull * 32 * 32));
}

// Banded alignment (lcs_band.cuh) of the pairs of band class cls, whose band
// fits a window of W words: one pair per lane.  All lanes of a warp run the
// same blocks of 32 text bases, each on its own pair; a lane whose pair is
// decided takes the next one from the class queue at the next block.
//
// A lane's pair takes a few hundred dependent steps per word, so a launch lasts
// 20 us (150 bp) to 50 us (1,000 bp) however few its pairs are; a stage of at
// most R.band_few leaves them to k_seg, whose groups of lanes finish a pair in
// a fraction of that (14 passes of 10k reads of 200-1,000 bp: 70 -> 20 us).
__device__ __forceinline__ int band_pairs(const RoundState* st) {
    int n = 0;
#pragma unroll
    for (int c = 0; c < kBandClasses; c++) n += st->n_pairs[kSysClasses + c];
    return n;
}

template <int W, bool BATCH>
__device__ __forceinline__ void band_class(const DevReads& R, RoundState* st, const AlignArgs& A,
                                           int cls) {
    // text bases per unrolled group
    constexpr int G = 8;
    const int np = min(st->n_pairs[cls], A.seg_cap);
    if (np <= 0) return;
    const int pass = BATCH ? st->pass : 0;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const Pair* list = A.pairs + (size_t)cls * A.seg_cap;
    int* work = A.work + cls;
    BandLane<W> L;
    L.clear();
    Pair p{-1, -1};
    bool busy = false, more = true;
    unsigned long long cells = 0;
    unsigned acc = 0, done = 0;  // done: blocks of 32 text bases this lane ran on a pair
    while (true) {
        // lanes without a pair take the next ones (one atomic per warp)
        unsigned need = __ballot_sync(kFull, !busy);
        while (need && more) {
            int base = 0;
            if (lane == 0) base = atomicAdd(work, __popc(need));
            base = __shfl_sync(kFull, base, 0);
            if (!busy) {
                const int i = base + __popc(need & lt_mask);
                if (i < np) {
                    p = list[i];
                    L.start(R.packed + R.pack_off[p.cand], R.len_gf[p.cand],
                            R.packed + R.pack_off[p.rep], R.len_gf[p.rep],
                            R.cut_base[p.cand]);
                    busy = true;
                }
            }
            if (base + __popc(need) >= np) more = false;
            need = __ballot_sync(kFull, !busy);
        }
        if (!__any_sync(kFull, busy)) break;
        // one block of 32 text bases; an idle lane runs it with no bases
        uint32_t tw0 = 0, tw1 = 0;
        if (busy) {
            if (L.x0 < L.T) tw0 = __ldg(L.pt + (L.x0 >> 4));
            if (L.x0 + 16 < L.T) tw1 = __ldg(L.pt + (L.x0 >> 4) + 1);
        }
#pragma unroll 1
        for (int j0 = 0; j0 < 32; j0 += G) L.template steps<G>(j0 < 16 ? tw0 : tw1, j0);
        if (busy) {
            done++;
            const int d = L.finish_block();
            if (d >= 0) {
                cells += (unsigned long long)L.T * (unsigned long long)L.q;
                if (d) {
                    acc++;
                    on_accept<BATCH>(st, A, p, pass);
                }
                busy = false;
                L.T = 0;
            }
        }
    }
    acc = (unsigned)warp_sum_i((int)acc);
    if (!BATCH && lane == 0 && acc) atomicAdd(&st->cnt_accepted, (unsigned long long)acc);
    if (cells) atomicAdd(&st->cells, cells);
    // cells: 32 bases x the window's W words x 32 bits per block
    if (done) atomicAdd(&st->cells_done, (unsigned long long)done * (32ull * 32 * W));
}

// Both classes in one launch, the longer work first: a warp that finds the
// eight-word queue empty goes on with the four-word one.  As two launches, a pass
// paid for both where it has neither (200k reads of 100-150 bp, 147 passes: 13.8 ->
// 13.5 ms; 14 passes of 10k reads 1.39 -> 1.37 ms).
template <bool BATCH>
__global__ void __launch_bounds__(kAlignThreads) k_band(DevReads R, RoundState* st, AlignArgs A) {
    chain_wait();
    if (st->done) return;
    if (BATCH && (st->pair_overflow || st->n_tent == 0)) return;
    if (band_pairs(st) <= R.band_few) return;  // k_seg's
    band_class<8, BATCH>(R, st, A, kSysClasses + 1);
    band_class<4, BATCH>(R, st, A, kSysClasses + 0);
}

// The pairs of the segment classes (lcs_seg.cuh) in one launch: each warp
// takes pairs from the classes' queues, widest windows (longest work) first.
// G lanes per pair: 8 for windows of up to 128 words (fewest instructions per
// cell: a step costs 3 W + 3 integer ops for W words, and a segment G steps to
// fill and drain), 16 and 32 for the wider ones.  A stage with fewer pairs
// than half the grid's warps is bound by its longest pair instead, and every
// pair gets a whole warp (fewest words per lane, the shortest step).
//
// Bound by the ALU pipe like the systolic kernels it replaces for these pairs;
// it wins by the cells it does not step.  Alignment stage, systolic and
// group-banded kernels before -> this one: 200k reads of 300-10,000 bp at
// t = 0.95 40.6 -> 20.9 ms (3.36e12 -> 1.67e12 cells), 3k reads of 2-30 kbp at
// t = 0.80 420 -> 199 ms, 30k reads of 150-5,000 bp at t = 0.90 60 -> 34 ms
// (most of its passes hold few pairs: latency), 1k such reads at t = 0.95
// 2.66 -> 1.44 ms.  With the narrow runs, the wide form, short step loops and
// 256 steps per segment for G = 16 (they fill and drain half as often): 13.6,
// 116, 5.8 and 0.87 ms; 147 TCUPS stepped on the long reads, of 197 at three
// ALU operations per 32 cells.
//
// MODE kSegWide: the pairs of the wide class, a warp each with up to 24 words
// per lane (half the warps per SM: the masks take 15 KB a warp).  They ran on
// four or eight warps of k_align, whose bits are the whole pattern: 7,400 pairs
// of 3k reads of 2-30 kbp took 53 ms there, 17 here.
// MODE kSegNarrow: the pairs of the narrow class on their strip (8 lanes a pair, or a
// warp), launched first; a pair it does not accept goes to the queue of its
// full window behind it.  It took the place of a greedy walk with one thread
// per pair, whose longest walk (up to 4,096 dependent steps) held up every
// pass and which needed T/q > 3.6 at t = 0.95 where the strip accepts from 2.7
// on: alignment stage 20.9 -> 18.2 ms (200k reads of 300-10,000 bp), 34 -> 16.7
// ms (30k reads of 150-5,000 bp, t = 0.90, 92 passes), 29.6 -> 15.0 ms (100k
// such reads, t = 0.95, 103 passes), 2.9 -> 1.05 ms (10k reads, 14 passes).
constexpr int kSegFull = 0, kSegNarrow = 1, kSegWide = 2;
template <int MODE>
constexpr int kSegModeW = MODE == kSegWide ? kSegWideW : kSegMaxW;

template <bool BATCH, int MODE>
__global__ void __launch_bounds__(kAlignThreads, MODE == kSegWide ? 1 : 2) k_seg(DevReads R,
                                                                                RoundState* st,
                                                                                AlignArgs A) {
    constexpr bool NARROW = MODE == kSegNarrow;
    constexpr int M = kSegModeW<MODE>;
    using L = SegSmem<M>;
    extern __shared__ __align__(16) uint32_t seg_sm[];  // L::kWords per warp
    chain_wait();
    if (st->done) return;
    if (BATCH && (st->pair_overflow || st->n_tent == 0)) return;
    constexpr int c0 = MODE == kSegNarrow ? kNarrowClass
                       : MODE == kSegWide ? kWideClass
                                          : kSysClasses + kBandClasses;
    // plain rounds: the narrow class runs here too, a warp per pair, first (one
    // launch less per round; its pairs go on to their full window in place)
    constexpr bool BOTH = MODE == kSegFull && !BATCH;
    static_assert(kNarrowClass == kSysClasses + kBandClasses + kSegClasses, "the class after");
    constexpr int nc = MODE == kSegFull ? kSegClasses + (BOTH ? 1 : 0) : 1;
    // the lane-banded classes' pairs too when they are few (k_band)
    const int first =
        MODE == kSegFull && BATCH && band_pairs(st) <= R.band_few ? -kBandClasses : 0;
    int total = 0;
    for (int c = first; c < nc; c++) total += min(st->n_pairs[c0 + c], A.seg_cap);
    if (total <= 0) return;
    const bool alone = total <= (int)gridDim.x * (kAlignThreads / 64);
    const int pass = BATCH ? st->pass : 0;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    uint32_t* peq = seg_sm + (threadIdx.x >> 5) * L::kWords;
    for (int i = lane; i < M * 32; i += 32) peq[L::kNoBase + i] = 0u;
    unsigned long long cells = 0, done = 0;
    unsigned acc = 0;
    for (int cls = nc - 1; cls >= first; cls--) {
        const int np = min(st->n_pairs[c0 + cls], A.seg_cap);
        if (np <= 0) continue;
        const bool narrow = NARROW || (BOTH && cls == kSegClasses);
        const int G = MODE == kSegWide || alone || (BOTH && narrow) || cls == 4 ? 32
                      : cls == 3                                                ? 16
                                                                                : 8;
        const int S = G >= 16 && !narrow ? kSegSteps32 : kSegSteps8;
        const int g = lane / G;
        const bool leader = (lane & (G - 1)) == 0;
        uint32_t* vb = peq + L::kPeq + g * (G * M + G * M / 16);
        uint16_t* codes = reinterpret_cast<uint16_t*>(peq + L::kPeq + L::kV);
        __syncwarp();
        for (int i = lane; i < kSegCodes; i += 32) codes[i] = L::kNoBase;
        codes += g * (S + 2 * G);
        const Pair* list = A.pairs + (size_t)(c0 + cls) * A.seg_cap;
        int* work = A.work + c0 + cls;
        SegPair P = {};
        Pair p{-1, -1};
        bool more = true;
        while (true) {
            // idle groups take the next pairs (one atomic per warp)
            unsigned need = __ballot_sync(kFull, leader && !P.busy);
            while (need && more) {
                int base = 0;
                if (lane == 0) base = atomicAdd(work, __popc(need));
                base = __shfl_sync(kFull, base, 0);
                const int mine = base + __popc(need & lt_mask);  // meaningful in idle leaders
                const int i = __shfl_sync(kFull, mine, 0, G);
                if (!P.busy && i < np) {
                    p = list[i];
                    const int T = R.len_gf[p.rep], q = R.len_gf[p.cand], c = R.cut_base[p.cand];
                    const int trivial = trivial_decision(T, q, c);
                    if (trivial < 0) {
                        const int64_t po = R.pack_off[p.rep];
                        P.T = T;
                        P.q = q;
                        P.c = c;
                        P.stride = (int)((R.pack_off[p.rep + 1] - po) >> 1);
                        P.planes = R.bm + 2 * po;
                        P.pq = R.packed + R.pack_off[p.cand];
                        P.slope = narrow ? seg_narrow_slope(T, q, c) : 0.0f;
                        P.busy = true;
                        seg_start(P, S, narrow);
                    } else if (leader) {
                        cells += (unsigned long long)T * (unsigned long long)q;
                        if (trivial) {
                            acc++;
                            on_accept<BATCH>(st, A, p, pass);
                        }
                    }
                }
                if (base + __popc(need) >= np) more = false;
                need = __ballot_sync(kFull, leader && !P.busy);
            }
            if (!__any_sync(kFull, P.busy)) break;
            const int wl =
                __reduce_max_sync(kFull, P.busy ? (P.n_words + G - 1) / G : 1);
            int steps = 0;
            const int d = seg_dispatch<M>(P, wl, peq, vb, codes, G, S, lane, steps);
            if (!P.busy) continue;
            if (leader) done += (unsigned long long)steps * (32 * G * seg_tile(wl));
            if (d < 0) continue;
            if (BOTH && d == 0 && P.narrow &&
                seg_words(P.T, P.q, P.c, kSegSteps32) <= R.group_max_w) {
                seg_start(P, S, false);
                continue;
            }
            if (leader) {
                if (P.narrow && d == 0) {
                    const int to = full_class(seg_words(P.T, P.q, P.c, kSegSteps32), P.q,
                                              R.group_max_w);
                    const int slot = atomicAdd(&st->n_pairs[to], 1);
                    if (slot < A.seg_cap)
                        const_cast<Pair*>(A.pairs)[(size_t)to * A.seg_cap + slot] = p;
                    else
                        st->pair_overflow = 1;
                } else {
                    cells += (unsigned long long)P.T * (unsigned long long)P.q;
                    if (d) {
                        acc++;
                        on_accept<BATCH>(st, A, p, pass);
                    }
                }
            }
            P = SegPair{};
        }
    }
    // (cells: steps x the window's words x 32 bits)
    acc = (unsigned)warp_sum_i((int)acc);
    cells = warp_sum_ull(cells);
    done = warp_sum_ull(done);
    __shared__ unsigned long long s_sum[3];
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
    __syncthreads();
    if (lane == 0) {
        atomicAdd(&s_sum[0], cells);
        atomicAdd(&s_sum[1], done);
        atomicAdd(&s_sum[2], (unsigned long long)acc);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_sum[0]) atomicAdd(&st->cells, s_sum[0]);
        if (s_sum[1]) atomicAdd(&st->cells_done, s_sum[1]);
        if (!BATCH && s_sum[2]) atomicAdd(&st->cnt_accepted, s_sum[2]);
    }
}

// Pairs whose pattern has more rows than one group of 8 warps x 32 lanes x 8
// words holds (class kLongClass): one block per pair runs the pattern in
// chunks of 65,536 rows (lcs_sys_pair's chunk mode), the carry sequence
// between chunks in the block's pair of global buffers; the decision is the
// zero count summed over the chunks against the cutoff (no early exit).
constexpr int kChunkRows = 32 * kMaxPatternWords;

template <bool BATCH>
__global__ void __launch_bounds__(kAlignThreads, 1) k_align_long(DevReads R, RoundState* st,
                                                                 AlignArgs A, uint32_t* carry,
                                                                 int carry_words) {
    __shared__ SysGroup S;
    __shared__ int s_idx;
    extern __shared__ __align__(16) uint32_t peq_all[];  // sys_peq_words(8) per warp
    if (st->done) return;
    if (BATCH && (st->pair_overflow || st->n_tent == 0)) return;
    const int np = min(st->n_pairs[kLongClass], A.seg_cap);
    if (np <= 0 || !carry) return;
    const int pass = BATCH ? st->pass : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t* buf0 = carry + (size_t)blockIdx.x * 2 * carry_words;
    uint32_t* buf1 = buf0 + carry_words;
    unsigned long long acc = 0, cells = 0, done = 0;
    while (true) {
        if (threadIdx.x == 0) s_idx = atomicAdd(A.work + kLongClass, 1);
        __syncthreads();
        const int i = s_idx;
        __syncthreads();
        if (i >= np) break;
        const Pair p = A.pairs[(size_t)kLongClass * A.seg_cap + i];
        const int T = R.len_gf[p.rep], q = R.len_gf[p.cand], c = R.cut_base[p.cand];
        int ok = trivial_decision(T, q, c);
        if (ok < 0) {
            const uint32_t* pq = R.packed + R.pack_off[p.cand];
            const uint32_t* pt = R.packed + R.pack_off[p.rep];
            const int nch = (q + kChunkRows - 1) / kChunkRows;
            int ztot = 0;
            bool err = false;
            for (int k = 0; k < nch && !err; k++) {
                if (threadIdx.x == 0) {
                    for (int b = 0; b < 8; b++) {
                        S.ready[b] = 0;
                        S.consumed[b] = 0;
                    }
                    S.stop = 0;
                    S.result = 0;
                    S.error = 0;
                }
                __syncthreads();
                const int qk = min(kChunkRows, q - k * kChunkRows);
                const int B = (((qk + 31) >> 5) + 32 * 8 - 1) / (32 * 8);
                const uint32_t* cin = k > 0 ? ((k & 1) ? buf0 : buf1) : nullptr;
                uint32_t* cout = k + 1 < nch ? ((k & 1) ? buf1 : buf0) : nullptr;
                if (warp < B)
                    done += (unsigned long long)lcs_sys_pair<8>(
                                S, peq_all + warp * sys_peq_words(8),
                                pq + (size_t)k * (kChunkRows / 16), qk, pt, T, c, B, warp, lane,
                                &st->error, true, cin, cout) *
                            (32ull * 32 * 32 * 8);
                __syncthreads();
                err = *(volatile int*)&S.error != 0;
                ztot += *(volatile int*)&S.result;
                __syncthreads();
            }
            ok = err ? 0 : (ztot >= c ? 1 : 0);
        }
        if (threadIdx.x == 0) {
            cells += (unsigned long long)T * (unsigned long long)q;
            if (ok) {
                acc++;
                on_accept<BATCH>(st, A, p, pass);
            }
        }
    }
    if (threadIdx.x == 0) {
        if (!BATCH && acc) atomicAdd(&st->cnt_accepted, acc);
        if (cells) atomicAdd(&st->cells, cells);
    }
    if (lane == 0 && done) atomicAdd(&st->cells_done, done);
}

__device__ void reset_align_counters(RoundState* st, int* align_work) {
    st->n_pig = 0;
    for (int c = 0; c < kAlignClasses; c++) {
        st->n_pairs[c] = 0;
        align_work[c] = 0;
    }
    align_work[kSingleWorkSlot] = 0;  // k_align_single's shared queue
}

// Next representative (plain form), on the last block's copy of the round
// state (k_compact).
__device__ void advance_plain(RoundState* st, int32_t* cluster) {
    st->rounds++;
    st->passes++;
    if (st->error || st->pair_overflow) {
        st->done = 1;
        return;
    }
    const int n = st->n_next;
    if (n == 0) {
        st->done = 1;
        return;
    }
    // a run stopped after pass_limit rounds (timing runs, checkpoints) leaves
    // the next representative unclustered, so that cluster[] alone is the
    // loop's state: a resumed run takes it as the smallest unclustered read
    if (st->pass_limit > 0 && st->passes >= st->pass_limit) {
        st->done = 1;
        return;
    }
    const int rep = st->next_min;
    cluster[rep] = rep;
    st->rep = rep;
    st->n_remain = n;
    st->n_next = 0;
    st->next_min = 0x7fffffff;
    st->n_pig = 0;
    for (int c = 0; c < kAlignClasses; c++) st->n_pairs[c] = 0;
}

// The batched form's state for the next pass (in the same place).
__device__ void advance_batch(RoundState* st, const int32_t* tent, int seg_cap,
                              int acc_cap, int amb_cap, int drop, int r_even) {
    st->passes++;
    st->pass++;
    if (st->error) {
        st->done = 1;
        return;
    }
    // shorter bitmaps that left too many pairs open (reads that are less
    // random than the filter's estimate assumes): longer ones for some passes,
    // twice as many every time
    if (st->bits_hold > 0) st->bits_hold--;
    if (st->bits_depth > 0 &&
        (long long)kOpenLimit * st->n_amb > (long long)st->n_tent * st->n_remain) {
        st->bits_cap = st->bits_depth - 1;
        st->bits_hold = 1 << min(++st->bits_fails, 16);
    }
    st->bits_depth = 0;
    if (st->pair_overflow || st->acc_overflow) {
        // queues too small for this many tentatives: the pass changed nothing
        // (the compaction copied the remain list unchanged); redo it with fewer
        if (st->R == 1) {
            st->error = 2;
            st->done = 1;
            return;
        }
        st->R = max(1, st->R / 8);
        st->n_next = 0;
        return;
    }
    const int nt = st->n_tent;
    if (nt > 0) st->cursor = tent[nt - 1] + 1;
    const int surv = max(1, st->survivors);
    // a pass that queued fewer pairs than the device keeps in flight ran on
    // the latency of its longest pairs: grow R faster, and also where its
    // representatives absorbed many reads (the tentatives' repeated work is
    // then free; 30k reads of 150-5,000 bp at t = 0.90 spent 18 of 43 passes
    // at R = 1)
    int queued = 0, fullest = 0;
    for (int c = 0; c < kAlignClasses; c++) {
        queued += st->n_pairs[c];
        fullest = max(fullest, st->n_pairs[c]);
    }
    if (queued >= kFewPairs && st->absorbed > kAbsorbHigh * surv) {
        st->R = max(1, st->R / 2);
    } else {
        // (drop mode has no filter pass to share between tentatives: R grows
        // only while the passes are too small to fill the device, since every
        // tentative that an earlier one absorbs wastes its alignments)
        long long r = (long long)st->R * (queued < kFewPairs ? 8 : (drop ? 1 : 2));
        // queue use grows with the tentatives: keep the fullest alignment
        // queue and the accept list under 3/4 of their capacity (an overflow
        // costs a redone pass; without the cap, drop mode, where every
        // candidate pairs with every tentative, alternates between overflow
        // and a small R)
        if (nt > 0 && fullest > 0) r = min(r, (long long)nt * (3ll * seg_cap / 4) / fullest);
        if (nt > 0 && st->n_acc > 0) r = min(r, (long long)nt * (3ll * acc_cap / 4) / st->n_acc);
        // and the bitmap filter's queue of open pairs
        if (nt > 0 && amb_cap > 0 && st->n_amb > 0)
            r = min(r, (long long)nt * (3ll * amb_cap / 4) / st->n_amb);
        const int top = r_even > 0 && st->n_next >= kEvenRemain ? r_even : st->R_max;
        st->R = (int)max(1ll, min((long long)min(top, st->R_max), r));
    }
    const int n = st->n_next;
    st->n_next = 0;
    st->next_min = 0x7fffffff;
    if (n == 0) {
        st->done = 1;
        return;
    }
    st->n_remain = n;
    if (st->pass_limit > 0 && st->passes >= st->pass_limit) st->done = 1;  // timing runs
}

struct CompactArgs {
    int32_t* cluster;
    int* align_work;
    // batched form
    const uint32_t* best;
    const int32_t* tent;
    int seg_cap, acc_cap, amb_cap, drop;
    int r_even;  // hash_even_r(), 0: none
};

constexpr int kCompactPer = 4;

// Drops clustered reads from the remain list.  Batched: a candidate claimed in
// this pass (k_bclaim) joins its tentative here.  The last block to finish
// advances the round state (a launch of its own took about 4 us per round).
template <bool BATCH>
__global__ void __launch_bounds__(256) k_compact(RoundState* st, const int32_t* __restrict__ remain_in,
                                                 int32_t* __restrict__ remain_out, CompactArgs C) {
    __shared__ int s_min, s_applied, s_base, s_warp[8];
    chain_wait();
    if (st->done) return;
    if (threadIdx.x == 0) {
        s_min = 0x7fffffff;
        s_applied = 0;
    }
    __syncthreads();
    const int n = st->n_remain;
    const int lane = threadIdx.x & 31;
    const uint32_t pass = BATCH ? (uint32_t)st->pass : 0u;
    const bool apply = BATCH && st->n_tent > 0 && !st->pair_overflow && !st->acc_overflow;
    int local_min = 0x7fffffff;
    unsigned applied = 0;
    // a block takes kCompactPer x 256 entries at a time and reserves its output
    // with one addition (one per warp and 32 entries, on one address, took
    // most of the 23 us of a 900k-entry list)
    constexpr int T = kCompactPer * 256;
    for (int base = blockIdx.x * T; base < n; base += gridDim.x * T) {
        int j[kCompactPer];
        unsigned m[kCompactPer];
        int mine = 0;  // kept entries of this warp
#pragma unroll
        for (int u = 0; u < kCompactPer; u++) {
            const int idx = base + 256 * u + (int)threadIdx.x;
            bool keep = false;
            if (idx < n) {
                j[u] = remain_in[idx];
                keep = C.cluster[j[u]] == -1;
                if (apply && keep) {
                    const uint32_t key = C.best[j[u]];
                    if ((key >> 12) == pass) {
                        C.cluster[j[u]] = C.tent[4095u - (key & 0xfffu)];
                        applied++;
                        keep = false;
                    }
                }
            }
            m[u] = __ballot_sync(kFull, keep);
            mine += __popc(m[u]);
        }
        if (lane == 0) s_warp[threadIdx.x >> 5] = mine;
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                const int c = s_warp[w];
                s_warp[w] = tot;
                tot += c;
            }
            s_base = tot ? atomicAdd(&st->n_next, tot) : 0;
        }
        __syncthreads();
        int pos = s_base + s_warp[threadIdx.x >> 5];
#pragma unroll
        for (int u = 0; u < kCompactPer; u++) {
            if ((m[u] >> lane) & 1u) {
                remain_out[pos + __popc(m[u] & ((1u << lane) - 1u))] = j[u];
                local_min = min(local_min, j[u]);
            }
            pos += __popc(m[u]);
        }
        __syncthreads();
    }
    if (!BATCH) {
        local_min = __reduce_min_sync(kFull, local_min);
        if (lane == 0 && local_min != 0x7fffffff) atomicMin(&s_min, local_min);
    } else {
        applied = __reduce_add_sync(kFull, applied);
        if (lane == 0 && applied) atomicAdd(&s_applied, (int)applied);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!BATCH && s_min != 0x7fffffff) atomicMin(&st->next_min, s_min);
        if (BATCH && s_applied) {
            atomicAdd(&st->absorbed, s_applied);
            atomicAdd(&st->cnt_accepted, (unsigned long long)s_applied);
        }
        __threadfence();
        s_base = atomicAdd(&st->ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_base || threadIdx.x >= 32) return;
    // the last block's first warp: the state comes over in one go, past L1
    // (read field by field, 17 queue sizes among them, it took 6 us)
    __shared__ RoundState s_st;
    constexpr int W = sizeof(RoundState) / 4;
    static_assert(sizeof(RoundState) % 4 == 0, "whole words");
    __threadfence();
    int* words = reinterpret_cast<int*>(&s_st);
    for (int i = lane; i < W; i += 32) words[i] = __ldcg(reinterpret_cast<const int*>(st) + i);
    if (!BATCH && lane <= kSingleWorkSlot) C.align_work[lane] = 0;
    __syncwarp();
    if (lane == 0) {
        s_st.ticket = 0;
        if (BATCH)
            advance_batch(&s_st, C.tent, C.seg_cap, C.acc_cap, C.amb_cap, C.drop, C.r_even);
        else
            advance_plain(&s_st, C.cluster);
    }
    __syncwarp();
    for (int i = lane; i < W; i += 32) reinterpret_cast<int*>(st)[i] = words[i];
}

// ---------------------------------------------------------------- batched form

// Next R unclustered indices at or after the cursor, in increasing order.
__global__ void __launch_bounds__(1024) k_bselect(RoundState* st, const int32_t* __restrict__ cluster,
                                                  int n, int32_t* tent, uint32_t* tidx,
                                                  uint32_t* tt, uint32_t* ttrow,
                                                  int* align_work) {
    __shared__ int warp_cnt[4 * 32];
    __shared__ int s_nt;
    chain_wait();
    if (st->done) return;
    const int Rq = st->R;
    const int pass = st->pass;
    int pos = st->cursor;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_nt = 0;
    __syncthreads();
    // 4,096 reads per step (four per thread): once most reads are clustered the
    // unclustered ones are far apart
    while (pos < n) {
        const int nt = s_nt;
        if (nt >= Rq) break;
        unsigned m[4];
        bool un[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int idx = pos + 1024 * k + threadIdx.x;
            un[k] = idx < n && cluster[idx] == -1;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            m[k] = __ballot_sync(kFull, un[k]);
            if (lane == 0) warp_cnt[32 * k + warp] = __popc(m[k]);
        }
        __syncthreads();
        if (warp == 0) {
            // exclusive prefix over the 128 (quarter, warp) counts
            int run = nt;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int c = warp_cnt[32 * k + lane];
                int incl = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int o = __shfl_up_sync(kFull, incl, d);
                    if (lane >= d) incl += o;
                }
                warp_cnt[32 * k + lane] = run + incl - c;
                run += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0) s_nt = min(Rq, run);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int idx = pos + 1024 * k + threadIdx.x;
            const int rank = warp_cnt[32 * k + warp] + __popc(m[k] & ((1u << lane) - 1u));
            if (un[k] && rank < Rq) {
                tent[rank] = idx;
                tidx[idx] = ((uint32_t)pass << 12) | (uint32_t)rank;
            }
        }
        pos += 4 * blockDim.x;
        __syncthreads();
    }
    const int nt = s_nt;
    for (int i = threadIdx.x; i < nt * kTTWords; i += blockDim.x) tt[i] = 0u;
    if (threadIdx.x < kTTWords) ttrow[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        st->n_tent = nt;
        st->n_acc = 0;
        st->n_amb = 0;
        st->acc_overflow = 0;
        st->pair_overflow = 0;
        st->survivors = 0;
        st->absorbed = 0;
        reset_align_counters(st, align_work);
        if (nt == 0) st->done = 1;
    }
}

// Per-tentative tables, transposed (k_bfilter_tab): for each k-mer the counts
// of a group's RG tentatives lie side by side (RG u16 = RG/8 16-byte words),
// so one candidate entry (k-mer, count c) costs RG/8 vector loads and, per
// pair of tentatives, one paired 16-bit min against (c, c) and one paired
// 16-bit add into the lane's sums.  A sum is at most the candidate's k-mer
// count (< 65536), so the halves never carry into each other, and a warp-wide
// 32-bit reduction adds both halves at once.
template <int K>
struct TabGroup {
    static constexpr int RG = K <= 5 ? 32 : K == 6 ? 16 : 4;
    static constexpr int NB = 1 << (2 * K);
    // u16 per k-mer row: the group's RG counts, padded by 16 bytes where a
    // row is read with 16-byte loads.  A warp reads random rows; with a
    // 32-byte (64-byte) stride the first 16 bytes of a row fall in only 4 (2)
    // of the 8 16-byte bank groups of a 128-byte line, with 48 (80) bytes in
    // all 8, which cuts the bank conflicts of a quarter-warp's loads.
    static constexpr int ROW = RG >= 8 ? RG + 8 : RG;
    static constexpr int smem = NB * ROW * 2;  // 80 KB (k 5), 192 KB (k 6), 128 KB (k 7)
};
constexpr int kTabThreads = 1024;

template <int K>
__global__ void __launch_bounds__(kTabThreads, 1) k_bfilter_tab(DevReads R, RoundState* st,
                                                                const int32_t* __restrict__ remain,
                                                                const int32_t* __restrict__ tent,
                                                                Pair* pairs, int seg_cap) {
    constexpr int RG = TabGroup<K>::RG;
    constexpr int ROW = TabGroup<K>::ROW;
    constexpr int W = RG / 2;  // packed sums per lane
    constexpr int WARPS = kTabThreads / 32;
    extern __shared__ __align__(16) uint16_t tab[];  // [NB][ROW], RG counts used per row
    __shared__ int4 tcomp[RG];
    __shared__ int ttent[RG];
    // a pass with a single tentative is k_filter's (launched before this one)
    if (st->done || st->n_tent <= 1) return;
    const int nt = st->n_tent;
    const int n = st->n_remain;
    const int ngroups = (nt + RG - 1) / RG;
    const int parts = max(1, (int)gridDim.x / ngroups);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned n_pf = 0, n_wf = 0, n_al = 0;
    unsigned long long bytes = 0;
    int cur_group = -1;
    for (int item = blockIdx.x; item < ngroups * parts; item += gridDim.x) {
        const int g = item % ngroups, part = item / ngroups;
        const int t0 = g * RG;
        const int ng = min(RG, nt - t0);
        if (g != cur_group) {
            __syncthreads();
            if (threadIdx.x < RG) {
                const int i = t0 + threadIdx.x;
                ttent[threadIdx.x] = threadIdx.x < ng ? tent[i] : 0x7fffffff;
                tcomp[threadIdx.x] = threadIdx.x < ng ? R.comp[tent[i]] : make_int4(0, 0, 0, 0);
            }
            uint4* t4 = reinterpret_cast<uint4*>(tab);
            for (int i = threadIdx.x; i < TabGroup<K>::smem / 16; i += kTabThreads)
                t4[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            // kernel_makeTable (func.cu:712-723) for each tentative: order > 0 only
            for (int t = warp; t < ng; t += WARPS) {
                const int rep = ttent[t];
                const uint32_t* e = R.kmer + R.kmer_off[rep];
                const int ne = R.n_kmer[rep];
                for (int i = lane; i < ne; i += 32) {
                    const uint32_t v = __ldg(e + i);
                    const uint32_t c = v & 0xffffu;
                    if (c) tab[(v >> 16) * ROW + t] = (uint16_t)c;
                }
            }
            __syncthreads();
            cur_group = g;
        }
        const int per = (n + parts - 1) / parts;
        const int lo = part * per, hi = min(n, lo + per);
        for (int idx = lo + warp; idx < hi; idx += WARPS) {
            const int q = remain[idx];
            if (g == 0) bytes += cand_bytes(R, q, false);  // once per launch
            // lane t < RG: order and composition bound of tentative t
            bool ok = false;
            if (lane < ng) {
                ok = ttent[lane] < q &&
                     prefilter_pass(tcomp[lane], R.comp[q], R.cut_base[q] - R.strict);
                n_pf += ttent[lane] < q;
            }
            const unsigned mask = __ballot_sync(kFull, ok);
            if (!mask) continue;
            n_wf += ok;
            uint32_t acc[W];
#pragma unroll
            for (int w = 0; w < W; w++) acc[w] = 0u;
            const int ne4 = (R.n_kmer[q] + 3) >> 2;
            const uint4* e4 = reinterpret_cast<const uint4*>(R.kmer + R.kmer_off[q]);
            for (int i = lane; i < ne4; i += 32) {
                const uint4 v = __ldcs(e4 + i);
                const uint32_t ev[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const uint32_t c = ev[e] & 0xffffu;
                    const uint32_t cc = c | (c << 16);
                    const uint32_t* row = reinterpret_cast<const uint32_t*>(tab + (ev[e] >> 16) * ROW);
                    if constexpr (RG >= 8) {
#pragma unroll
                        for (int w = 0; w < W; w += 4) {
                            const uint4 m = *reinterpret_cast<const uint4*>(row + w);
                            acc[w] = __vadd2(acc[w], __vminu2(m.x, cc));
                            acc[w + 1] = __vadd2(acc[w + 1], __vminu2(m.y, cc));
                            acc[w + 2] = __vadd2(acc[w + 2], __vminu2(m.z, cc));
                            acc[w + 3] = __vadd2(acc[w + 3], __vminu2(m.w, cc));
                        }
                    } else {
                        const uint2 m = *reinterpret_cast<const uint2*>(row);
                        acc[0] = __vadd2(acc[0], __vminu2(m.x, cc));
                        acc[1] = __vadd2(acc[1], __vminu2(m.y, cc));
                    }
                }
            }
            const int cw = R.cut_word[q];
            uint32_t mine = 0;
#pragma unroll
            for (int w = 0; w < W; w++) {
                const uint32_t s = __reduce_add_sync(kFull, acc[w]);
                if ((lane >> 1) == w) mine = s;
            }
            const int sum = (int)((lane & 1) ? (mine >> 16) : (mine & 0xffffu));
            const bool pass = ok && !(sum < cw);
            if (pass) push_pair(st, pairs, seg_cap, R, ttent[lane], q, kBandMaxW);
            n_al += pass;
        }
    }
    n_pf = (unsigned)warp_sum_i((int)n_pf);
    n_wf = (unsigned)warp_sum_i((int)n_wf);
    n_al = (unsigned)warp_sum_i((int)n_al);
    if (lane == 0) {
        if (n_pf) atomicAdd(&st->cnt_prefilter, (unsigned long long)n_pf);
        if (n_wf) atomicAdd(&st->cnt_word, (unsigned long long)n_wf);
        if (n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
        if (bytes) atomicAdd(&st->filter_bytes, bytes);
    }
}

// Drop mode, batched (clusteringDrop, func.cu:1068-1097): only the lossless
// composition bound (kernel_preFilter, func.cu:738-754) runs before the
// alignment.  A CTA stages 32 tentatives; one warp per candidate, lane t
// tests tentative t.
__global__ void __launch_bounds__(kFilterThreads) k_bprefilter(DevReads R, RoundState* st,
                                                               const int32_t* __restrict__ remain,
                                                               const int32_t* __restrict__ tent,
                                                               Pair* pairs, int seg_cap) {
    constexpr int RG = 32;
    __shared__ int4 tcomp[RG];
    __shared__ int ttent[RG];
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    const int nt = st->n_tent;
    const int n = st->n_remain;
    const int ngroups = (nt + RG - 1) / RG;
    const int parts = max(1, (int)gridDim.x / ngroups);
    const int lane = threadIdx.x & 31;
    unsigned n_pf = 0, n_al = 0;
    unsigned long long bytes = 0;
    int cur_group = -1;
    for (int item = blockIdx.x; item < ngroups * parts; item += gridDim.x) {
        const int g = item % ngroups, part = item / ngroups;
        const int t0 = g * RG;
        const int ng = min(RG, nt - t0);
        if (g != cur_group) {
            __syncthreads();
            if (threadIdx.x < RG) {
                const int i = t0 + threadIdx.x;
                ttent[threadIdx.x] = threadIdx.x < ng ? tent[i] : 0x7fffffff;
                tcomp[threadIdx.x] = threadIdx.x < ng ? R.comp[tent[i]] : make_int4(0, 0, 0, 0);
            }
            __syncthreads();
            cur_group = g;
        }
        // this item's slice of the candidate list, one warp per candidate
        const int per = (n + parts - 1) / parts;
        const int lo = part * per, hi = min(n, lo + per);
        for (int idx = lo + (threadIdx.x >> 5); idx < hi; idx += kFilterThreads / 32) {
            const int q = remain[idx];
            if (g == 0) bytes += cand_bytes(R, q, true);  // once per launch
            bool ok = false;
            if (lane < ng) {
                ok = ttent[lane] < q &&
                     prefilter_pass(tcomp[lane], R.comp[q], R.cut_base[q] - R.strict);
                n_pf += ttent[lane] < q;
            }
            if (ok) push_pair(st, pairs, seg_cap, R, ttent[lane], q, kBandMaxW);
            n_al += ok;
        }
    }
    n_pf = (unsigned)warp_sum_i((int)n_pf);
    n_al = (unsigned)warp_sum_i((int)n_al);
    if (lane == 0) {
        if (n_pf) atomicAdd(&st->cnt_prefilter, (unsigned long long)n_pf);
        if (n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
        if (bytes) atomicAdd(&st->filter_bytes, bytes);
    }
}

// ---- word filter by two-level k-mer count bitmaps (k <= kMaxBits2K) -------
//
// Per read two 4^k-bit bitmaps: level 1 holds the k-mers with a stored count
// of at least one, level 2 those with at least two; E3 is the excess above
// two, sum over k-mers of max(count - 2, 0).  The word sum of kernel_filter
// (func.cu:803-826) is S = sum over k-mers of min(c_t, c_q), and since
// min(c_t, c_q) = [both >= 1] + [both >= 2] + max(min(c_t, c_q) - 2, 0),
//     lo = D1 + D2 <= S <= lo + min(E3_t, E3_q),
// with D1, D2 the popcounts of the two levels' intersections.  The second
// level keeps the gap small where one level leaves it wide (reads holding a
// large share of the k-mer space, whose counts are mostly 1 or 2).  lo decides
// every pair outside the gap; the few pairs inside it go to k_bexact_t, which
// forms S itself.
//
// lo is an entry of a matrix product: the candidates' bitmaps (both levels end
// to end, 0/1) times the tentatives' transposed.  k_bfilter_bits forms it on
// the tensor cores: tiles of 128 candidates x up to 240 tentatives, the
// bitmaps spread to 4-bit values on their way into shared memory (any fixed
// order of a read's k-mers gives the same sum, so the spread is two
// multiplications, a shift and four masks per 32 k-mers), accumulators in
// tensor memory.
//
// A pass takes as short bitmaps as decide its pairs: both levels (depth 0),
// the first alone (1: S <= D + the smaller sum(count - 1)), or the first with
// its halves or quarters or'd together (2, 3: k-mers that share a bit count as
// one, their counts added; D no longer bounds S from below).  Every CTA
// estimates, from a sample of the pass's own pairs taken as unrelated reads,
// how many each depth would leave open, and takes the cheapest: the longest
// reads need both levels (5,000 bp hold most of the 6-mers),
// reads of 1,000 bp a quarter of the first.
//
// A CTA per SM: one warp issues the MMAs, 23 warps load and spread the
// bitmaps into a ring of two stages (512 k-mers of every row), and four warps
// read the finished tile's sums, apply the composition bound and queue the
// pairs while the next tile is summed in the other accumulator.  A producer
// lane loads 16 bytes of a row, eight lanes 128 contiguous bytes, and word w of
// its 16 bytes goes to the w-th chunk of 256 k-mers: full lines from L2 and whole
// rows of shared memory per store.
//
// The producers' hand-overs bound it: every warp takes part in every stage, so
// a stage lasts as long as one warp's wait, stores, fence and arrival.  Filter
// stage of 100k reads of 150-5,000 bp, t = 0.95 (90 passes of up to 92,000 x
// 1,024 pairs): 149 ms (AND + POPC lanes), 26.3 (four stages of 256 k-mers),
// 23.9 (two of the spread's shifts as multiplications), 21.8 (the depths, and
// an epilogue of 8 instead of ~17 ALU operations a pair, which alone changed
// nothing), 19.7 (stages of 512 k-mers, splits of the tentatives that fill the
// last wave).  30k reads, t = 0.90, k = 7: 42 -> 4.85 ms, with R_max 1024
// instead of 256, which the lanes' form could not stage; 10k reads of 200-1,000
// bp: 2.36 -> 0.75 ms.
// On the way there, with four stages, 84,800 x 1,024 pairs, 0.42 ms: eight
// producer loads of 32 bytes of a row each 0.49; 12 producers 0.53; the MMAs
// issued by a producer 0.73; branches per column in the epilogue 0.63.
// An open pair's exact sum (2 to 4 ns) in products of 1,024 bits of a pair (0.6
// ps): what a shorter bitmap may leave open for what it saves.
constexpr float kOpenCost = 6000.0f;
constexpr int kBitsProducers = 23;  // 4 rows per 8 lanes, 28 warps: 72 registers each
constexpr int kBitsEpilogue = 4;
constexpr int kBitsThreads = 32 * (1 + kBitsEpilogue + kBitsProducers);
constexpr int kBitsStages = 2;  // of two chunks of 256 k-mers
constexpr int kBitsChunkBytes = (128 + kTcMaxN) * kTcRowBytes;
constexpr int kBitsStageBytes = 2 * kBitsChunkBytes;
constexpr int kTentPad = kMaxBatch + 16;  // a tile's columns are read sixteen at a time
constexpr int kBitsSmem = 1024 + kBitsStages * kBitsStageBytes + kTentPad * (16 + 8 + 4 + 4);
static_assert(128 % 8 == 0 && kTcMaxN % 16 == 0, "whole groups of eight rows");
constexpr int kBitsRows = (128 + kTcMaxN + 4 * kBitsProducers - 1) / (4 * kBitsProducers);

// A limit of 0 polls (set_spin_limit) asks the tensor-core filters to give up:
// their stages then wait for one arrival more than there are, so that every
// warp's waits run out at their first poll and no product is issued.  In the
// waits themselves (a limit of 0 as it is, or a note of the first product) this
// took 0.4 to 1.4% of the hashed filter's time.
__device__ __forceinline__ int never_full() { return c_spin_limit <= 0 ? 1 : 0; }
constexpr int kDrainLimit = 1 << 14;  // polls for the products in flight (microseconds)

__device__ __forceinline__ uint2 comp_halves(const int4 c) {
    return make_uint2((uint32_t)min(c.x, 0xffff) | (uint32_t)min(c.y, 0xffff) << 16,
                      (uint32_t)min(c.z, 0xffff) | (uint32_t)min(c.w, 0xffff) << 16);
}

template <int K>
__global__ void __launch_bounds__(kBitsThreads, 1) k_bfilter_bits(
    DevReads R, RoundState* st, const int32_t* __restrict__ remain,
    const int32_t* __restrict__ tent, Pair* pairs, int seg_cap, Pair* amb, int amb_cap) {
    constexpr int NQ = (1 << (2 * K)) / 128;        // 16-byte words of one bitmap
    constexpr int GL = NQ >= 8 ? NQ / 8 : 1;        // groups of four stages per level
    constexpr int DEPTHS = K >= kMinFoldK ? kMaxDepth : K == 5 ? 1 : 0;
    // (a job without room for the folded bitmaps takes none of them)
    const int depths = R.kfold ? DEPTHS : min(DEPTHS, 1);
    extern __shared__ __align__(1024) uint8_t bsm_raw[];
    __shared__ uint64_t full[kBitsStages], empty[kBitsStages], tfull[2], tempty[2], drain;
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit, s_open[kMaxDepth + 1];
    if (threadIdx.x <= kMaxDepth) s_open[threadIdx.x] = 0;
    chain_wait();
    if (st->done) return;
    const int nt = st->n_tent;
    if (nt <= 1) return;  // a single tentative's pass runs k_filter instead
    const int n = st->n_remain;
    const int lane = threadIdx.x & 31, mtiles = (n + 127) >> 7;
    // The tentatives' split: a tile costs about its rows, candidates' and
    // tentatives', and the launch the most tiles of a CTA.  Each lane weighs
    // one split (every warp of every CTA finds the same).
    int tiles_n = (nt + kTcMaxN - 1) / kTcMaxN + lane;
    {
        const int cols = (((nt + tiles_n - 1) / tiles_n) + 15) & ~15;
        const int waves = (mtiles * tiles_n + (int)gridDim.x - 1) / (int)gridDim.x;
        tiles_n = (int)(__reduce_min_sync(kFull, (unsigned)(waves * (128 + cols)) << 6 |
                                                     (unsigned)tiles_n) & 63u);
    }
    const int N = (((nt + tiles_n - 1) / tiles_n) + 15) & ~15;  // tentatives per tile
    tiles_n = (nt + N - 1) / N;
    const int tiles = mtiles * tiles_n;
    if ((int)blockIdx.x >= tiles) return;
    uint8_t* stage0 = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(bsm_raw) + 1023) & ~(uintptr_t)1023);
    int4* tcomp = reinterpret_cast<int4*>(stage0 + kBitsStages * kBitsStageBytes);
    uint2* tpair = reinterpret_cast<uint2*>(tcomp + kTentPad);   // comp in 16-bit halves
    float* tex = reinterpret_cast<float*>(tpair + kTentPad);     // excess / kTcSpreadUnit
    int32_t* s_tent = reinterpret_cast<int32_t*>(tex + kTentPad);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kBitsStages; i++) {
            mbar_init(&full[i], kBitsProducers + never_full());
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], kBitsEpilogue);
        }
        mbar_init(&drain, 1);
        s_quit = 0;
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc_all(&s_tmem);
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
        const int rep = tent[t];
        const int4 c = R.comp[rep];
        s_tent[t] = rep;
        tcomp[t] = c;
        tpair[t] = comp_halves(c);
    }
    __syncthreads();
    if (DEPTHS > 0) {
        // the chance that a sampled pair of unrelated reads stays open
        const int rep = tent[threadIdx.x % nt];
        const int q = remain[(int)((long long)threadIdx.x * n / kBitsThreads)];
        const int xq = R.kextra[q], xr = R.kextra[rep], cw = R.cut_word[q];
        const int kq = R.n_kmer[q] + xq, kr = R.n_kmer[rep] + xr;
#pragma unroll
        for (int d = 1; d <= DEPTHS; d++) {
            if (d > depths) break;
            const int eq = d == 1 ? xq : R.kfextra[(size_t)(d - 2) * R.n + q];
            const int er = d == 1 ? xr : R.kfextra[(size_t)(d - 2) * R.n + rep];
            const float w = 1.0f / (float)((1 << (2 * K)) >> (d - 1));
            const float fq = (float)(kq - eq) * w, mean = (float)(kr - er) * fq;
            const float var = mean * (1.0f - fq) * (1.0f - (float)(kr - er) * w);
            const float z = ((float)(cw - min(eq, er)) - mean) * rsqrtf(2.0f * var + 1.0f);
            int open = rep < q ? (int)(32768.0f * erfcf(z)) : 0;
            open = __reduce_add_sync(kFull, open);
            if (lane == 0 && open) atomicAdd(&s_open[d], open);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (warp >= 1 && warp <= 4) tc_fill_scales(tmem, warp);
    int depth = 0;
    float cost = (float)(2 * GL);
#pragma unroll
    for (int d = 1; d <= DEPTHS; d++) {
        const float c = (float)(GL >> (d - 1)) +
                        kOpenCost * (float)s_open[d] * (1.0f / (65536.0f * kBitsThreads));
        if (d <= depths && (st->bits_hold == 0 || d <= st->bits_cap) && c < cost)
            depth = d, cost = c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) st->bits_depth = depth;
    // groups of two stages (1,024 bits) per tile (k = 4: half of them zeros)
    const int groups = K == 4 ? 1 : depth == 0 ? 2 * GL : GL >> (depth - 1);
    const int CH = 2 * groups;
    const int32_t* ex = depth == 0   ? R.kextra3
                        : depth == 1 ? R.kextra
                                     : R.kfextra + (size_t)(depth - 2) * R.n;
    for (int t = threadIdx.x; t < nt; t += blockDim.x)
        tex[t] = (float)ex[s_tent[t]] * (1.0f / kTcSpreadUnit);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const int limit = max(c_spin_limit, 1);
    bool ok = true;  // this warp's waits all ended
    if (warp == 0) {
        if (lane == 0) {
            const uint32_t idesc = tc_idesc_fp4(N);
            int s = 0, it = 0;
            uint32_t ph = 0;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, it++) {
                const int buf = it & 1;
                // (the first use of each accumulator passes at once)
                ok = mbar_wait(&tempty[buf], ((it >> 1) & 1) ^ 1, limit, &s_quit);
                for (int c = 0; ok && c < CH; c++) {
                    ok = mbar_wait(&full[s], ph, limit, &s_quit);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = tc_desc_lo(smem_u32(stage0 + s * kBitsStageBytes));
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        tc_mma_stage(tmem + buf * kTcMaxN, tmem, a + u * kBitsChunkBytes / 16,
                                     a + (u * kBitsChunkBytes + 128 * kTcRowBytes) / 16, idesc,
                                     c == 0 && u == 0);
                    tc_commit(&empty[s]);
                    if (++s == kBitsStages) s = 0, ph ^= 1;
                }
                if (ok) tc_commit(&tfull[buf]);
            }
        }
    } else if (warp <= kBitsEpilogue) {
        const int row = (warp & 3) * 32 + lane;
        unsigned n_wf = 0, n_al = 0;
        unsigned long long n_pf = 0, bytes = 0;
        int it = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, it++) {
            const int m = tile / tiles_n, t0 = (tile - m * tiles_n) * N;
            const int t1 = min(nt, t0 + N);
            const int idx = m * 128 + row;
            int q = -1, cw = 0, exq = 0, cbq = 0;
            int4 cq = make_int4(0, 0, 0, 0);
            if (idx < n) {
                q = remain[idx];
                cw = R.cut_word[q];
                exq = ex[q];
                cq = R.comp[q];
                cbq = R.cut_base[q] - R.strict;
                // once per launch
                if (t0 == 0) bytes += kCandFixedBytes + (K == 4 ? 64ull : 128ull * groups);
            }
            const int buf = it & 1;
            ok = mbar_wait_warp(&tfull[buf], (it >> 1) & 1, limit, &s_quit);
            if (!ok) break;
            tc_fence_after();
            const uint32_t addr = tmem + ((uint32_t)(warp & 3) << 21) + buf * kTcMaxN;
            // tentatives of the tile before q (the list ascends)
            int ntq = q < 0 ? t0 : t1;
            if (q >= 0 && q <= s_tent[t1 - 1]) {
                int lo = t0, hi = t1;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s_tent[mid] < q) lo = mid + 1;
                    else hi = mid;
                }
                ntq = lo;
            }
            // the sums' scale, and the composition in 16-bit halves (no row
            // with a count above that takes the short form below)
            const float cwf = (float)cw * (1.0f / kTcSpreadUnit);
            const float exf = (float)exq * (1.0f / kTcSpreadUnit);
            const uint2 ch = comp_halves(cq);
            const bool halves = max(max(cq.x, cq.y), max(cq.z, cq.w)) <= 0xffff;
            for (int c0 = t0; c0 < t1; c0 += 16) {
                uint32_t raw[16];
                float v[16];
                const int ncol = ntq - c0;
                if (!__any_sync(kFull, ncol > 0)) break;
                tc_load16(raw, addr + (c0 - t0));
                tc_load_wait(raw, v);
                if (__all_sync(kFull, ncol >= 16 && halves)) {
                    // sixteen independent chains: the largest bound, and how
                    // many fail kernel_preFilter (func.cu:738-754)
                    float top[2] = {-1.0f, -1.0f};
                    uint32_t fail[2] = {0, 0};
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const uint2 tp = tpair[c0 + j];
                        const uint32_t d =
                            __dp2a_lo(__vminu2(tp.x, ch.x), 0x0101u,
                                      __dp2a_lo(__vminu2(tp.y, ch.y), 0x0101u, 0u - (uint32_t)cbq));
                        fail[j & 1] += d >> 31;
                        top[j & 1] = fmaxf(top[j & 1], v[j] + fminf(tex[c0 + j], exf));
                    }
                    if (!__any_sync(kFull, fmaxf(top[0], top[1]) >= cwf)) {
                        n_pf += 16;
                        n_wf += 16 - (fail[0] + fail[1]);
                        continue;
                    }
                }
                // a row at its own place in the tentatives, or a pair left open
                uint32_t pre = 0, hit = 0;
#pragma unroll
                for (int j = 0; j < 16; j++) {  // (entries past nt: any values, masked below)
                    pre |= prefilter_pass(tcomp[c0 + j], cq, cbq) ? 1u << j : 0u;
                    hit |= v[j] + fminf(tex[c0 + j], exf) >= cwf ? 1u << j : 0u;
                }
                const uint32_t before = ncol >= 16 ? 0xffffu : ncol > 0 ? (1u << ncol) - 1u : 0u;
                pre &= before;
                hit &= pre;
                n_pf += __popc(before);
                n_wf += __popc(pre);
                while (hit) {
                    const int j = __ffs(hit) - 1;
                    hit &= hit - 1;
                    float vj = v[0];
#pragma unroll
                    for (int i = 1; i < 16; i++) vj = j == i ? v[i] : vj;
                    const int rep = s_tent[c0 + j];
                    if (depth < 2 && vj >= cwf) {
                        push_pair(st, pairs, seg_cap, R, rep, q, kBandMaxW);
                        n_al++;
                    } else {
                        const int slot = atomicAdd(&st->n_amb, 1);
                        if (slot < amb_cap) amb[slot] = Pair{rep, q};
                        else st->pair_overflow = 1;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[buf]);
        }
        n_wf = (unsigned)warp_sum_i((int)n_wf);
        n_al = (unsigned)warp_sum_i((int)n_al);
        n_pf = warp_sum_ull(n_pf);
        bytes = warp_sum_ull(bytes);
        if (lane == 0) {
            if (n_pf) atomicAdd(&st->cnt_prefilter, n_pf);
            if (n_wf) atomicAdd(&st->cnt_word, (unsigned long long)n_wf);
            if (n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
            if (bytes) atomicAdd(&st->filter_bytes, bytes);
        }
    } else {
        // producers: lane piece p = lane % 8 (16 bytes of 128) of rows r0 +
        // 92 j (rows 0..127: the tile's candidates, then its tentatives)
        const int tid = threadIdx.x - 32 * (1 + kBitsEpilogue);
        const uint4* kb1 = reinterpret_cast<const uint4*>(
            depth < 2 ? R.kbits : R.kfold + (depth == 3 ? (size_t)R.n * (2 * NQ) : 0));
        const uint4* kb2 = reinterpret_cast<const uint4*>(R.kbits2);
        const int rowq = depth < 2 ? NQ : NQ >> (depth - 1);
        const int p = tid & 7, r0 = tid >> 3;
        constexpr int RS = 4 * kBitsProducers;  // rows per sweep
        static_assert(RS % 8 == 4 && RS * kBitsRows == 128 + kTcMaxN, "row layout");
        const int off0 = r0 * kTcRowBytes + ((p ^ (r0 & 7)) << 4);
        const int odd = ((p ^ ((r0 + 4) & 7)) << 4) - ((p ^ (r0 & 7)) << 4);
        const int rows = (128 + N - r0 + RS - 1) / RS;
        // (rows past the last candidate or tentative hold read 0: their sums
        // are not looked at)
        auto read_of = [&](int tile, int r) -> int {
            if (tile >= tiles) return 0;
            const int m = tile / tiles_n, t0 = (tile - m * tiles_n) * N;
            if (r < 128) return m * 128 + r < n ? remain[m * 128 + r] : 0;
            r -= 128;
            return r < N && t0 + r < nt ? tent[t0 + r] : 0;
        };
        int ft = blockIdx.x, fg = 0;  // the next group to load
        int cur[kBitsRows], nxt[kBitsRows];
#pragma unroll
        for (int j = 0; j < kBitsRows; j++) {
            cur[j] = read_of(ft, r0 + RS * j);
            nxt[j] = read_of(ft + gridDim.x, r0 + RS * j);
        }
        auto load = [&](uint4 (&v)[kBitsRows]) {
#pragma unroll
            for (int j = 0; j < kBitsRows; j++) {
                if constexpr (K == 4) {
                    v[j] = make_uint4(0u, 0u, 0u, 0u);
                    if (p < 4) v[j] = __ldg((p < 2 ? kb1 : kb2) + (size_t)cur[j] * NQ + (p & 1));
                } else {
                    v[j] = __ldg((fg < GL ? kb1 : kb2) + (size_t)cur[j] * rowq +
                                 8 * (fg & (GL - 1)) + p);
                }
            }
            if (++fg == groups) {
                fg = 0;
                ft += gridDim.x;
#pragma unroll
                for (int j = 0; j < kBitsRows; j++) {
                    cur[j] = nxt[j];
                    nxt[j] = read_of(ft + gridDim.x, r0 + RS * j);
                }
            }
        };
        int s = 0;
        uint32_t ph = 1;  // the first round of stages is free
        // the two stages of one group
        auto store = [&](const uint4 (&v)[kBitsRows]) {
#pragma unroll
            for (int w = 0; w < 4; w += 2) {
                ok = mbar_wait_warp(&empty[s], ph, limit, &s_quit);
                if (!ok) return;
                uint8_t* base = stage0 + s * kBitsStageBytes + off0;
#pragma unroll
                for (int j = 0; j < kBitsRows; j++) {
                    // (row r0 + RS j: RS is 4 mod 8, so the swizzle alternates)
                    if (j >= rows) break;
                    uint8_t* d = base + j * RS * kTcRowBytes + (j & 1 ? odd : 0);
                    *reinterpret_cast<uint4*>(d) = tc_spread(w ? v[j].z : v[j].x);
                    *reinterpret_cast<uint4*>(d + kBitsChunkBytes) =
                        tc_spread(w ? v[j].w : v[j].y);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
                if (++s == kBitsStages) s = 0, ph ^= 1;
            }
        };
        const int mine =
            (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * groups;
        uint4 va[kBitsRows], vb[kBitsRows];
        load(va);
        for (int i = 0; ok && i < mine; i += 2) {
            load(vb);
            store(va);
            if (!ok || i + 1 >= mine) break;
            load(va);
            store(vb);
        }
    }
    if (!ok) {
        // a wait gave up: the others stop at their next poll
        s_quit = 1;
        st->error = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (s_quit && lane == 0 && !never_full()) {
            // the MMAs in flight, before the accumulators are given back
            const int none = 0;
            tc_commit(&drain);
            mbar_wait(&drain, 0, kDrainLimit, &none);
        }
        __syncwarp();
        tmem_free_all(tmem);
    }
}

// Carry-save adder: a + b + c = s + 2 * carry, bit by bit (two LOP3s).
__device__ __forceinline__ void csa(uint32_t& s, uint32_t& carry, uint32_t a, uint32_t b,
                                    uint32_t c) {
    s = a ^ b ^ c;
    carry = (a & b) | (c & (a ^ b));
}

// The open pairs grouped by tentative.  In the early passes of long-read
// jobs most pairs are open (477k of 668k in the seventh pass of the 200k-read
// workload, ~4,600 per tentative); one table per pair would be zeroed and
// refilled ~4,600 times per tentative.  A counting sort of the queue by tentative index
// (k_amb_count, k_amb_scan, k_amb_place) lets k_bexact_t build each
// tentative's table once per CTA for a run of its pairs.  The order of the
// pairs inside a tentative's run does not matter: each decision is a pure
// function of its pair.
//
// amb_idx holds four arrays of kMaxBatch + 1: per tentative the pair count
// (kept zero between passes), the run offsets, the placement cursors and the
// work items (runs of up to kExactChunk pairs), as exclusive prefix sums.
constexpr int kExactChunk = 64;
constexpr int kAmbThreads = 256;

__device__ __forceinline__ int amb_n(const RoundState* st, int amb_cap) {
    return min(st->n_amb, amb_cap);
}

// Per-CTA histogram of the open pairs' tentatives, added into the global one.
__global__ void __launch_bounds__(kAmbThreads) k_amb_count(RoundState* st, const Pair* __restrict__ amb,
                                                          int amb_cap, const uint32_t* __restrict__ tidx,
                                                          int* amb_idx) {
    __shared__ int h[kMaxBatch];
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    const int na = amb_n(st, amb_cap);
    if (na <= 0) return;
    const int nt = st->n_tent;
    for (int t = threadIdx.x; t < nt; t += blockDim.x) h[t] = 0;
    __syncthreads();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < na; k += gridDim.x * blockDim.x)
        atomicAdd(&h[tidx[amb[k].rep] & 0xfff], 1);
    __syncthreads();
    for (int t = threadIdx.x; t < nt; t += blockDim.x)
        if (h[t]) atomicAdd(&amb_idx[t], h[t]);
}

// One CTA of 1,024 threads: run offsets, cursors and work items; the counts
// go back to zero for the next pass.
__global__ void __launch_bounds__(1024) k_amb_scan(RoundState* st, int amb_cap, int* amb_idx) {
    __shared__ int ws[2][32];
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    if (amb_n(st, amb_cap) <= 0) return;
    const int nt = st->n_tent;
    int* cnt = amb_idx;
    int* off = amb_idx + (kMaxBatch + 1);
    int* cur = amb_idx + 2 * (kMaxBatch + 1);
    int* items = amb_idx + 3 * (kMaxBatch + 1);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c = t < nt ? cnt[t] : 0;
    const int ch = (c + kExactChunk - 1) / kExactChunk;
    int ic = c, ich = ch;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int a = __shfl_up_sync(kFull, ic, d), b = __shfl_up_sync(kFull, ich, d);
        if (lane >= d) ic += a, ich += b;
    }
    if (lane == 31) ws[0][warp] = ic, ws[1][warp] = ich;
    __syncthreads();
    int bc = 0, bch = 0;
    for (int w = 0; w < warp; w++) bc += ws[0][w], bch += ws[1][w];
    const int ec = bc + ic - c, ech = bch + ich - ch;
    if (t < nt) {
        off[t] = ec;
        cur[t] = ec;
        items[t] = ech;
        cnt[t] = 0;
    }
    if (t == nt - 1) {
        off[nt] = ec + c;
        items[nt] = ech + ch;
    }
}

// Each CTA places a contiguous range of the queue: a shared histogram, one
// global reservation per (CTA, tentative), then the pairs.
__global__ void __launch_bounds__(kAmbThreads) k_amb_place(RoundState* st, const Pair* __restrict__ amb,
                                                          int amb_cap, const uint32_t* __restrict__ tidx,
                                                          int* amb_idx, Pair* amb2) {
    __shared__ int h[kMaxBatch];
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    const int na = amb_n(st, amb_cap);
    if (na <= 0) return;
    const int nt = st->n_tent;
    int* cur = amb_idx + 2 * (kMaxBatch + 1);
    const int per = (na + gridDim.x - 1) / gridDim.x;
    const int lo = blockIdx.x * per, hi = min(na, lo + per);
    if (lo >= hi) return;
    for (int t = threadIdx.x; t < nt; t += blockDim.x) h[t] = 0;
    __syncthreads();
    for (int k = lo + threadIdx.x; k < hi; k += blockDim.x) atomicAdd(&h[tidx[amb[k].rep] & 0xfff], 1);
    __syncthreads();
    for (int t = threadIdx.x; t < nt; t += blockDim.x)
        if (h[t]) h[t] = atomicAdd(&cur[t], h[t]);
    __syncthreads();
    for (int k = lo + threadIdx.x; k < hi; k += blockDim.x) {
        const Pair p = amb[k];
        amb2[atomicAdd(&h[tidx[p.rep] & 0xfff], 1)] = p;
    }
}

// The word sum S of the open pairs, run by run: a CTA takes a contiguous range
// of work items, builds the tentative's count table in shared memory when the
// tentative changes, and each warp streams one candidate's (k-mer, count)
// entries against it (kernel_filter, func.cu:803-826).
template <int K>
__global__ void __launch_bounds__(kAmbThreads) k_bexact_t(DevReads R, RoundState* st,
                                                        const Pair* __restrict__ amb2,
                                                        const int* __restrict__ amb_idx,
                                                        int amb_cap,
                                                        const int32_t* __restrict__ tent,
                                                        Pair* pairs, int seg_cap) {
    constexpr int NB = 1 << (2 * K);
    extern __shared__ __align__(16) uint16_t xtab[];  // NB counts
    __shared__ int s_items[kMaxBatch + 1];
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    if (amb_n(st, amb_cap) <= 0) return;
    const int nt = st->n_tent;
    const int* off = amb_idx + (kMaxBatch + 1);
    const int* items = amb_idx + 3 * (kMaxBatch + 1);
    for (int i = threadIdx.x; i <= nt; i += blockDim.x) s_items[i] = items[i];
    __syncthreads();
    const int total = s_items[nt];
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int i0 = blockIdx.x * per, i1 = min(total, i0 + per);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    unsigned n_al = 0;
    int cur_t = -1;
    for (int item = i0; item < i1; item++) {
        // the tentative of this item: the last t with s_items[t] <= item
        int lo = 0, hi = nt;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_items[mid] <= item) lo = mid;
            else hi = mid;
        }
        const int t = lo;
        if (t != cur_t) {
            __syncthreads();
            uint4* t4 = reinterpret_cast<uint4*>(xtab);
            for (int i = threadIdx.x; i < NB / 8; i += blockDim.x) t4[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            const int rep = tent[t];
            const uint32_t* et = R.kmer + R.kmer_off[rep];
            const int ne = R.n_kmer[rep];
            for (int i = threadIdx.x; i < ne; i += blockDim.x) {
                const uint32_t v = __ldg(et + i);
                const uint32_t c = v & 0xffffu;
                if (c) xtab[v >> 16] = (uint16_t)c;  // kernel_makeTable: only order > 0
            }
            __syncthreads();
            cur_t = t;
        }
        const int k0 = off[t] + (item - s_items[t]) * kExactChunk;
        const int k1 = min(off[t + 1], k0 + kExactChunk);
        for (int k = k0 + warp; k < k1; k += warps) {
            const Pair p = amb2[k];
            const uint32_t* eq = R.kmer + R.kmer_off[p.cand];
            const int nq = R.n_kmer[p.cand];
            int sum = 0;
            for (int i = lane; i < nq; i += 32) {
                const uint32_t v = __ldg(eq + i);
                sum += min((uint32_t)xtab[v >> 16], v & 0xffffu);
            }
            sum = warp_sum_i(sum);
            if (!(sum < R.cut_word[p.cand])) {
                if (lane == 0) push_pair(st, pairs, seg_cap, R, p.rep, p.cand, kBandMaxW);
                n_al++;
            }
        }
    }
    if (lane == 0 && n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
}

// The word sum S of the open pairs where reads are short (the hashed form: at
// most 1,023 k-mers): one warp per pair, straight from the queue.  The
// representative's k-mers set bits of a presence bitmap of the warp's own in
// shared memory, the candidate's look them up: D shared k-mers and the two
// reads' excesses over distinct k-mers bound S (D <= S <= D + the smaller
// excess).  In short reads few k-mers repeat, so that decides nearly every
// pair; the rest is summed with an open-addressed table in the same place
// (hslots words, a power of two and at least twice the longest list).
//
// Instruction issue and the chain of loads (pair, offsets, lists: ~10 us in a
// pass of few pairs) bound it.  1M reads of 100-150 bp, k = 7, t = 0.90, passes
// of ~25,000 open pairs: 17 us; 38 us with a table for every pair (850
// instructions each); 62 us sorted by tentative with a table of all k-mers
// each, as for longer reads (32 KB of table for some 25 pairs).  The job's
// passes: 140.4 -> 130.9 ms.
constexpr int kDirectWarps = 8;
constexpr int kDirectMaxSlots = 2048;

__device__ __forceinline__ int direct_words(const DevReads& R) {
    return max(R.hslots, (1 << (2 * R.k)) / 32);
}

// S by the table; the lists are distinct k-mers, so the table's inserts end.
__device__ __noinline__ int direct_sum(uint32_t* tab, int slots, const uint32_t* er, int nr,
                                       const uint32_t* eq, int nq) {
    constexpr uint32_t kEmpty = 0xffffffffu;  // no entry: a k-mer has at most 14 bits
    const int lane = threadIdx.x & 31, mask = slots - 1, shift = 33 - __ffs(slots);
    for (int i = lane; i < slots; i += 32) tab[i] = kEmpty;
    __syncwarp();
    for (int i = lane; i < nr; i += 32) {
        const uint32_t v = __ldg(er + i);
        int h = ((v >> 16) * 0x9e3779b1u) >> shift;
        for (int n = 0; n < slots && atomicCAS(tab + h, kEmpty, v) != kEmpty; n++)
            h = (h + 1) & mask;
    }
    __syncwarp();
    int sum = 0;
    for (int i = lane; i < nq; i += 32) {
        const uint32_t v = __ldg(eq + i);
        int h = ((v >> 16) * 0x9e3779b1u) >> shift;
        uint32_t e = tab[h];
        for (int n = 0; n < slots && e != kEmpty && e >> 16 != v >> 16; n++)
            e = tab[h = (h + 1) & mask];
        if (e >> 16 == v >> 16) sum += (int)min(e & 0xffffu, v & 0xffffu);
    }
    __syncwarp();
    return __reduce_add_sync(kFull, sum);
}

__global__ void __launch_bounds__(32 * kDirectWarps) k_bexact_d(DevReads R, RoundState* st,
                                                              const Pair* __restrict__ amb,
                                                              int amb_cap, Pair* pairs,
                                                              int seg_cap) {
    extern __shared__ __align__(16) uint32_t dtab[];
    constexpr int U = 5;  // 150 bp reads in one go
    chain_wait();
    if (st->done || st->n_tent == 0) return;
    const int na = amb_n(st, amb_cap);
    const int nw = gridDim.x * kDirectWarps;
    const int lane = threadIdx.x & 31;
    if (blockIdx.x * kDirectWarps >= na) return;
    const int words = (1 << (2 * R.k)) / 32;
    uint32_t* bits = dtab + (threadIdx.x >> 5) * direct_words(R);
    unsigned n_al = 0;
    for (int k = blockIdx.x * kDirectWarps + (threadIdx.x >> 5); k < na; k += nw) {
        const Pair p = amb[k];
        const uint32_t* er = R.kmer + R.kmer_off[p.rep];
        const uint32_t* eq = R.kmer + R.kmer_off[p.cand];
        const int nr = R.n_kmer[p.rep], nq = R.n_kmer[p.cand];
        const int cw = R.cut_word[p.cand];
        for (int i = lane; i < words / 4; i += 32)
            reinterpret_cast<uint4*>(bits)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        // (an absent entry stands as a k-mer with count 1 that sets no bit)
        int ex_r = 0, d_ex = 0;  // d_ex: the candidate's excess << 16 | shared k-mers
        for (int i0 = lane; i0 < nr; i0 += 32 * U) {
            uint32_t v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = i0 + 32 * u < nr ? __ldg(er + i0 + 32 * u) : 1u;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (i0 + 32 * u < nr) atomicOr(bits + (v[u] >> 21), 1u << ((v[u] >> 16) & 31));
                ex_r += (int)(v[u] & 0xffffu) - 1;
            }
        }
        __syncwarp();
        for (int i0 = lane; i0 < nq; i0 += 32 * U) {
            uint32_t v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = i0 + 32 * u < nq ? __ldg(eq + i0 + 32 * u) : 1u;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t hit = bits[v[u] >> 21] >> ((v[u] >> 16) & 31) & 1u;
                d_ex += (int)((v[u] & 0xffffu) - 1u) << 16;
                d_ex += i0 + 32 * u < nq ? (int)hit : 0;
            }
        }
        __syncwarp();
        ex_r = __reduce_add_sync(kFull, ex_r);
        d_ex = __reduce_add_sync(kFull, d_ex);
        int sum = d_ex & 0xffff;
        if (sum < cw && sum + min(ex_r, d_ex >> 16) >= cw)
            sum = direct_sum(bits, R.hslots, er, nr, eq, nq);
        if (sum >= cw) {
            if (lane == 0) push_pair(st, pairs, seg_cap, R, p.rep, p.cand, kBandMaxW);
            n_al++;
        }
    }
    add_counts(st, lane, 0, 0, n_al, 0);
}

// ---- word filter by inverted index (sparse k-mer spaces) -------------------
//
// With short reads and k = 7 a tentative holds ~1% of the 4^k k-mers, so the
// table form spends almost every lookup on a zero.  Instead, each pass lists,
// per k-mer, the tentatives that hold it (k_bindex), and every candidate walks
// the lists of its own k-mers once, adding min(count in tentative, count in
// candidate) into one 16-bit counter per tentative (k_bfilter_idx).  The sums
// are the same integers kernel_filter forms (func.cu:803-826); only the order
// of the additions differs.

constexpr int kIndexThreads = 1024;

// One CTA: histogram of the tentatives' k-mers, exclusive scan into idx_off,
// scatter of (tentative << 16 | count) into idx_post.  The order inside one
// k-mer's list is arbitrary; the filter's sums do not depend on it.  With
// off16/post16 (capacity below 65536) it also writes the 16-bit copy that
// k_bfilter_idx keeps in shared memory: (tentative << 6 | min(count, 63)).
template <int K>
__global__ void __launch_bounds__(kIndexThreads, 1) k_bindex(DevReads R, RoundState* st,
                                                          const int32_t* __restrict__ tent,
                                                          uint32_t* idx_off, uint32_t* idx_post,
                                                          uint16_t* off16, uint16_t* post16,
                                                          long long idx_cap) {
    constexpr int NB = 1 << (2 * K);
    constexpr int PER = NB >= kIndexThreads ? NB / kIndexThreads : 1;
    extern __shared__ uint32_t cnt[];  // NB counters, then the scatter cursors
    __shared__ uint32_t wsum[32];
    if (st->done || st->n_tent == 0) return;
    const int nt = st->n_tent;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < NB; i += kIndexThreads) cnt[i] = 0u;
    __syncthreads();
    for (int t = warp; t < nt; t += kIndexThreads / 32) {
        const int rep = tent[t];
        const uint32_t* e = R.kmer + R.kmer_off[rep];
        const int ne = R.n_kmer[rep];
        for (int i = lane; i < ne; i += 32) {
            const uint32_t v = __ldg(e + i);
            if (v & 0xffffu) atomicAdd(&cnt[v >> 16], 1u);
        }
    }
    __syncthreads();
    // exclusive scan: thread i owns counters [i*PER, i*PER + PER)
    const int base = threadIdx.x * PER;
    uint32_t run = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) run += base + j < NB ? cnt[base + j] : 0u;
    uint32_t incl = run;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int w = 0; w < kIndexThreads / 32; w++) {
        const uint32_t s = wsum[w];
        if (w < warp) before += s;
        total += s;
    }
    uint32_t pos = before + incl - run;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (base + j < NB) {
            const uint32_t c = cnt[base + j];
            idx_off[base + j] = pos;
            if (off16) off16[base + j] = (uint16_t)pos;
            cnt[base + j] = pos;  // becomes the scatter cursor
            pos += c;
        }
    }
    if (threadIdx.x == 0) {
        idx_off[NB] = total;
        if (off16) off16[NB] = (uint16_t)total;
    }
    if ((long long)total > idx_cap) {
        // cannot happen for length-sorted reads (the capacity holds the R_max
        // longest k-mer lists); stop the job instead of writing past the end
        if (threadIdx.x == 0) {
            st->error = 3;
            st->done = 1;
        }
        return;
    }
    __syncthreads();
    for (int t = warp; t < nt; t += kIndexThreads / 32) {
        const int rep = tent[t];
        const uint32_t* e = R.kmer + R.kmer_off[rep];
        const int ne = R.n_kmer[rep];
        for (int i = lane; i < ne; i += 32) {
            const uint32_t v = __ldg(e + i);
            const uint32_t c = v & 0xffffu;
            if (c) {
                const uint32_t at = atomicAdd(&cnt[v >> 16], 1u);
                idx_post[at] = ((uint32_t)t << 16) | c;
                if (post16) post16[at] = (uint16_t)(((uint32_t)t << 6) | min(c, 63u));
            }
        }
    }
}

// Shared memory of k_bfilter_idx, in 32-bit words, every region on a 16-byte
// boundary.  SMEM form: the whole index as 16-bit entries (offsets, and
// postings (tentative << 6 | min(count, 63)), 63 meaning "read the exact count
// from the 32-bit list"); otherwise the 32-bit offsets only.  Then the
// tentatives, and per warp the 16-bit sums (two per word).
constexpr int kIdxGroups = 8;  // groups of 32 k-mer entries held in registers at a time
struct IndexSmem {
    int off_words, post_words, tent_words, acc_words;
    __host__ __device__ IndexSmem(int k, int r_max, long long cap, bool smem_index) {
        const int nb1 = (1 << (2 * k)) + 1;
        off_words = smem_index ? ((nb1 + 7) & ~7) / 2 : (nb1 + 3) & ~3;
        post_words = smem_index ? (int)(((cap + 7) & ~7LL) / 2) : 0;
        tent_words = (r_max + 3) & ~3;
        acc_words = ((r_max + 1) / 2 + 3) & ~3;
    }
    __host__ __device__ int warp_words() const { return acc_words; }
    __host__ __device__ int bytes(int warps) const {
        return 4 * (off_words + post_words + tent_words + warps * warp_words());
    }
};

template <int K, bool SMEM>
__global__ void __launch_bounds__(1024, 1) k_bfilter_idx(
    DevReads R, RoundState* st, const int32_t* __restrict__ remain,
    const int32_t* __restrict__ tent, const uint32_t* __restrict__ idx_off,
    const uint32_t* __restrict__ idx_post, const uint16_t* __restrict__ off16,
    const uint16_t* __restrict__ post16, int r_max, long long cap, Pair* pairs, int seg_cap) {
    constexpr int NB = 1 << (2 * K);
    extern __shared__ __align__(16) uint32_t sm[];
    if (st->done || st->n_tent == 0) return;
    const IndexSmem L(K, r_max, cap, SMEM);
    const int warps = blockDim.x >> 5;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t* s_off16 = reinterpret_cast<uint16_t*>(sm);
    uint32_t* s_off32 = sm;
    uint16_t* s_post16 = reinterpret_cast<uint16_t*>(sm + L.off_words);
    int32_t* s_tent = reinterpret_cast<int32_t*>(sm + L.off_words + L.post_words);
    uint32_t* const acc = sm + L.off_words + L.post_words + L.tent_words + warp * L.warp_words();
    const int nt = st->n_tent;
    const int n = st->n_remain;
    if (SMEM) {
        const int total = (int)idx_off[NB];
        const uint4* g = reinterpret_cast<const uint4*>(post16);
        uint4* d = reinterpret_cast<uint4*>(s_post16);
        for (int i = threadIdx.x; i < (total + 7) >> 3; i += blockDim.x) d[i] = __ldg(g + i);
        const uint4* go = reinterpret_cast<const uint4*>(off16);
        uint4* dof = reinterpret_cast<uint4*>(s_off16);
        for (int i = threadIdx.x; i < (NB + 1 + 7) >> 3; i += blockDim.x) dof[i] = __ldg(go + i);
    } else {
        for (int i = threadIdx.x; i < NB + 1; i += blockDim.x) s_off32[i] = __ldg(idx_off + i);
    }
    for (int i = threadIdx.x; i < nt; i += blockDim.x) s_tent[i] = tent[i];
    for (int i = lane; i < L.acc_words; i += 32) acc[i] = 0u;
    __syncthreads();
    unsigned long long n_pf = 0, bytes = 0;
    unsigned n_wf = 0, n_al = 0;
    const int nwarps = gridDim.x * warps;
    // software pipeline over the warp's candidates: the next candidate's read
    // index and k-mer list position load while this one is summed
    int idx = blockIdx.x * warps + warp;
    int q_nx = idx < n ? remain[idx] : 0;
    const uint32_t* e_nx = R.kmer + (idx < n ? R.kmer_off[q_nx] : 0);
    int ne_nx = idx < n ? R.n_kmer[q_nx] : 0;
    for (; idx < n; idx += nwarps) {
        const int q = q_nx;
        const uint32_t* const e = e_nx;
        const int ne = ne_nx;
        if (idx + nwarps < n) q_nx = remain[idx + nwarps];
        // tentatives before q: the first ntq of the ascending list (all of
        // them for every candidate past the last tentative)
        int lo = 0, hi = nt;
        if (s_tent[nt - 1] < q) lo = nt;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_tent[mid] < q) lo = mid + 1;
            else hi = mid;
        }
        const int ntq = lo;
        n_pf += ntq;
        bytes += kCandFixedBytes + 4ull * (unsigned)ne;
        // sum over q's k-mers of min(count in q, count in tentative), per
        // tentative.  The warp takes 32 k-mers at a time, one per lane, and
        // lays their tentative lists end to end (a prefix sum of the list
        // lengths); then every lane takes one position of that concatenation
        // per step and finds the k-mer it belongs to by binary search over the
        // lanes' start positions, so no lane idles while another list is long.
        // Up to kIdxGroups groups of 32 entries load at once.
        for (int c0 = 0; c0 < (ntq > 0 ? ne : 0); c0 += 32 * kIdxGroups) {
            uint32_t vg[kIdxGroups];
#pragma unroll
            for (int g = 0; g < kIdxGroups; g++) {
                const int i = c0 + 32 * g + lane;
                vg[g] = i < ne ? __ldcs(e + i) : 0u;
            }
            if (c0 == 0 && idx + nwarps < n) {
                // the next candidate's list position (its index arrived by now)
                e_nx = R.kmer + R.kmer_off[q_nx];
                ne_nx = R.n_kmer[q_nx];
            }
#pragma unroll
            for (int g = 0; g < kIdxGroups; g++) {
                if (c0 + 32 * g >= ne) break;
                const uint32_t v = vg[g];
                const uint32_t km = v >> 16;
                const uint32_t c = v & 0xffffu;
                const uint32_t s0 = SMEM ? s_off16[km] : s_off32[km];
                const uint32_t sz = c ? (SMEM ? s_off16[km + 1] : s_off32[km + 1]) - s0 : 0u;
                uint32_t incl = sz;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(kFull, incl, d);
                    if (lane >= d) incl += o;
                }
                const uint32_t excl = incl - sz;
                const uint32_t total = __shfl_sync(kFull, incl, 31);
                const uint32_t jbase = s0 - excl;  // posting index = jbase + position
                for (uint32_t base = 0; base < total; base += 32) {
                    const uint32_t p = base + lane;
                    // the last lane whose list starts at or before p owns p
                    int o = 0;
#pragma unroll
                    for (int step = 16; step >= 1; step >>= 1) {
                        const uint32_t x = __shfl_sync(kFull, excl, o + step);
                        if (x <= p) o += step;
                    }
                    const uint32_t j = __shfl_sync(kFull, jbase, o) + p;
                    const uint32_t co = __shfl_sync(kFull, c, o);
                    if (p < total) {
                        uint32_t t, ct;
                        if (SMEM) {
                            const uint32_t pp = s_post16[j];
                            t = pp >> 6;
                            ct = pp & 63u;
                            if (ct == 63u) ct = __ldg(idx_post + j) & 0xffffu;
                        } else {
                            const uint32_t pp = __ldg(idx_post + j);
                            t = pp >> 16;
                            ct = pp & 0xffffu;
                        }
                        // 16-bit halves cannot carry: a sum is at most the
                        // candidate's k-mer count, below 65536
                        if (t < (uint32_t)ntq)
                            atomicAdd(&acc[t >> 1], min(ct, co) << ((t & 1u) << 4));
                    }
                }
            }
        }
        if (!(ntq > 0 && ne > 0) && idx + nwarps < n) {
            e_nx = R.kmer + R.kmer_off[q_nx];
            ne_nx = R.n_kmer[q_nx];
        }
        if (ntq == 0) continue;
        __syncwarp();
        // the tentatives whose sum reaches the cutoff pass the word filter;
        // the composition bound (kernel_preFilter, func.cu:738-754) decides
        // the rest.  The sums are cleared on the way.
        const int cw = R.cut_word[q];
        uint4* a4 = reinterpret_cast<uint4*>(acc);
        const int w4 = (ntq + 7) >> 3;
        for (int i = lane; i < w4; i += 32) {
            const uint4 a = a4[i];
            a4[i] = make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int h = 0; h < 8; h++) {
                const int t = 8 * i + h;
                const int s = (int)((w[h >> 1] >> ((h & 1) << 4)) & 0xffffu);
                if (t < ntq && !(s < cw)) {
                    n_wf++;
                    const int rep = s_tent[t];
                    if (prefilter_pass(R.comp[rep], R.comp[q], R.cut_base[q] - R.strict)) {
                        push_pair(st, pairs, seg_cap, R, rep, q, kBandMaxW);
                        n_al++;
                    }
                }
            }
        }
        __syncwarp();
    }
    // n_pf and bytes are the same in every lane; n_wf and n_al are per lane
    n_wf = (unsigned)warp_sum_i((int)n_wf);
    n_al = (unsigned)warp_sum_i((int)n_al);
    if (lane == 0) {
        if (n_pf) atomicAdd(&st->cnt_prefilter, n_pf);
        if (n_wf) atomicAdd(&st->cnt_word, (unsigned long long)n_wf);
        if (n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
        if (bytes) atomicAdd(&st->filter_bytes, bytes);
    }
}

// ---- word filter by hashed k-mer counts (short reads, sparse k-mer spaces) --
//
// A read's k-mers fall into H buckets by a hash; n(b) is the number of its
// k-mers (with their multiplicities) in bucket b.  Since min(x, y) <= x y for
// counts of at least one,
//     S = sum over k-mers of min(c_t, c_q) <= sum over buckets of n_t n_q,
// an entry of a matrix product again.  A row holds the counts as E2M1 values
// (half the count: 1, 2, 3, 4, 6, 8 and 12 exist), rounded up, and 12 above 8.
// That keeps the bound: where one of the two counts is at most 12 the product
// of the stored ones is at least the smaller count, and where both are above
// it is 144, so that
//     S <= P + min(X_t, X_q),   X = sum over buckets of max(n - 144, 0).
// A pair below its cutoff is rejected; the others go to k_bexact_d, which
// forms S itself.  H is chosen per job (api.cu) so that unrelated reads rarely
// reach the cutoff: P is about L^2 / H for reads of L k-mers.
//
// A CTA keeps the rows of its group of tentatives in shared memory for the
// whole launch (up to 240 x H / 2 bytes) and streams tiles of 128 candidates
// against them: four warps per stage copy rows with cp.async into a ring of
// three 32 KB stages (512 buckets of 128 rows), one warp issues the MMAs, and
// two teams of four warps, one per accumulator, compare the finished tiles' sums
// with the rows' cutoffs while the next tile is summed in the other.
//
// 990k candidates x 1,024 tentatives, H = 1,536: 0.75 ms (1.35e12 pairs/s; the
// masks 1.5 ms); 1M reads of 100-150 bp at t = 0.90 spent 127 ms in the filter
// stage instead of 211, and 108 since k_bexact_d and hash_even_r.  An MMA (64
// buckets) takes N / 2 cycles, and the MMAs alone would take 0.36 ms; the MMA
// thread's wait for a stage adds about 200 cycles that nothing covers (issuing
// blocks while the tensor pipe is busy), so a stage holds eight MMAs.  On the
// way there, average of the first 249 passes (0.39 ms as it is): 16 KB stages
// with eight warps on each 0.43 ms; an arrival per copying thread 0.43; rows by
// TMA gathers of four 1.07 (67 cycles a gather); two warps owning each 16 KB
// stage 0.41; the next stage's wait in the middle of the MMAs 0.43; one team of
// four on the sums 0.43.
constexpr int kHashEpilogue = 8;  // two teams of four, one per accumulator
constexpr int kHashStages = 3;
constexpr int kHashStepBuckets = 512;  // buckets per stage
constexpr int kHashProducers = 4 * kHashStages;  // four warps per stage of the ring
constexpr int kHashThreads = 32 * (1 + kHashEpilogue + kHashProducers);
constexpr int kHashChunkBytes = 128 * kTcRowBytes;  // 256 buckets of 128 rows
constexpr int kHashStageBytes = 2 * kHashChunkBytes;
constexpr int kHashRowBytes = 125 * 1024;  // the tentatives' rows
constexpr int kHashSmem = 1024 + kHashStages * kHashStageBytes + kHashRowBytes + 4 * kMaxBatch;

// Tentatives per group for H buckets.
__host__ __device__ __forceinline__ int hash_group(int buckets) {
    const int n = (kHashRowBytes / (buckets / 2)) & ~15;
    return n < kTcMaxN ? n : kTcMaxN;
}

// The largest number of tentatives, within 1/16 of r_max, whose groups are all
// full and leave the fewest of the device's SMs without one; 0: r_max itself.
// (r_max 1,024 in groups of at most 160: seven groups padded to 1,120, on 147
// of 152 SMs; 960: six on 150.)
int hash_even_r(int buckets, int r_max) {
    const int gmax = hash_group(buckets), sms = num_sms();
    int best = 0, used = 0;
    for (int g = r_max / gmax; g > 0 && 16 * g * gmax >= 15 * r_max; g--)
        if (g * (sms / g) > used) best = g * gmax, used = g * (sms / g);
    return best < r_max ? best : 0;
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool fill) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem),
                 "r"(fill ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__global__ void __launch_bounds__(kHashThreads, 1) k_bfilter_hash(
    DevReads R, RoundState* st, const int32_t* __restrict__ remain,
    const int32_t* __restrict__ tent, Pair* amb, int amb_cap) {
    extern __shared__ __align__(1024) uint8_t hsm_raw[];
    __shared__ uint64_t full[kHashStages], empty[kHashStages], tfull[2], tempty[2], drain;
    __shared__ uint32_t s_tmem;
    __shared__ int s_quit;
    chain_wait();
    if (st->done) return;
    const int nt = st->n_tent;
    if (nt == 0) return;
    const int n = st->n_remain;
    const int gmax = hash_group(R.hbuckets);
    const int groups = (nt + gmax - 1) / gmax;
    const int N = (((nt + groups - 1) / groups) + 15) & ~15;  // tentatives per group
    const int step = max(1, (int)gridDim.x / groups);         // CTAs per group
    const int mtiles = (n + 127) >> 7;
    const int g = blockIdx.x % groups, m0 = blockIdx.x / groups;
    if (m0 >= step || m0 >= mtiles) return;
    const int t0 = g * N, t1 = min(nt, t0 + N);
    const int CH = R.hbuckets / kHashStepBuckets;  // stages per tile
    const int RQ = R.hbuckets >> 5;  // 16-byte pieces of a row
    uint8_t* ring = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(hsm_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* brow = ring + kHashStages * kHashStageBytes;
    int32_t* s_tent = reinterpret_cast<int32_t*>(brow + kHashRowBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kHashStages; i++) {
            mbar_init(&full[i], kHashProducers / kHashStages + never_full());
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], kHashEpilogue / 2);
        }
        mbar_init(&drain, 1);
        s_quit = 0;
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc_all(&s_tmem);
    for (int t = threadIdx.x; t < nt; t += blockDim.x) s_tent[t] = tent[t];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (warp >= 1 && warp <= 4) tc_fill_scales(tmem, warp);
    // the group's rows, chunk by chunk of 256 buckets (rows past the last
    // tentative: read 0, whose sums are not looked at)
    for (int i = threadIdx.x; i < N * RQ; i += blockDim.x) {
        const int r = i / RQ, x = i - r * RQ, c = x >> 3, p = x & 7;
        const int read = t0 + r < nt ? s_tent[t0 + r] : 0;
        cp_async16(brow + (c * N + r) * kTcRowBytes + ((p ^ (r & 7)) << 4),
                   R.hrow + (size_t)read * RQ + x, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const int limit = max(c_spin_limit, 1);
    bool ok = true;  // this warp's waits all ended
    if (warp == 0) {
        if (lane == 0) {
            const uint32_t idesc = tc_idesc_fp4(N);
            const uint32_t a0 = tc_desc_lo(smem_u32(ring)), b0 = tc_desc_lo(smem_u32(brow));
            int s = 0, it = 0;
            uint32_t ph = 0;
            for (int m = m0; ok && m < mtiles; m += step, it++) {
                const int buf = it & 1;
                // (the first use of each accumulator passes at once)
                ok = mbar_wait(&tempty[buf], ((it >> 1) & 1) ^ 1, limit, &s_quit);
                for (int c = 0; ok && c < CH; c++) {
                    ok = mbar_wait(&full[s], ph, limit, &s_quit);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = a0 + s * (kHashStageBytes / 16);
                    const uint32_t b = b0 + 2 * c * N * (kTcRowBytes / 16);
                    tc_mma_stage(tmem + buf * kTcMaxN, tmem, a, b, idesc, c == 0);
                    tc_mma_stage(tmem + buf * kTcMaxN, tmem, a + kHashChunkBytes / 16,
                                 b + N * (kTcRowBytes / 16), idesc, false);
                    tc_commit(&empty[s]);
                    if (++s == kHashStages) s = 0, ph ^= 1;
                }
                if (ok) tc_commit(&tfull[buf]);
            }
        }
    } else if (warp <= kHashEpilogue) {
        const int row = (warp & 3) * 32 + lane, buf = (warp - 1) >> 2;
        unsigned n_wf = 0;
        unsigned long long n_pf = 0, bytes = 0;
        uint32_t ph = 0;
        const int first = m0 + buf * step;
        int q = first * 128 + row < n ? remain[first * 128 + row] : -1;
        int cw = q >= 0 ? R.cut_word[q] : 0, exq = q >= 0 ? R.hextra[q] : 0;
        for (int m = first; m < mtiles; m += 2 * step, ph ^= 1) {
            // this team's next row while its tile is summed
            const int nidx = (m + 2 * step) * 128 + row;
            const int nq = nidx < n ? remain[nidx] : -1;
            ok = mbar_wait_warp(&tfull[buf], ph, limit, &s_quit);
            if (!ok) break;
            tc_fence_after();
            const int ncw = nq >= 0 ? R.cut_word[nq] : 0, nexq = nq >= 0 ? R.hextra[nq] : 0;
            // tentatives of the group before q (the list ascends)
            int ntq = t1;
            if (q <= s_tent[t1 - 1]) {
                int lo = t0, hi = t1;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s_tent[mid] < q) lo = mid + 1;
                    else hi = mid;
                }
                ntq = lo;
            }
            if (q >= 0) {
                n_pf += (unsigned)(ntq - t0);
                if (g == 0) bytes += kCandFixedBytes + 16ull * RQ;  // once per launch
            }
            __syncwarp();
            // the row's cutoff in the accumulator's quarters; no pair of a row
            // without a candidate reaches it
            const float thr = q >= 0 && ntq > t0 ? 0.25f * (float)(cw - exq) : 3.0e38f;
            const uint32_t addr = tmem + ((uint32_t)(warp & 3) << 21) + buf * kTcMaxN;
            auto columns = [&](const float (&v)[16], int c0) {
                float top = v[0];
#pragma unroll
                for (int j = 1; j < 16; j++) top = fmaxf(top, v[j]);
                if (top >= thr) {
                    uint32_t hit = 0;
#pragma unroll
                    for (int j = 0; j < 16; j++) hit |= v[j] >= thr ? 1u << j : 0u;
                    if (c0 + 16 > ntq) hit &= ntq > c0 ? (1u << (ntq - c0)) - 1u : 0u;
                    const int4 cq = R.comp[q];
                    const int cbq = R.cut_base[q] - R.strict;
                    while (hit) {
                        const int j = __ffs(hit) - 1;
                        hit &= hit - 1;
                        const int rep = s_tent[c0 + j];
                        if (exq > 0) {
                            float vj = v[0];
#pragma unroll
                            for (int i = 1; i < 16; i++) vj = j == i ? v[i] : vj;
                            if (4.0f * vj + (float)min(R.hextra[rep], exq) < (float)cw) continue;
                        }
                        n_wf++;
                        // the composition bound (kernel_preFilter, func.cu:738-754)
                        if (!prefilter_pass(R.comp[rep], cq, cbq)) continue;
                        const int slot = atomicAdd(&st->n_amb, 1);
                        if (slot < amb_cap) amb[slot] = Pair{rep, q};
                        else st->pair_overflow = 1;
                    }
                }
                __syncwarp();
            };
            // sixteen columns at a time, the next sixteen on their way
            uint32_t ra[16], rb[16];
            float v[16];
            tc_load16(ra, addr);
            for (int c0 = t0; c0 < t1; c0 += 32) {
                tc_load_wait(ra, v);
                if (c0 + 16 < t1) tc_load16(rb, addr + (c0 + 16 - t0));
                columns(v, c0);
                if (c0 + 16 >= t1) break;
                tc_load_wait(rb, v);
                if (c0 + 32 < t1) tc_load16(ra, addr + (c0 + 32 - t0));
                columns(v, c0 + 16);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[buf]);
            q = nq;
            cw = ncw;
            exq = nexq;
        }
        n_wf = (unsigned)warp_sum_i((int)n_wf);
        n_pf = warp_sum_ull(n_pf);
        bytes = warp_sum_ull(bytes);
        if (lane == 0) {
            if (n_pf) atomicAdd(&st->cnt_prefilter, n_pf);
            if (n_wf) atomicAdd(&st->cnt_word, (unsigned long long)n_wf);
            if (bytes) atomicAdd(&st->filter_bytes, bytes);
        }
    } else {
        // producers: a warp owns a quarter of the rows of one stage of the
        // ring, so the stages' copies run independently and a stage is handed
        // over the moment its own have landed.  Lane piece p of rows 4 k + lane
        // / 8 of the quarter, both chunks.
        const int w = warp - 1 - kHashEpilogue;
        const int s = w % kHashStages, quarter = w / kHashStages;
        const int p = lane & 7, r0 = quarter * 32 + (lane >> 3);
        const int off0 = r0 * kTcRowBytes + ((p ^ (r0 & 7)) << 4);
        const int odd = ((p ^ ((r0 + 4) & 7)) << 4) - ((p ^ (r0 & 7)) << 4);
        uint8_t* d = ring + s * kHashStageBytes + off0;
        const int total = (mtiles - m0 + step - 1) / step * CH;
        constexpr int KR = 8;  // rows per lane: 32, four at a time
        int idx[KR];
        auto rows_of = [&](int i) {
            const int m = m0 + i / CH * step;
#pragma unroll
            for (int k = 0; k < KR; k++) {
                const int x = m * 128 + r0 + 4 * k;
                idx[k] = i < total && x < n ? remain[x] : 0;
            }
        };
        rows_of(s);
        uint32_t ph = 1;  // the first round of stages is free
        for (int i = s; i < total; i += kHashStages, ph ^= 1) {
            ok = mbar_wait_warp(&empty[s], ph, limit, &s_quit);
            if (!ok) break;
            const uint4* src = R.hrow + 16 * (i % CH) + p;
#pragma unroll
            for (int k = 0; k < KR; k++) {
                const uint4* r = src + (size_t)idx[k] * RQ;
                uint8_t* to = d + 4 * k * kTcRowBytes + (k & 1 ? odd : 0);
                cp_async16(to, r, true);
                cp_async16(to + kHashChunkBytes, r + 8, true);
            }
            cp_async_commit();
            rows_of(i + kHashStages);
            cp_async_wait<0>();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    }
    if (!ok) {
        // a wait gave up: the others stop at their next poll
        s_quit = 1;
        st->error = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        if (s_quit && lane == 0 && !never_full()) {
            // the MMAs in flight, before the accumulators are given back
            const int none = 0;
            tc_commit(&drain);
            mbar_wait(&drain, 0, kDrainLimit, &none);
        }
        __syncwarp();
        tmem_free_all(tmem);
    }
}

// ---- word filter by tentative masks (short reads, sparse k-mer spaces) ----
//
// Per pass, for every k-mer m a row of R_max bits, bit t set iff tentative t
// holds m with a non-zero count (k_bmask; 2 MB for k = 7 and R_max 1024, held
// in L2).  A group of lanes per candidate (eight lanes of 16 bytes hold a row
// of 1,024 tentatives; four candidates per warp) copies the rows of the
// candidate's k-mers into shared memory and counts per tentative the rows
// that have its bit:
//     D1 = sum over k-mers of [c_t >= 1][c_q >= 1],
// in bit-sliced counters (plane b holds bit b of 32 tentatives' counts) that
// carry-save adders fill.  Since min(c_t, c_q) = [both >= 1] + (min - 1),
//     D1 <= S <= D1 + min(E_t, E_q),   E = sum over k-mers of (count - 1),
// so D1 >= cutoff passes a pair and D1 + min(E_t, E_q) < cutoff rejects it;
// the pairs between go to k_bexact_t, which forms S itself.  Per pair the
// kernel reads one bit per candidate k-mer and spends about three logic
// instructions per 32 pairs and k-mer, where the index form takes a warp
// step per posting of every shared k-mer.  A count never exceeds the
// candidate's k-mer entries: eight planes hold it where every read has at
// most kMaskEntries8 entries, ten up to kMaskMaxEntries (the form's limit).

constexpr int kMaskThreads = 256;

// One warp per tentative: sets the tentative's bit in the rows of its k-mers
// (the rows were zeroed before) and writes its excess E_t.
__global__ void __launch_bounds__(256) k_bmask(DevReads R, RoundState* st,
                                               const int32_t* __restrict__ tent, uint32_t* tmask,
                                               int32_t* tex, int rwq) {
    if (st->done || st->n_tent == 0) return;
    const int nt = st->n_tent;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const size_t row_words = 4 * (size_t)rwq;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += nw) {
        const int rep = tent[t];
        const uint32_t* e = R.kmer + R.kmer_off[rep];
        const int ne = R.n_kmer[rep];
        const uint32_t bit = 1u << (t & 31);
        int ex = 0;
        for (int i = lane; i < ne; i += 32) {
            const uint32_t v = __ldg(e + i);
            const uint32_t c = v & 0xffffu;
            if (c) {
                atomicOr(tmask + (v >> 16) * row_words + (t >> 5), bit);
                ex += (int)c - 1;
            }
        }
        ex = warp_sum_i(ex);
        if (lane == 0) tex[t] = ex;
    }
}

// p += w0 + .. + w7, bit-sliced (NP planes, counts below 2^NP), in two parts:
// a Harley-Seal tree of carry-save adders into the planes of weight 1, 2 and
// 4 that returns the carry of weight 8, and bs_carry, which adds a carry
// into the planes from `from` up.  Two trees' carries meet in one more adder
// first (bs_pair8), so the ripple runs once per 16 words.
template <int NP>
__device__ __forceinline__ uint32_t bs_tree8(uint32_t (&p)[NP], uint32_t w0, uint32_t w1,
                                             uint32_t w2, uint32_t w3, uint32_t w4, uint32_t w5,
                                             uint32_t w6, uint32_t w7) {
    uint32_t t1, t2, t3, t4, f1, f2, e8;
    csa(p[0], t1, p[0], w0, w1);
    csa(p[0], t2, p[0], w2, w3);
    csa(p[1], f1, p[1], t1, t2);
    csa(p[0], t3, p[0], w4, w5);
    csa(p[0], t4, p[0], w6, w7);
    csa(p[1], f2, p[1], t3, t4);
    csa(p[2], e8, p[2], f1, f2);
    return e8;
}
template <int NP>
__device__ __forceinline__ void bs_carry(uint32_t (&p)[NP], int from, uint32_t c) {
#pragma unroll
    for (int b = 0; b < NP; b++) {
        if (b < from) continue;
        const uint32_t t = p[b] & c;
        p[b] ^= c;
        c = t;
    }
}
// Two weight-8 carries: one adder into plane 3, its weight-16 carry rippled.
template <int NP>
__device__ __forceinline__ void bs_pair8(uint32_t (&p)[NP], uint32_t a8, uint32_t b8) {
    uint32_t c16;
    csa(p[3], c16, p[3], a8, b8);
    bs_carry<NP>(p, 4, c16);
}

// Bits of the counts >= v.
template <int NP>
__device__ __forceinline__ uint32_t bs_ge(const uint32_t (&p)[NP], int v) {
    if (v <= 0) return 0xffffffffu;
    if (v > (1 << NP) - 1) return 0u;
    uint32_t gt = 0, eq = 0xffffffffu;
#pragma unroll
    for (int b = NP - 1; b >= 0; b--) {
        const uint32_t vb = ((v >> b) & 1) ? 0xffffffffu : 0u;
        gt |= eq & p[b] & ~vb;
        eq &= ~(p[b] ^ vb);
    }
    return gt | eq;
}

template <int NP>
__device__ __forceinline__ int bs_get(const uint32_t (&p)[NP], int bit) {
    int v = 0;
#pragma unroll
    for (int b = 0; b < NP; b++) v |= (int)((p[b] >> bit) & 1u) << b;
    return v;
}

struct MaskCounts {
    unsigned long long n_pf = 0, bytes = 0;
    unsigned n_wf = 0, n_al = 0;
};

// Rows stream through shared memory with cp.async, kMaskStages steps deep:
// each lane copies its own 16-byte words and reads back only those, so no
// warp barrier is needed (the kernel is bound by L2 latency, and the copies
// in flight hold no registers).
constexpr int kMaskStages = 3;
constexpr int kMaskStepBytes = 8 * 32 * 16;  // one step: 8 words of 16 bytes per lane

// Rows of 16-byte words: lane (g, x) of a warp, g = lane / LPR, x = lane %
// LPR, works for candidate g of the warp's 32 / LPR consecutive candidates
// (consecutive in the remain list, so of similar length) and holds the counts
// of word x of the rows (tentatives 128 x .. 128 x + 127).  Each step a group
// copies the rows of 8 of its candidate's k-mers; a step's entries load two
// issues before its copies, and the copies kMaskStages - 1 steps before their
// counts.
template <int LPR, int NP>
__device__ __forceinline__ void mask_candidates(const DevReads& R, RoundState* st,
                                                const int32_t* __restrict__ remain,
                                                const int32_t* s_tent, uint4* stage, int nt,
                                                int n, const uint4* __restrict__ tm4, int rwq,
                                                const int32_t* __restrict__ tex, Pair* pairs,
                                                int seg_cap, Pair* amb, int amb_cap,
                                                MaskCounts& mc) {
    constexpr int G = 32 / LPR;   // candidates per warp
    constexpr int EPL = 8 / LPR;  // entries a lane loads per step
    const int lane = threadIdx.x & 31;
    const int g = lane / LPR, x = lane % LPR;
    const bool xin = x < ((nt + 127) >> 7);
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int stride = nwarps * G;
    // software pipeline over the warp's candidate sets: the read index of the
    // set after next and the list position of the next load while this set
    // is counted
    auto read_at = [&](int i) { return i < n ? remain[i] : -1; };
    int q1 = read_at(wid * G + g);
    int q2 = read_at(wid * G + stride + g);
    int64_t off1 = q1 >= 0 ? R.kmer_off[q1] : 0;
    int nk1 = q1 >= 0 ? R.n_kmer[q1] : 0;
    for (int base = wid * G; base < n; base += stride) {
        const int q = q1;
        const int64_t off = off1;
        const int nk = nk1;
        q1 = q2;
        q2 = read_at(base + 2 * stride + g);
        // tentatives before q: the first ntq of the ascending list
        int ntq = 0;
        if (q >= 0) {
            int lo = 0, hi = nt;
            if (s_tent[nt - 1] < q) lo = nt;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_tent[mid] < q) lo = mid + 1;
                else hi = mid;
            }
            ntq = lo;
        }
        const int ne = ntq > 0 ? nk : 0;
        const uint32_t* e = R.kmer + (ntq > 0 ? off : 0);
        if (x == 0) {
            mc.n_pf += ntq;
            if (ntq > 0) mc.bytes += kCandFixedBytes + 4ull * (unsigned)ne;
        }
        const int nsteps = __reduce_max_sync(kFull, (ne + 7) >> 3);
        if (nsteps == 0) {
            off1 = q1 >= 0 ? R.kmer_off[q1] : 0;
            nk1 = q1 >= 0 ? R.n_kmer[q1] : 0;
            continue;
        }
        // entries [8 j + EPL x, + EPL) of the candidate (the lists are padded
        // to 16 bytes, with slack after the last: whole vectors load).  They
        // stream from HBM, so they load two issues ahead of their copies.
        auto load_raw = [&](int j, uint32_t (&en)[EPL]) {
            const int i0 = 8 * j + EPL * x;
#pragma unroll
            for (int k = 0; k < EPL; k++) en[k] = 0u;
            if (i0 < ne) {
                if constexpr (EPL == 1) {
                    en[0] = __ldcs(e + i0);
                } else if constexpr (EPL == 2) {
                    const uint2 v = __ldcs(reinterpret_cast<const uint2*>(e + i0));
                    en[0] = v.x, en[1] = v.y;
                } else {
#pragma unroll
                    for (int k = 0; k < EPL; k += 4) {
                        const uint4 v = __ldcs(reinterpret_cast<const uint4*>(e + i0 + k));
                        en[k] = v.x, en[k + 1] = v.y, en[k + 2] = v.z, en[k + 3] = v.w;
                    }
                }
            }
        };
        int ex = 0;
        // stage buffers in turn: copies of step j go to `wr`, counts of step
        // s read `rd`
        uint4* const st0 = stage + lane;
        constexpr int SB = kMaskStepBytes / 16;
        int wr = 0, rd = 0;
        // step j: slot u of stage wr gets word x of the row of entry 8 j + u
        // (a row index of -1: no row, count 0 or past the list)
        auto issue = [&](int j, const uint32_t (&en)[EPL]) {
            int rb[EPL];
#pragma unroll
            for (int k = 0; k < EPL; k++) {
                const int c = 8 * j + EPL * x + k < ne ? (int)(en[k] & 0xffffu) : 0;
                ex += c > 0 ? c - 1 : 0;
                rb[k] = c > 0 ? (int)(en[k] >> 16) * rwq : -1;
            }
            uint4* dst = st0 + wr * SB;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int r = EPL == 8 ? rb[u % EPL]
                                       : __shfl_sync(kFull, rb[u % EPL], g * LPR + u / EPL);
                const bool ok = xin && r >= 0;
                cp_async16(dst + 32 * u, tm4 + (ok ? r + x : 0), ok);
            }
            wr = wr == kMaskStages - 1 ? 0 : wr + 1;
        };
        uint32_t P[4][NP];
#pragma unroll
        for (int w = 0; w < 4; w++)
#pragma unroll
            for (int b = 0; b < NP; b++) P[w][b] = 0u;
        uint32_t c8[4] = {0u, 0u, 0u, 0u};  // weight-8 carries of an odd step
        uint32_t en0[EPL], en1[EPL];        // entries of the next two steps to issue
        load_raw(0, en0);
        load_raw(1, en1);
        int nexti = 0;  // next step to issue
        auto issue_next = [&]() {
            issue(nexti, en0);
#pragma unroll
            for (int k = 0; k < EPL; k++) en0[k] = en1[k];
            load_raw(nexti + 2, en1);
            nexti++;
        };
#pragma unroll
        for (int j = 0; j < kMaskStages - 1; j++) {
            if (j < nsteps) issue_next();
            cp_async_commit();
        }
        off1 = q1 >= 0 ? R.kmer_off[q1] : 0;
        nk1 = q1 >= 0 ? R.n_kmer[q1] : 0;
        for (int s = 0; s < nsteps; s++) {
            if (s + kMaskStages - 1 < nsteps) issue_next();
            cp_async_commit();
            cp_async_wait<kMaskStages - 1>();  // this lane's copies of step s
            const uint4* src = st0 + rd * SB;
            rd = rd == kMaskStages - 1 ? 0 : rd + 1;
            uint4 w[8];
#pragma unroll
            for (int u = 0; u < 8; u++) w[u] = src[32 * u];
            const uint32_t e0 = bs_tree8<NP>(P[0], w[0].x, w[1].x, w[2].x, w[3].x, w[4].x, w[5].x, w[6].x, w[7].x);
            const uint32_t e1 = bs_tree8<NP>(P[1], w[0].y, w[1].y, w[2].y, w[3].y, w[4].y, w[5].y, w[6].y, w[7].y);
            const uint32_t e2 = bs_tree8<NP>(P[2], w[0].z, w[1].z, w[2].z, w[3].z, w[4].z, w[5].z, w[6].z, w[7].z);
            const uint32_t e3 = bs_tree8<NP>(P[3], w[0].w, w[1].w, w[2].w, w[3].w, w[4].w, w[5].w, w[6].w, w[7].w);
            if (s & 1) {
                bs_pair8<NP>(P[0], c8[0], e0);
                bs_pair8<NP>(P[1], c8[1], e1);
                bs_pair8<NP>(P[2], c8[2], e2);
                bs_pair8<NP>(P[3], c8[3], e3);
            } else {
                c8[0] = e0, c8[1] = e1, c8[2] = e2, c8[3] = e3;
            }
        }
        if (nsteps & 1) {
#pragma unroll
            for (int w = 0; w < 4; w++) bs_carry<NP>(P[w], 3, c8[w]);
        }
        // E_q over the group's lanes
#pragma unroll
        for (int off = 1; off < LPR; off <<= 1) ex += __shfl_xor_sync(kFull, ex, off);
        if (ntq == 0 || !xin) continue;
        const int cw = R.cut_word[q];
        // counts >= v need a bit at or above plane floor(log2 v): most words
        // have none and skip the comparisons
        const int vlo = cw - ex;
        const int lb = vlo > 0 ? 31 - __clz(vlo) : 0;
        int4 cq = make_int4(0, 0, 0, 0);
        int cbq = 0;
        bool have_cq = false;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int t0 = 32 * (4 * x + w);
            if (t0 >= ntq) break;
            const uint32_t valid = ntq - t0 >= 32 ? 0xffffffffu : (1u << (ntq - t0)) - 1u;
            uint32_t hiw = 0u;
#pragma unroll
            for (int b = 0; b < NP; b++)
                if (b >= lb) hiw |= P[w][b];
            if (vlo > (1 << NP) - 1 || !((vlo <= 0 ? 0xffffffffu : hiw) & valid)) continue;
            uint32_t pass = bs_ge<NP>(P[w], cw) & valid;
            uint32_t open = bs_ge<NP>(P[w], vlo) & valid & ~pass;
            if (!(pass | open)) continue;
            if (!have_cq) {
                cq = R.comp[q];
                cbq = R.cut_base[q] - R.strict;
                have_cq = true;
            }
            while (pass) {
                const int t = t0 + __ffs(pass) - 1;
                pass &= pass - 1;
                mc.n_wf++;
                const int rep = s_tent[t];
                // the composition bound (kernel_preFilter, func.cu:738-754)
                if (prefilter_pass(R.comp[rep], cq, cbq)) {
                    push_pair(st, pairs, seg_cap, R, rep, q, kBandMaxW);
                    mc.n_al++;
                }
            }
            while (open) {
                const int b = __ffs(open) - 1;
                open &= open - 1;
                const int t = t0 + b;
                if (bs_get<NP>(P[w], b) + min(tex[t], ex) < cw) continue;
                mc.n_wf++;
                const int rep = s_tent[t];
                if (prefilter_pass(R.comp[rep], cq, cbq)) {
                    const int slot = atomicAdd(&st->n_amb, 1);
                    if (slot < amb_cap) amb[slot] = Pair{rep, q};
                    else st->pair_overflow = 1;
                }
            }
        }
    }
    cp_async_wait<0>();
}

constexpr int kMaskSmem = (kMaskThreads / 32) * kMaskStages * kMaskStepBytes;

template <int NP>
__global__ void __launch_bounds__(kMaskThreads, 2) k_bfilter_mask(
    DevReads R, RoundState* st, const int32_t* __restrict__ remain,
    const int32_t* __restrict__ tent, const uint4* __restrict__ tm4, int rwq,
    const int32_t* __restrict__ tex, Pair* pairs, int seg_cap, Pair* amb, int amb_cap) {
    __shared__ int32_t s_tent[kMaxBatch];
    extern __shared__ __align__(16) uint4 mstage[];
    if (st->done || st->n_tent == 0) return;
    const int nt = st->n_tent;
    const int n = st->n_remain;
    for (int i = threadIdx.x; i < nt; i += blockDim.x) s_tent[i] = tent[i];
    __syncthreads();
    uint4* stage = mstage + (threadIdx.x >> 5) * kMaskStages * (kMaskStepBytes / 16);
    MaskCounts mc;
    const int quads = (nt + 127) >> 7;  // 16-byte words of the pass's rows
    if (quads > 4)
        mask_candidates<8, NP>(R, st, remain, s_tent, stage, nt, n, tm4, rwq, tex, pairs, seg_cap,
                           amb, amb_cap, mc);
    else if (quads > 2)
        mask_candidates<4, NP>(R, st, remain, s_tent, stage, nt, n, tm4, rwq, tex, pairs, seg_cap,
                           amb, amb_cap, mc);
    else if (quads > 1)
        mask_candidates<2, NP>(R, st, remain, s_tent, stage, nt, n, tm4, rwq, tex, pairs, seg_cap,
                           amb, amb_cap, mc);
    else
        mask_candidates<1, NP>(R, st, remain, s_tent, stage, nt, n, tm4, rwq, tex, pairs, seg_cap,
                           amb, amb_cap, mc);
    const unsigned n_wf = (unsigned)warp_sum_i((int)mc.n_wf);
    const unsigned n_al = (unsigned)warp_sum_i((int)mc.n_al);
    mc.n_pf = warp_sum_ull(mc.n_pf);
    mc.bytes = warp_sum_ull(mc.bytes);
    if ((threadIdx.x & 31) == 0) {
        if (mc.n_pf) atomicAdd(&st->cnt_prefilter, mc.n_pf);
        if (n_wf) atomicAdd(&st->cnt_word, (unsigned long long)n_wf);
        if (n_al) atomicAdd(&st->cnt_aligned, (unsigned long long)n_al);
        if (mc.bytes) atomicAdd(&st->filter_bytes, mc.bytes);
    }
}

// Survival of the tentatives in greedy order (a tentative survives iff no
// surviving earlier tentative accepted it), then the claims: the first
// surviving tentative of each accepted candidate, by keyed atomicMax.
//
// Row i of tt holds the tentatives that accepted tentative i (all before it).
// Thread i decides tentative i: claimed once one of them survives, a survivor
// once all of them are claimed.  Each step decides at least the first open
// tentative, and in practice nearly all within a few steps, where one warp
// going through the rows in order took 40 us a pass.  Every block repeats
// this (the rows are in L2) instead of waiting for a launch that does it once.
__global__ void __launch_bounds__(kMaxBatch) k_bclaim(RoundState* st, const int32_t* __restrict__ tent,
                                                      const uint32_t* __restrict__ tt,
                                                      const uint32_t* __restrict__ ttrow,
                                                      const Pair* __restrict__ acc,
                                                      const uint32_t* __restrict__ tidx,
                                                      uint32_t* best, int32_t* cluster) {
    __shared__ __align__(16) uint32_t surv[kTTWords], open[kTTWords];
    chain_wait();
    if (st->done || st->n_tent == 0 || st->pair_overflow || st->acc_overflow) return;
    const int nt = st->n_tent;
    const int na = st->n_acc;
    // (a block without claims leaves them to the others; block 0 marks the survivors)
    if (blockIdx.x > 0 && (long long)blockIdx.x * kMaxBatch >= na) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = threadIdx.x;
    const uint32_t flagged = ttrow[warp];
    bool undecided = i < nt && ((flagged >> lane) & 1u);
    bool alive = i < nt && !undecided;
    uint4 row[kTTWords / 4];
    if (undecided) {
#pragma unroll
        for (int w = 0; w < kTTWords / 4; w++)
            row[w] = reinterpret_cast<const uint4*>(tt)[(size_t)i * (kTTWords / 4) + w];
    }
    while (true) {
        const unsigned ms = __ballot_sync(kFull, alive), mo = __ballot_sync(kFull, undecided);
        if (lane == 0) surv[warp] = ms, open[warp] = mo;
        if (!__syncthreads_or((int)mo)) break;
        if (undecided) {
            uint32_t by_surv = 0, by_open = 0;
#pragma unroll
            for (int w = 0; w < kTTWords / 4; w++) {
                const uint4 s4 = reinterpret_cast<const uint4*>(surv)[w];
                const uint4 o4 = reinterpret_cast<const uint4*>(open)[w];
                by_surv |= (row[w].x & s4.x) | (row[w].y & s4.y) | (row[w].z & s4.z) | (row[w].w & s4.w);
                by_open |= (row[w].x & o4.x) | (row[w].y & o4.y) | (row[w].z & o4.z) | (row[w].w & o4.w);
            }
            if (by_surv) undecided = false;
            else if (!by_open) undecided = false, alive = true;
        }
        __syncthreads();
    }
    if (blockIdx.x == 0) {
        if (alive) cluster[tent[i]] = tent[i];
        const int count = __syncthreads_count(alive);
        if (threadIdx.x == 0) {
            st->survivors = count;
            st->rounds += count;
        }
    }
    const uint32_t pass = (uint32_t)st->pass;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < na; k += gridDim.x * blockDim.x) {
        const Pair p = acc[k];
        const int t = tidx[p.rep] & 0xfff;
        if ((surv[t >> 5] >> (t & 31)) & 1u) atomicMax(&best[p.cand], (pass << 12) | (4095u - t));
    }
}

__global__ void k_init(RoundState* st, int32_t* cluster, int32_t* remain, uint32_t* tidx,
                       uint32_t* best, int n, int batched, int r_max, int pass_limit,
                       int* align_work) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        if (batched) {
            cluster[i] = -1;
            remain[i] = i;
            tidx[i] = 0xffffffffu;
            best[i] = 0u;
        } else {
            cluster[i] = i == 0 ? 0 : -1;
            if (i > 0) remain[i - 1] = i;
        }
    }
    if (i == 0) {
        RoundState s = {};
        s.rep = 0;
        s.n_remain = batched ? n : n - 1;
        s.next_min = 0x7fffffff;
        s.done = n <= 0 ? 1 : 0;
        s.pass = 1;
        // as many tentatives as leave the device idle in any case (kFewPairs)
        s.R = min(r_max, max(1, kFewPairs / max(n, 1)));
        s.R_max = r_max;
        s.pass_limit = pass_limit;
        *st = s;
        for (int c = 0; c <= kSingleWorkSlot; c++) align_work[c] = 0;
    }
}

// Resume from a checkpoint: cluster[] (already on the device) is the state of
// an unfinished clustering -- every read either unclustered (-1) or joined to
// a representative taken earlier -- which is all the state the reference's
// loop carries between rounds (cluster[] and the next representative, the
// smallest unclustered read; cuda-version/func.cu:1001-1066).  Three steps:
// a fresh round state, the remain list of the unclustered reads (any order:
// every consumer of the list is order-independent) with their smallest index,
// then the next representative (plain) or the tentative cursor (batched).
__global__ void k_resume_state(RoundState* st, int r_max, int pass_limit, int* align_work) {
    RoundState s = {};
    s.rep = -1;
    s.next_min = 0x7fffffff;
    s.pass = 1;
    s.R = 1;
    s.R_max = r_max;
    s.pass_limit = pass_limit;
    *st = s;
    for (int c = 0; c <= kSingleWorkSlot; c++) align_work[c] = 0;
}

__global__ void k_resume_scan(RoundState* st, const int32_t* __restrict__ cluster,
                              int32_t* remain, uint32_t* tidx, uint32_t* best, int n,
                              int batched) {
    const int lane = threadIdx.x & 31;
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int i = base + lane;
        const bool un = i < n && cluster[i] == -1;
        if (batched && i < n) {
            tidx[i] = 0xffffffffu;
            best[i] = 0u;
        }
        const unsigned m = __ballot_sync(kFull, un);
        if (!m) continue;
        int pos = 0;
        if (lane == 0) {
            pos = atomicAdd(&st->n_remain, __popc(m));
            atomicMin(&st->next_min, base + __ffs(m) - 1);
        }
        pos = __shfl_sync(kFull, pos, 0);
        if (un) remain[pos + __popc(m & ((1u << lane) - 1u))] = i;
    }
}

__global__ void k_resume_start(RoundState* st, int32_t* cluster, int batched) {
    if (st->n_remain == 0) {
        st->done = 1;
        return;
    }
    const int first = st->next_min;
    st->next_min = 0x7fffffff;
    if (batched) {
        st->cursor = first;
    } else {
        // the next round's representative; it stays in the remain list, which
        // the plain filter skips, as after every compaction
        cluster[first] = first;
        st->rep = first;
    }
}

// ---------------------------------------------------------------- launchers

// Launch of a kernel that begins with chain_wait; with B.chained behind a
// programmatic edge (not between the events of a timed step, which stand
// between the kernels).
template <class... P, class... A>
void launch_next(const RoundBuffers& B, void (*kernel)(P...), int grid, int threads, int smem,
                 cudaStream_t s, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = B.chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class KernelT>
int grid_for(KernelT kernel, int threads, int smem, int cap_per_sm) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (per_sm < 1) per_sm = 1;
    if (per_sm > cap_per_sm) per_sm = cap_per_sm;
    return num_sms() * per_sm;
}

// The job's block shape: a grid of at most `blocks` CTAs per SM (0: the full
// grid, every CTA that fits).  The kernels loop over their work, so any grid
// size gives the same result.
int shaped(int grid, int blocks) {
    return blocks > 0 ? min(grid, num_sms() * blocks) : grid;
}

// tent: null for a plain round; the batched form's tentatives otherwise (the
// kernel then runs only in a pass with a single tentative).
template <int K, bool DROP, bool LATE>
void launch_filter_t(const DevReads& R, RoundBuffers& B, const int32_t* remain, cudaStream_t s,
                     const int32_t* tent = nullptr) {
    const int smem = DROP ? 0 : (1 << (2 * K)) * 2;
    static int grid = 0;
    if (!grid) {
        if (smem > 0)
            cudaFuncSetAttribute(k_filter<K, DROP, LATE>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        grid = grid_for(k_filter<K, DROP, LATE>, kFilterThreads, smem, 8);
    }
    launch_next(B, k_filter<K, DROP, LATE>, shaped(grid, R.filter_blocks), kFilterThreads, smem, s,
                R, B.st, remain, B.pairs, B.seg_cap, tent);
}

template <int K>
void launch_bfilter_tab_t(const DevReads& R, RoundBuffers& B, const int32_t* remain,
                          cudaStream_t s) {
    // passes with one tentative (the first passes of adaptive R) stream the
    // candidates once against one table: the plain kernel does that at HBM
    // speed, the grouped-table kernel skips them
    launch_filter_t<K, false, false>(R, B, remain, s, B.tent);
    constexpr int smem = TabGroup<K>::smem;
    static int grid = 0;
    if (!grid) {
        cudaFuncSetAttribute(k_bfilter_tab<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        grid = grid_for(k_bfilter_tab<K>, kTabThreads, smem, 2);
    }
    k_bfilter_tab<K><<<shaped(grid, R.filter_blocks), kTabThreads, smem, s>>>(
        R, B.st, remain, B.tent, B.pairs, B.seg_cap);
}

template <int K, bool DROP>
void launch_bfilter_t(const DevReads& R, RoundBuffers& B, const int32_t* remain, cudaStream_t s) {
    if constexpr (!DROP) {
        launch_bfilter_tab_t<K>(R, B, remain, s);
    } else {
        static int grid = 0;
        if (!grid) grid = grid_for(k_bprefilter, kFilterThreads, 0, 8);
        launch_next(B, k_bprefilter, shaped(grid, R.filter_blocks), kFilterThreads, 0, s, R, B.st,
                    remain, B.tent, B.pairs, B.seg_cap);
    }
}

template <int K>
void launch_bfilter_idx_t(const DevReads& R, RoundBuffers& B, const int32_t* remain,
                          cudaStream_t s) {
    const bool in_smem = B.idx_post16 != nullptr;
    const int threads = in_smem ? 1024 : 256;
    const int ismem = (1 << (2 * K)) * 4;
    const int fsmem = IndexSmem(K, B.r_max, B.idx_cap, in_smem).bytes(threads / 32);
    static bool attr = false;
    if (!attr) {
        // the device's largest size, set once: jobs of one process may run
        // concurrently with different index sizes
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaFuncSetAttribute(k_bindex<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, ismem);
        cudaFuncSetAttribute(k_bfilter_idx<K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin);
        cudaFuncSetAttribute(k_bfilter_idx<K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin);
        attr = true;
    }
    k_bindex<K><<<1, kIndexThreads, ismem, s>>>(R, B.st, B.tent, B.idx_off, B.idx_post,
                                                B.idx_off16, B.idx_post16, (long long)B.idx_cap);
    if (in_smem) {
        const int grid = grid_for(k_bfilter_idx<K, true>, threads, fsmem, 2);
        k_bfilter_idx<K, true><<<shaped(grid, R.filter_blocks), threads, fsmem, s>>>(
            R, B.st, remain, B.tent, B.idx_off, B.idx_post, B.idx_off16, B.idx_post16, B.r_max,
            (long long)B.idx_cap, B.pairs, B.seg_cap);
    } else {
        const int grid = grid_for(k_bfilter_idx<K, false>, threads, fsmem, 8);
        k_bfilter_idx<K, false><<<shaped(grid, R.filter_blocks), threads, fsmem, s>>>(
            R, B.st, remain, B.tent, B.idx_off, B.idx_post, nullptr, nullptr, B.r_max,
            (long long)B.idx_cap, B.pairs, B.seg_cap);
    }
}

// The exact sums of the open pairs: the queue sorted by tentative, then one
// table per run.
template <int K>
void launch_exact_t(const DevReads& R, RoundBuffers& B, cudaStream_t s) {
    constexpr int xsmem = (1 << (2 * K)) * 2;
    static int grid = 0;
    if (!grid) {
        cudaFuncSetAttribute(k_bexact_t<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, xsmem);
        grid = grid_for(k_bexact_t<K>, kAmbThreads, xsmem, 8);
    }
    const int ga = num_sms() * 2;
    launch_next(B, k_amb_count, ga, kAmbThreads, 0, s, B.st, B.amb, B.amb_cap, B.tidx, B.amb_idx);
    launch_next(B, k_amb_scan, 1, 1024, 0, s, B.st, B.amb_cap, B.amb_idx);
    launch_next(B, k_amb_place, ga, kAmbThreads, 0, s, B.st, B.amb, B.amb_cap, B.tidx, B.amb_idx,
                B.amb2);
    launch_next(B, k_bexact_t<K>, shaped(grid, R.filter_blocks), kAmbThreads, xsmem, s, R, B.st,
                B.amb2, B.amb_idx, B.amb_cap, B.tent, B.pairs, B.seg_cap);
}

template <int K>
void launch_bfilter_bits_t(const DevReads& R, RoundBuffers& B, const int32_t* remain,
                           cudaStream_t s) {
    // passes with one tentative (the first passes of adaptive R) go to the
    // plain kernel, which streams the candidates against one table
    launch_filter_t<K, false, false>(R, B, remain, s, B.tent);
    static int grid = 0;
    if (!grid) {
        cudaFuncSetAttribute(k_bfilter_bits<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kBitsSmem);
        grid = grid_for(k_bfilter_bits<K>, kBitsThreads, kBitsSmem, 1);
    }
    launch_next(B, k_bfilter_bits<K>, grid, kBitsThreads, kBitsSmem, s, R, B.st, remain, B.tent,
                B.pairs, B.seg_cap, B.amb, B.amb_cap);
    launch_exact_t<K>(R, B, s);
}

void launch_bfilter_hash(const DevReads& R, RoundBuffers& B, const int32_t* remain,
                           cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_bfilter_hash, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kHashSmem);
        cudaFuncSetAttribute(k_bexact_d, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kDirectWarps * kDirectMaxSlots * (int)sizeof(uint32_t));
        attr = true;
    }
    launch_next(B, k_bfilter_hash, num_sms(), kHashThreads, kHashSmem, s, R, B.st, remain, B.tent,
                B.amb, B.amb_cap);
    const int words = std::max(R.hslots, (1 << (2 * R.k)) / 32);  // as direct_words()
    const int smem = kDirectWarps * words * (int)sizeof(uint32_t);
    const int grid = num_sms() * std::min(8, 220 * 1024 / (smem + 1024));
    launch_next(B, k_bexact_d, shaped(grid, R.filter_blocks), 32 * kDirectWarps, smem, s, R, B.st,
                B.amb, B.amb_cap, B.pairs, B.seg_cap);
}

template <int K>
void launch_bfilter_mask_t(const DevReads& R, RoundBuffers& B, const int32_t* remain,
                           cudaStream_t s) {
    static int grid8 = 0, grid10 = 0;
    if (!grid8) {
        cudaFuncSetAttribute(k_bfilter_mask<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMaskSmem);
        cudaFuncSetAttribute(k_bfilter_mask<10>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMaskSmem);
        grid8 = grid_for(k_bfilter_mask<8>, kMaskThreads, kMaskSmem, 2);
        grid10 = grid_for(k_bfilter_mask<10>, kMaskThreads, kMaskSmem, 2);
    }
    cudaMemsetAsync(B.tmask, 0, sizeof(uint4) * ((size_t)1 << (2 * K)) * B.tmask_rwq, s);
    k_bmask<<<kMaxBatch / 8, 256, 0, s>>>(R, B.st, B.tent, reinterpret_cast<uint32_t*>(B.tmask),
                                          B.tmask_ex, B.tmask_rwq);
    // eight count planes where no read has more than 255 k-mer entries, else ten
    if (B.tmask_planes <= 8)
        k_bfilter_mask<8><<<shaped(grid8, R.filter_blocks), kMaskThreads, kMaskSmem, s>>>(
            R, B.st, remain, B.tent, B.tmask, B.tmask_rwq, B.tmask_ex, B.pairs, B.seg_cap, B.amb,
            B.amb_cap);
    else
        k_bfilter_mask<10><<<shaped(grid10, R.filter_blocks), kMaskThreads, kMaskSmem, s>>>(
            R, B.st, remain, B.tent, B.tmask, B.tmask_rwq, B.tmask_ex, B.pairs, B.seg_cap, B.amb,
            B.amb_cap);
    launch_exact_t<K>(R, B, s);
}

template <bool BATCH>
void launch_filter_any(const DevReads& R, RoundBuffers& B, const int32_t* remain, int drop,
                       cudaStream_t s) {
    if (!BATCH && !drop && R.k >= kWideK) {
        static int grid = 0;
        if (!grid) grid = grid_for(k_filter_g, kFilterThreads, 0, 8);
        k_gtab<<<64, 256, 0, s>>>(R, B.st, 0);
        k_filter_g<<<shaped(grid, R.filter_blocks), kFilterThreads, 0, s>>>(
            R, B.st, remain, B.pairs, B.seg_cap);
        k_gtab<<<64, 256, 0, s>>>(R, B.st, 1);
        return;
    }
    if (BATCH && !drop && R.hbuckets) {
        launch_bfilter_hash(R, B, remain, s);
        return;
    }
    if (BATCH && !drop && B.tmask) {
        switch (R.k) {
            case 4: launch_bfilter_mask_t<4>(R, B, remain, s); break;
            case 5: launch_bfilter_mask_t<5>(R, B, remain, s); break;
            case 6: launch_bfilter_mask_t<6>(R, B, remain, s); break;
            default: launch_bfilter_mask_t<7>(R, B, remain, s); break;
        }
        return;
    }
    if (BATCH && !drop && B.amb) {
        switch (R.k) {
            case 4: launch_bfilter_bits_t<4>(R, B, remain, s); break;
            case 5: launch_bfilter_bits_t<5>(R, B, remain, s); break;
            case 6: launch_bfilter_bits_t<6>(R, B, remain, s); break;
            default: launch_bfilter_bits_t<7>(R, B, remain, s); break;
        }
        return;
    }
    if (BATCH && !drop && B.idx_off) {
        switch (R.k) {
            case 4: launch_bfilter_idx_t<4>(R, B, remain, s); break;
            case 5: launch_bfilter_idx_t<5>(R, B, remain, s); break;
            case 6: launch_bfilter_idx_t<6>(R, B, remain, s); break;
            default: launch_bfilter_idx_t<7>(R, B, remain, s); break;
        }
        return;
    }
    if (drop) {
        if (BATCH) launch_bfilter_t<4, true>(R, B, remain, s);
        else launch_filter_t<4, true, true>(R, B, remain, s);
        return;
    }
    switch (R.k) {
        case 4:
            BATCH ? launch_bfilter_t<4, false>(R, B, remain, s) : launch_filter_t<4, false, true>(R, B, remain, s);
            break;
        case 5:
            BATCH ? launch_bfilter_t<5, false>(R, B, remain, s) : launch_filter_t<5, false, true>(R, B, remain, s);
            break;
        case 6:
            BATCH ? launch_bfilter_t<6, false>(R, B, remain, s) : launch_filter_t<6, false, true>(R, B, remain, s);
            break;
        default:
            BATCH ? launch_bfilter_t<7, false>(R, B, remain, s) : launch_filter_t<7, false, true>(R, B, remain, s);
            break;
    }
}

AlignArgs align_args(RoundBuffers& B) {
    AlignArgs A;
    A.pairs = B.pairs;
    A.seg_cap = B.seg_cap;
    A.cluster = B.cluster;
    A.work = reinterpret_cast<int*>(B.st + 1);
    A.tidx = B.tidx;
    A.tt = B.tt;
    A.ttrow = B.ttrow;
    A.acc = B.acc;
    A.acc_cap = B.acc_cap;
    return A;
}

template <int G, int W, bool BATCH>
void launch_align_t(const DevReads& R, RoundBuffers& B, int cls, cudaStream_t s) {
    constexpr int smem = (kAlignThreads / 32) * sys_peq_words(W) * 4;
    static int grid = 0;
    if (!grid) {
        cudaFuncSetAttribute(k_align<G, W, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        grid = grid_for(k_align<G, W, BATCH>, kAlignThreads, smem, 8);
    }
    k_align<G, W, BATCH><<<shaped(grid, R.align_blocks), kAlignThreads, smem, s>>>(
        R, B.st, align_args(B), cls);
}

template <bool BATCH, int MODE>
void launch_seg_t(const DevReads& R, RoundBuffers& B, cudaStream_t s) {
    constexpr int smem = (kAlignThreads / 32) * SegSmem<kSegModeW<MODE>>::kWords * 4;
    static int grid = 0;
    if (!grid) {
        cudaFuncSetAttribute(k_seg<BATCH, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        grid = grid_for(k_seg<BATCH, MODE>, kAlignThreads, smem, 8);
    }
    launch_next(B, k_seg<BATCH, MODE>, shaped(grid, R.align_blocks), kAlignThreads, smem, s, R,
                B.st, align_args(B));
}

template <bool BATCH>
void launch_band_t(const DevReads& R, RoundBuffers& B, cudaStream_t s) {
    static int grid = 0;
    if (!grid) grid = grid_for(k_band<BATCH>, kAlignThreads, 0, 8);
    launch_next(B, k_band<BATCH>, shaped(grid, R.align_blocks), kAlignThreads, 0, s, R, B.st,
                align_args(B));
}

template <bool BATCH>
void launch_align_long_t(const DevReads& R, RoundBuffers& B, cudaStream_t s) {
    constexpr int smem = (kAlignThreads / 32) * sys_peq_words(8) * 4;
    static bool set = false;
    if (!set) {
        cudaFuncSetAttribute(k_align_long<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem);
        set = true;
    }
    k_align_long<BATCH><<<num_sms(), kAlignThreads, smem, s>>>(R, B.st, align_args(B),
                                                               B.long_carry, B.long_words);
}

// Kernels launch_align_classes launches.
template <bool BATCH>
int align_launches(const DevReads& R, const RoundBuffers& B) {
    return (BATCH ? 1 : 0) +
           (R.group_max_w > 0 ? (BATCH ? 2 : 1) + (R.wide ? 1 : 0) : 0) +
           (R.wide == 2 ? (BATCH ? 4 : 7) + (B.long_carry ? 1 : 0) : 0);
}

template <bool BATCH>
void launch_align_classes(const DevReads& R, RoundBuffers& B, cudaStream_t s) {
    if constexpr (BATCH) {
        launch_band_t<BATCH>(R, B, s);
    }
    if (R.group_max_w > 0) {
        if constexpr (BATCH) {
            launch_seg_t<BATCH, kSegNarrow>(R, B, s);
            if (R.wide) launch_seg_t<BATCH, kSegWide>(R, B, s);  // the longest work first
            launch_seg_t<BATCH, kSegFull>(R, B, s);
        } else {
            launch_seg_t<BATCH, kSegFull>(R, B, s);  // and the narrow runs
            if (R.wide) launch_seg_t<BATCH, kSegWide>(R, B, s);
        }
    }
    if (R.wide < 2) return;
    if constexpr (!BATCH) {
        launch_align_t<1, 1, BATCH>(R, B, 0, s);
        launch_align_t<1, 2, BATCH>(R, B, 1, s);
    }
    if constexpr (BATCH) {
        constexpr int smem = (kAlignThreads / 32) * sys_peq_words(8) * 4;
        static int grid = 0;
        if (!grid) {
            cudaFuncSetAttribute(k_align_single, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem);
            grid = grid_for(k_align_single, kAlignThreads, smem, 8);
        }
        // the single-warp classes share one work counter
        k_align_single<<<shaped(grid, R.align_blocks), kAlignThreads, smem, s>>>(
            R, B.st, align_args(B), reinterpret_cast<int*>(B.st + 1) + kSingleWorkSlot);
        launch_align_t<2, 8, BATCH>(R, B, 4, s);
        launch_align_t<4, 8, BATCH>(R, B, 5, s);
        launch_align_t<8, 8, BATCH>(R, B, 6, s);
    } else {
        launch_align_t<2, 2, BATCH>(R, B, 2, s);
        launch_align_t<4, 2, BATCH>(R, B, 3, s);
        launch_align_t<8, 2, BATCH>(R, B, 4, s);
        launch_align_t<8, 4, BATCH>(R, B, 5, s);
        launch_align_t<8, 8, BATCH>(R, B, 6, s);
    }
    if (B.long_carry) launch_align_long_t<BATCH>(R, B, s);
}

}  // namespace

// Work counters of the alignment classes live right after the RoundState in
// the same allocation.
static int* align_work_of(RoundState* st) { return reinterpret_cast<int*>(st + 1); }

void init_rounds(const DevReads& R, RoundBuffers& B, int batched, int r_max, cudaStream_t s,
                 int pass_limit) {
    const int n = R.n;
    const int threads = 256;
    const int blocks = n > 0 ? (n + threads - 1) / threads : 1;
    k_init<<<blocks, threads, 0, s>>>(B.st, B.cluster, B.remain[0], B.tidx, B.best, n, batched,
                                      r_max, pass_limit, align_work_of(B.st));
    // the open pairs' per-tentative counts start at zero (k_amb_scan keeps them so)
    if (B.amb_idx) cudaMemsetAsync(B.amb_idx, 0, sizeof(int32_t) * (kMaxBatch + 1), s);
}

void resume_rounds(const DevReads& R, RoundBuffers& B, int batched, int r_max, cudaStream_t s,
                   int pass_limit) {
    const int n = R.n;
    k_resume_state<<<1, 1, 0, s>>>(B.st, r_max, pass_limit, align_work_of(B.st));
    const int want = (n + 255) / 256, cap = num_sms() * 8;
    const int blocks = n > 0 ? (want < cap ? want : cap) : 1;
    k_resume_scan<<<blocks, 256, 0, s>>>(B.st, B.cluster, B.remain[0], B.tidx, B.best, n,
                                         batched);
    k_resume_start<<<1, 1, 0, s>>>(B.st, B.cluster, batched);
    if (B.amb_idx) cudaMemsetAsync(B.amb_idx, 0, sizeof(int32_t) * (kMaxBatch + 1), s);
}

void launch_plain_round(const DevReads& R, RoundBuffers& B, int drop, int parity, cudaStream_t s,
                        long long* count, cudaEvent_t* ev4) {
    const int32_t* rin = B.remain[parity];
    int32_t* rout = B.remain[parity ^ 1];
    B.chained = ev4 == nullptr;
    if (ev4) cudaEventRecordWithFlags(ev4[0], s, cudaEventRecordExternal);
    launch_filter_any<false>(R, B, rin, drop, s);
    if (R.pig_q && !drop)
        k_pigeon<false><<<num_sms() * 8, 256, 0, s>>>(R, B.st, B.pairs, B.seg_cap);
    if (ev4) cudaEventRecordWithFlags(ev4[1], s, cudaEventRecordExternal);
    launch_align_classes<false>(R, B, s);
    if (ev4) cudaEventRecordWithFlags(ev4[2], s, cudaEventRecordExternal);
    launch_next(B, k_compact<false>, num_sms() * 4, 256, 0, s, B.st, rin, rout,
                CompactArgs{B.cluster, align_work_of(B.st), nullptr, nullptr, 0, 0, 0, 0});
    if (ev4) cudaEventRecordWithFlags(ev4[3], s, cudaEventRecordExternal);
    if (count)
        *count += 2 + align_launches<false>(R, B) + (R.pig_q && !drop ? 1 : 0) +
                  (!drop && R.k >= kWideK ? 2 : 0);
}

void launch_align_stage(const DevReads& R, RoundBuffers& B, bool batched_mapping,
                        cudaStream_t s) {
    if (batched_mapping) launch_align_classes<true>(R, B, s);
    else launch_align_classes<false>(R, B, s);
}

int align_class_host(int words) {
    return words <= 32 ? 0 : words <= 64 ? 1 : words <= 128 ? 2 : words <= 256 ? 3
                         : words <= 512 ? 4 : words <= 1024 ? 5
                         : words <= kMaxPatternWords ? 6 : kLongClass;
}

void launch_batch_pass(const DevReads& R, RoundBuffers& B, int drop, int parity, cudaStream_t s,
                       long long* count, cudaEvent_t* ev4) {
    const int32_t* rin = B.remain[parity];
    int32_t* rout = B.remain[parity ^ 1];
    B.chained = ev4 == nullptr;
    launch_next(B, k_bselect, 1, 1024, 0, s, B.st, B.cluster, R.n, B.tent, B.tidx, B.tt, B.ttrow,
                align_work_of(B.st));
    if (ev4) cudaEventRecordWithFlags(ev4[0], s, cudaEventRecordExternal);
    launch_filter_any<true>(R, B, rin, drop, s);
    if (R.pig_q && !drop) k_pigeon<true><<<num_sms() * 8, 256, 0, s>>>(R, B.st, B.pairs, B.seg_cap);
    if (ev4) cudaEventRecordWithFlags(ev4[1], s, cudaEventRecordExternal);
    launch_align_classes<true>(R, B, s);
    if (ev4) cudaEventRecordWithFlags(ev4[2], s, cudaEventRecordExternal);
    const int r_even = B.r_auto && R.hbuckets && !drop ? hash_even_r(R.hbuckets, B.r_max) : 0;
    launch_next(B, k_bclaim, num_sms(), kMaxBatch, 0, s, B.st, B.tent, B.tt, B.ttrow, B.acc, B.tidx,
                B.best, B.cluster);
    launch_next(B, k_compact<true>, num_sms() * 4, 256, 0, s, B.st, rin, rout,
                CompactArgs{B.cluster, align_work_of(B.st), B.best, B.tent, B.seg_cap, B.acc_cap,
                            B.amb_cap, drop, r_even});
    if (ev4) cudaEventRecordWithFlags(ev4[3], s, cudaEventRecordExternal);
    if (count)
        *count += 4 + align_launches<true>(R, B) + (!drop ? 1 : 0) +
                  (R.pig_q && !drop ? 1 : 0) + (B.amb && !drop && !R.hbuckets ? 4 : 0);
    // (a word-filter form launches two kernels, six with the sorted queue of
    // open pairs: the bitmap form k_filter, k_bfilter_bits, the mask form
    // k_bmask, k_bfilter_mask, then k_amb_count, k_amb_scan, k_amb_place,
    // k_bexact_t; the hashed form k_bfilter_hash and k_bexact_d)
}

// Whether a job's per-pass k-mer index (at most `cap` postings) is kept in
// shared memory by the index filter: 16-bit offsets need cap < 65536, and the
// layout for a 1024-thread CTA must fit the device's per-block maximum.
bool index_in_smem(int k, int r_max, int64_t cap, int smem_optin) {
    if (cap <= 0 || cap >= 65536) return false;
    return IndexSmem(k, r_max, cap, true).bytes(1024 / 32) <= smem_optin;
}

int set_spin_limit(int polls) {
    const int v = polls < 0 ? kSpinLimit : polls;
    return cudaMemcpyToSymbol(c_spin_limit, &v, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace gsdr
