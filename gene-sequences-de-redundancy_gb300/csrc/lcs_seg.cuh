// lcs_seg.cuh -- bit-parallel LCS decision on a window of text rows that
// shrinks as the DP itself rules rows out, one pair per group of G lanes.
//
// Decides LCS(pattern, text) >= c (the test of the reference's kernel_align,
// cuda-version/func.cu:828-999) with Hyyro's recurrence
//     U = V & M[x];  V' = (V + U) | (V & ~M[x]);   LCS = zeros of V,
// but with the roles of the sequences exchanged against lcs_sys.cuh: the bits
// are positions of the text (the representative, the longer sequence) and the
// steps run over the bases of the pattern (the candidate).  L(i, x), the LCS
// of the first i pattern bases with text rows 0..x, is the number of zeros of
// V in rows 0..x after i steps.
//
// Rows in use.  A common subsequence of length >= c that reaches row x after i
// steps needs
//     L(i, x) + (q - i) >= c        (every later pattern base matched), and
//     (x + 1) - L(i, x) <= T - c    (text rows passed over so far).
// Both sides are monotone in x, so after i steps the rows such a path can be
// on form one interval, read off the zero counts.  The rows below it (smaller
// x) never change again: their zeros are counted once into `base`.  The rows
// past it are set back to the initial state, which holds the value of the row
// before them; a path enters them from inside the interval.  So every cell
// of a path with >= c matches is computed, no value exceeds the true LCS, and
// L' >= c exactly when LCS >= c.  An empty interval rejects the pair.  The
// interval starts at (T - c) rows, grows to at most (T - c) + (q - c), and
// falls as losses add up: on pairs of the 200k-read workload (T/q about 2.3,
// t = 0.95, mostly rejected) it averages a third of the T rows that the
// systolic form steps for all of the text.
//
// Work split.  The pattern runs in segments of S steps.  During a segment the
// window is fixed: words w_lo .. w_lo + G*W - 1, lane j of the group holding
// words j*W .. j*W + W - 1 (S more rows than the interval, which can grow by
// one row per step).  Within a segment the group is a systolic array as in
// lcs_sys.cuh: at step s lane j applies base s - j, taking the carry of the
// addition from lane j-1's step s-1 (one shuffle per step); a segment takes
// S + G steps.  Between segments V passes through shared memory, the window
// moves and W becomes the smallest that holds it.  A warp runs 32 / G pairs
// side by side at the W of its widest.
//
// Narrow runs also cut the window to a strip along a line x = slope * i.  That
// only drops cells, so L' is still a lower bound of the LCS: an accept is
// final, anything else is run again without the strip.  Used where the text is
// so much longer than the pattern that nearly every pair is accepted.
#pragma once
#include <stdint.h>

#include "lcs.cuh"

namespace gsdr {

constexpr int kSegMaxW = 16;        // words per lane
constexpr int kSegMaxWords = 32 * kSegMaxW;  // widest window (512 words, 16,384 rows)
constexpr int kSegWideW = 24;       // the same of the wide form (768 words, a warp per pair)
constexpr int kSegWideWords = 32 * kSegWideW;
constexpr int kSegSteps8 = 128;     // steps per segment, G = 8
constexpr int kSegSteps32 = 256;    // G = 16 and 32 (the array takes G steps to fill and drain)
// code entries per warp: groups x (leading G, S, trailing G)
constexpr int kSegCodes = 4 * (kSegSteps8 + 2 * 8);
static_assert(kSegCodes >= 2 * (kSegSteps32 + 2 * 16) && kSegCodes >= kSegSteps32 + 2 * 32, "codes");
// A warp's shared memory for up to M words per lane: the match masks and the
// all-zero rows behind them, V between segments (padded, seg_vidx), the codes.
template <int M>
struct SegSmem {
    static constexpr int kNoBase = 4 * M * 32;  // table offset of the all-zero rows
    static constexpr int kPeq = 5 * M * 32;
    static constexpr int kV = 32 * M + 2 * M;
    static constexpr int kWords = kPeq + kV + kSegCodes / 2;  // u32
};

// Words of the widest window a pair can need (segments of S steps).
__host__ __device__ __forceinline__ int seg_words(int T, int q, int c, int S) {
    const int nw = (T + 31) >> 5;
    const int w = ((T - c) + (q - c) + 1 + S) / 32 + 3;
    return w < nw ? w : nw;
}

// Narrow runs: rows on either side of the line, and the slope beyond which
// more text per pattern base is not needed (above the ratio of seg_narrow).
constexpr int kSegStrip = 96;
constexpr float kSegSlopeMore = 0.6f;

// T / q at which unrelated bases start to reach c nearly always, read off the
// decisions of the named workloads (1.55 at c/q = 0.80, 1.8 at 0.85, 2.2 at
// 0.90, 2.7 at 0.95): close to linear in log2(q / (q - c)).
__host__ __device__ __forceinline__ float seg_accept_ratio(int q, int c) {
    return 0.23f + 0.57f * log2f((float)q / (float)(q - c));
}
__host__ __device__ __forceinline__ float seg_narrow_slope(int T, int q, int c) {
    return fminf((float)T / (float)q, seg_accept_ratio(q, c) + kSegSlopeMore);
}
// Whether a narrow run comes first (`words`: the full window, max_words: the
// widest window the kernel may take): from that ratio on, and where the strip's
// widest window is at most half the full one's words.  A wrong guess costs the
// strip's run and changes no decision.
__host__ __device__ __forceinline__ bool seg_narrow(int T, int q, int c, int words,
                                                    int max_words) {
    if (c >= q || T <= q) return false;
    const float s = seg_narrow_slope(T, q, c);
    if ((float)T < seg_accept_ratio(q, c) * (float)q) return false;
    const int strip = (int)(kSegSteps8 * s + 2 * kSegStrip) / 32 + 2;
    return words >= 2 * strip && strip <= max_words;
}

__device__ __forceinline__ int seg_vidx(int k) { return k + (k >> 4); }

// The match masks of a window: rows of 32 * W words per base code, then the
// all-zero rows (SegSmem).  W a multiple of four: [code][W / 4][lane][4], one
// 16-byte load per four words (a quarter of the load instructions); otherwise
// [code][W][lane].  A lane's column starts at seg_lane<W>(lane); neither form has
// bank conflicts, whatever rows the lanes are at.
template <int W>
__device__ __forceinline__ int seg_lane(int lane) {
    return W % 4 == 0 ? 4 * lane : lane;
}

// Steps over the codes at e (one u16 table offset per step) on W words.  The
// loop is unrolled only as far as its instructions stay near the scheduler's
// instruction buffer: with 8 and 4 steps per iteration a third of the stalls
// were for instructions (2-30 kbp reads: alignment 182 -> 153 ms).
template <int W>
__device__ __forceinline__ void seg_steps(const uint16_t* __restrict__ e,
                                          const uint32_t* __restrict__ peq, uint32_t (&V)[W],
                                          uint32_t en, int nsteps) {
    uint32_t from = 0;
    constexpr int U = W <= 4 ? 8 : W <= 8 ? 4 : 2;
#pragma unroll 1
    for (int s = 0; s < nsteps; s += U) {
#pragma unroll
        for (int k = 0; k < U; k++) {
            uint32_t cin = from;
            const uint32_t* pm = peq + e[s + k];
            if constexpr (W % 4 == 0) {
#pragma unroll
                for (int i = 0; i < W; i += 4) {
                    const uint4 m = *reinterpret_cast<const uint4*>(pm + 32 * i);
                    uint32_t t0, t1, t2, t3;
                    add4_carry_en(t0, t1, t2, t3, V[i], V[i + 1], V[i + 2], V[i + 3], V[i] & m.x,
                                  V[i + 1] & m.y, V[i + 2] & m.z, V[i + 3] & m.w, cin,
                                  i == 0 ? en : 0xffffffffu);
                    V[i] = t0 | (V[i] & ~m.x);
                    V[i + 1] = t1 | (V[i + 1] & ~m.y);
                    V[i + 2] = t2 | (V[i + 2] & ~m.z);
                    V[i + 3] = t3 | (V[i + 3] & ~m.w);
                }
            } else {
                peq_step<W>(V, pm, cin, en);
            }
            from = __shfl_up_sync(0xffffffffu, cin, 1);
        }
    }
}

// The state of one group's pair (the same in each lane of the group).
struct SegPair {
    const uint32_t* planes;  // text bit planes: plane c at planes + c * stride
    const uint32_t* pq;      // pattern, packed
    int stride;
    float slope;             // narrow runs: rows per step
    int q, T, c;
    int i0;                  // pattern bases applied
    int w_lo;                // first word of the window
    int w_prev, keep;        // the window's first word and live words when V was saved
    int base;                // zeros of the words below w_lo
    int n_words;             // words the next segment needs
    bool busy, narrow;
};

// Window of the next segment: words w_lo .. from the live interval's end
// w_hi_live (exclusive); S more rows can come alive.
__device__ __forceinline__ void seg_next(SegPair& P, int w_hi_live, int S) {
    int hi = min((P.T + 31) >> 5, w_hi_live + S / 32);
    if (P.narrow) {
        const int x = (int)((float)min(P.i0 + S, P.q) * P.slope) + kSegStrip;
        hi = min(hi, (x >> 5) + 1);
    }
    P.n_words = max(hi - P.w_lo, 1);
}

__device__ __forceinline__ void seg_start(SegPair& P, int S, bool narrow) {
    P.i0 = P.w_lo = P.w_prev = P.keep = P.base = 0;
    P.narrow = narrow;
    seg_next(P, (P.T - P.c) / 32 + 1, S);
}

// One segment of every group of the warp at W words per lane.  Returns in each
// lane of a busy group -1 (go on), 1 (accept) or 0 (reject; with narrow set:
// not accepted).  peq / vb / codes: the warp's shared memory, vb and codes
// already offset to the group.
template <int W, int M>
__device__ __forceinline__ int seg_segment(SegPair& P, uint32_t* peq, uint32_t* vb,
                                           uint16_t* codes, int G, int S, int lane, int& steps) {
    constexpr uint32_t kNoBase = SegSmem<M>::kNoBase;
    const int j = lane & (G - 1);
    peq += seg_lane<W>(lane);
    uint32_t V[W];
    const int wb = P.w_lo + j * W;
    const int nwT = (P.T + 31) >> 5;
    // the window's match masks: the text's bit planes are the masks
    if constexpr (W % 4 == 0) {
#pragma unroll
        for (int i = 0; i < W; i += 4) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t m[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    m[u] = P.busy && wb + i + u < nwT
                               ? __ldg(P.planes + c * P.stride + wb + i + u) : 0u;
                *reinterpret_cast<uint4*>(peq + (c * W + i) * 32) =
                    make_uint4(m[0], m[1], m[2], m[3]);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; i++) {
            const bool in = P.busy && wb + i < nwT;
#pragma unroll
            for (int c = 0; c < 4; c++)
                peq[(c * W + i) * 32] = in ? __ldg(P.planes + c * P.stride + wb + i) : 0u;
        }
    }
#pragma unroll
    for (int i = 0; i < W; i++) {
        const int k = wb + i - P.w_prev;
        V[i] = k < P.keep ? vb[seg_vidx(k)] : 0xffffffffu;
    }
    const int left = P.busy ? min(S, P.q - P.i0) : 0;
    for (int w = j; w < S / 16; w += G) {
        const uint32_t v = 16 * w < left ? __ldg(P.pq + ((P.i0 >> 4) + w)) : 0u;
        uint32_t* d = reinterpret_cast<uint32_t*>(codes + G + 16 * w);
#pragma unroll
        for (int t = 0; t < 16; t += 2) {
            const uint32_t a = 16 * w + t < left ? ((v >> (30 - 2 * t)) & 3u) * (32u * W) : kNoBase;
            const uint32_t b =
                16 * w + t + 1 < left ? ((v >> (28 - 2 * t)) & 3u) * (32u * W) : kNoBase;
            d[t >> 1] = a | (b << 16);
        }
    }
    __syncwarp();
    // steps: the longest group's bases, plus G to drain, in eights
    const int most = __reduce_max_sync(0xffffffffu, left);
    steps = ((most + 7) & ~7) + G;
    seg_steps<W>(codes + (G - j), peq, V, j == 0 ? 0u : 0xffffffffu, steps);
    // zeros: inclusive prefix over the group's lanes
    int z = 0;
#pragma unroll
    for (int i = 0; i < W; i++) z += __popc(~V[i]);
    int incl = z;
    for (int d = 1; d < G; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (j >= d) incl += o;
    }
    const int i1 = P.i0 + left;
    const int L = P.base + __shfl_sync(0xffffffffu, incl, lane | (G - 1));
    int run = P.base + incl - z;
    const int need = P.c - (P.q - i1);  // rows with L(i, x) below it are done
    // a narrow run also leaves the rows below its strip
    const int strip = P.narrow ? ((int)((float)i1 * P.slope) - kSegStrip) >> 5 : 0;
    int dead = 0, live = 0, zdead = 0;
#pragma unroll
    for (int i = 0; i < W; i++) {
        const int w = wb + i;
        if (w < nwT && 32 * w - run <= P.T - P.c) live++;
        const int pz = __popc(~V[i]);
        run += pz;
        if (w < nwT && (run < need || w < strip)) dead++, zdead += pz;
        vb[seg_vidx(j * W + i)] = V[i];
    }
    int dl = dead | (live << 16);
    for (int d = G >> 1; d > 0; d >>= 1) {
        dl += __shfl_xor_sync(0xffffffffu, dl, d);
        zdead += __shfl_xor_sync(0xffffffffu, zdead, d);
    }
    __syncwarp();
    if (!P.busy) return -1;
    if (L >= P.c) return 1;
    dead = dl & 0xffff;
    live = dl >> 16;
    int hi_live = P.w_lo + live;
    if (live == G * W) hi_live = min(nwT, max(hi_live, (P.T - P.c + L) / 32 + 1));
    if (P.w_lo + dead >= hi_live || i1 >= P.q) return 0;
    P.w_prev = P.w_lo;
    P.keep = min(live, G * W);
    P.w_lo += dead;
    P.base += zdead;
    P.i0 = i1;
    seg_next(P, hi_live, S);
    return -1;
}

// One segment at the words per lane the warp's widest window needs (at most M).
template <int M>
__device__ __forceinline__ int seg_dispatch(SegPair& P, int wl, uint32_t* peq, uint32_t* vb,
                                            uint16_t* codes, int G, int S, int lane,
                                            int& steps) {
    if constexpr (M > 16) {
        if (wl > 20) return seg_segment<24, M>(P, peq, vb, codes, G, S, lane, steps);
        if (wl > 16) return seg_segment<20, M>(P, peq, vb, codes, G, S, lane, steps);
    }
    switch (wl) {
        case 1: return seg_segment<1, M>(P, peq, vb, codes, G, S, lane, steps);
        case 2: return seg_segment<2, M>(P, peq, vb, codes, G, S, lane, steps);
        case 3: return seg_segment<3, M>(P, peq, vb, codes, G, S, lane, steps);
        case 4: return seg_segment<4, M>(P, peq, vb, codes, G, S, lane, steps);
        case 5: return seg_segment<5, M>(P, peq, vb, codes, G, S, lane, steps);
        case 6: return seg_segment<6, M>(P, peq, vb, codes, G, S, lane, steps);
        case 7:
        case 8: return seg_segment<8, M>(P, peq, vb, codes, G, S, lane, steps);
        case 9:
        case 10:
        case 11:
        case 12: return seg_segment<12, M>(P, peq, vb, codes, G, S, lane, steps);
        default: return seg_segment<16, M>(P, peq, vb, codes, G, S, lane, steps);
    }
}
// ... and the cells they step are counted at the same words.
__device__ __forceinline__ int seg_tile(int wl) {
    return wl <= 6 ? wl : wl <= 8 ? 8 : (wl + 3) & ~3;
}

}  // namespace gsdr
