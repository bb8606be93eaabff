// Batched extension filter: the permutation-filter predicates of the reference
// (pi_filter.cu:55-115, CommonOperations.java:406-445) applied to every extension of many
// base configurations that adds one 3-cycle.  No reference counterpart as a batch: the
// reference filters the (n-1)! pi of a single cycle.
//
// Candidates of a base (spi, pi) over n symbols, in this order:
//   A. for every a<b<c (lexicographic) and orientation o: spi' = spi o rho with rho = (a b c)
//      (o = 0) or (a c b) (o = 1), pi' = pi; the added cycle is rho;
//   B. for every 0 <= g1 <= g2 <= g3 <= n (lexicographic) and orientation o: new symbols
//      x=n, y=n+1, z=n+2 inserted into pi before original positions g1, g2, g3 (x first on
//      ties), spi' = spi plus (x y z) (o = 0) or (x z y) (o = 1).
// Kept: the added cycle, as written, is in cyclic order in pi'; some cycle of spi' is
// oriented; no oriented cycle of spi' admits a 2-move.
//
// What a candidate's verdict depends on, and so what the kernel computes:
//   * No part-B candidate is kept.  Its added cycle must be in cyclic order in pi', and a
//     3-cycle in cyclic order is oriented (two ascents around it) and admits the 2-move on its
//     own three symbols (distances 1, 1, 1), so the last condition rejects it.
//   * Of the two orientations of a part-A triple exactly one is in cyclic order in pi.
//   * That candidate changes only the cycles its three symbols lie in.  The others keep their
//     cyclic sequence of positions, so one pass per base decides for every cycle whether it is
//     oriented and whether it is oriented with a 2-move ("bad").  A bad cycle outside the
//     three symbols' cycles rejects the candidate; otherwise only the new cycles through the
//     three symbols are walked.
// Both predicates are invariant under rotation of the cycle's written form: orientation counts
// ascents around the cycle, a 2-move is a triple of cycle positions with given distance
// parities whose symbols are in cyclic order.  For an odd length all three distances are odd,
// for an even length exactly two are.
//
// One block per base and span of triples: it clears its share of the base's keep bytes with
// 16-byte stores, decides the base's cycles, collects the triples that pass the per-base test
// into a shared list and walks those densely, one per thread; only kept bytes are written
// again.  Bound: the latency of a block's chain (load, cycle walks, list, candidate walks);
// the keep bytes themselves are 4.3 MB, under 1 us.  1,000 bases of six 3-cycles (n = 18,
// 4.29 M candidates), one B200: 236 us per call with one thread building and walking every
// candidate's whole configuration (226 M warp instructions), 20 us in this form (8 M).
// Spans of 256 / 1,024 triples 23.2 / 23.1 us, blocks of 128 threads 21.8 us.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "extension_filter.h"

namespace tdp {
namespace {

constexpr int kThreads = 256;
constexpr int kSpan = 512;  // part-A triples per block

struct ExtArgs {
    const uint8_t *spi;  // bases, rows of 64 bytes
    const uint8_t *pi;
    int n;
    int perBase;
    int triples;  // C(n, 3): part A has two candidates per triple
    int spans;    // blocks per base
    uint8_t *keep;
};

struct BaseSmem {
    uint8_t spi[64], index[64];           // successor, position in pi
    uint8_t cycle[64], step[64], len[64]; // least symbol of the cycle, steps from it, length
    uint8_t order[64][64];                // order[c][t]: symbol t steps after c (c least of its cycle)
    int ascents[64];
    unsigned long long oriented, bad;     // per cycle, at the bit of its least symbol
    int survivors;
    uint32_t list[kSpan];                 // a | b << 6 | c << 12 | orientation << 18
};

// Lexicographic index t of a < b < c over n symbols.  The index counted from the end is
// C(n-a, 3)-like in the number of symbols after a, so a is found by bisection over at most 60
// values and b from the root of a quadratic (exact in fp32 for these sizes, then corrected).
__device__ __forceinline__ void decode_triple(int t, int n, int triples, int &a, int &b, int &c) {
    const int left = triples - 1 - t;  // triples after this one
    int lo = 2, hi = n - 1;            // the largest m with C(m, 3) <= left is n - 1 - a
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (m * (m - 1) * (m - 2) / 6 <= left) lo = m;
        else hi = m - 1;
    }
    a = n - 1 - lo;
    const int rest = left - lo * (lo - 1) * (lo - 2) / 6;  // pairs after (b, c) among the symbols after a
    int m = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)rest)) * 0.5f);
    if (m * (m - 1) / 2 > rest) --m;
    if ((m + 1) * m / 2 <= rest) ++m;  // the largest m with C(m, 2) <= rest is n - 1 - b
    b = n - 1 - m;
    c = n - 1 - (rest - m * (m - 1) / 2);
}

__device__ __forceinline__ bool cyclic3(int ia, int ib, int ic) {
    return ((ia > ib) + (ib > ic) + (ic > ia)) <= 1;
}

// The positions of a walked cycle.  Up to 10 symbols fit one register at 6 bits each (merging
// three 3-cycles gives 9), so the pair loops read no memory; longer cycles use local memory.
struct PackedCycle {
    unsigned long long w = 0ull;
    __device__ __forceinline__ void set(int i, int v) { w |= (unsigned long long)v << (6 * i); }
    __device__ __forceinline__ int at(int i) const { return (int)(w >> (6 * i)) & 63; }
    __device__ __forceinline__ void clear() { w = 0ull; }
};
constexpr int kPackedCycle = 10;
struct LongCycle {
    uint8_t p[64];
    __device__ __forceinline__ void set(int i, int v) { p[i] = (uint8_t)v; }
    __device__ __forceinline__ int at(int i) const { return p[i]; }
    __device__ __forceinline__ void clear() {}
};

// Whether cycle steps i < j have a third step k > j that completes a 2-move: for an odd length
// j - i and k - j odd; for an even length not all three distances even.
template <typename C>
__device__ __forceinline__ bool two_move_from(const C &p, int i, int j, int len) {
    const bool odd = len & 1;
    if (odd && !((j - i) & 1)) return false;
    const int pi = p.at(i), pj = p.at(j);
    const int stride = (odd || !((j - i) & 1)) ? 2 : 1;
    for (int k = j + 1; k < len; k += stride)
        if (cyclic3(pi, pj, p.at(k))) return true;
    return false;
}

// The base's cycles; every thread of the block calls it.
__device__ void load_base(BaseSmem &S, const uint8_t *spi, const uint8_t *pi, int n) {
    const int t = threadIdx.x;
    if (t < 64) {
        S.spi[t] = t < n ? spi[t] : (uint8_t)t;
        S.ascents[t] = 0;
        if (t < n) S.index[pi[t]] = (uint8_t)t;
    }
    if (t == 0) {
        S.oriented = 0ull;
        S.bad = 0ull;
        S.survivors = 0;
    }
    __syncthreads();
    if (t < n) {
        // bounded walks: a row that is not a permutation cannot hang the block
        int least = t, len = 1;
        for (int y = S.spi[t]; y != t && len < 64; y = S.spi[y]) {
            least = min(least, y);
            ++len;
        }
        int back = 0;
        for (int y = t; y != least && back < 64; y = S.spi[y]) ++back;
        const int step = back == 0 ? 0 : len - back;
        S.cycle[t] = (uint8_t)least;
        S.step[t] = (uint8_t)step;
        S.len[t] = (uint8_t)len;
        S.order[least][step & 63] = (uint8_t)t;
        if (S.index[t] < S.index[S.spi[t]]) atomicAdd(&S.ascents[least], 1);
    }
    __syncthreads();
    if (t < n && S.cycle[t] == t && S.ascents[t] >= 2) atomicOr(&S.oriented, 1ull << t);
    __syncthreads();
    // pairs of steps i < j of every oriented cycle, four threads per symbol
    if (t < 4 * n) {
        const int x = t >> 2, c = S.cycle[x], i = S.step[x], len = S.len[x];
        if ((S.oriented >> c) & 1ull) {
            const bool odd = len & 1;
            const int pi0 = S.index[x];
            for (int j = i + 1 + (t & 3); j < len - 1; j += 4) {
                const bool oddStep = (j - i) & 1;
                if (odd && !oddStep) continue;
                const int pj = S.index[S.order[c][j]];
                for (int k = j + 1; k < len; k += (odd || !oddStep) ? 2 : 1)
                    if (cyclic3(pi0, pj, S.index[S.order[c][k]])) {
                        atomicOr(&S.bad, 1ull << c);
                        j = len;
                        break;
                    }
            }
        }
    }
    __syncthreads();
}

// Whether the candidate spi o (x0 x1 x2) is kept, given that no bad cycle lies outside the
// three symbols' cycles: every new cycle through them is walked and tested.
template <typename C>
__device__ __forceinline__ bool walk_candidate(const BaseSmem &S, int x0, int x1, int x2, int n) {
    const unsigned long long touched =
        (1ull << S.cycle[x0]) | (1ull << S.cycle[x1]) | (1ull << S.cycle[x2]);
    bool any = (S.oriented & ~touched) != 0ull;
    C p;
    int seen = 0;
#pragma unroll 1
    for (int start = 0; start < 3; ++start) {
        if ((seen >> start) & 1) continue;
        const int s = start == 0 ? x0 : start == 1 ? x1 : x2;
        int cur = s, len = 0, ascents = 0;
        p.clear();
        do {
            p.set(len++, S.index[cur]);
            int from = cur;
            if (cur == x0) from = x1, seen |= 1;
            if (cur == x1) from = x2, seen |= 2;
            if (cur == x2) from = x0, seen |= 4;
            const int next = S.spi[from];
            ascents += S.index[cur] < S.index[next] ? 1 : 0;
            cur = next;
        } while (cur != s && len < n);
        if (ascents < 2) continue;
        any = true;
        for (int i = 0; i < len - 2; ++i)
            for (int j = i + 1; j < len - 1; ++j)
                if (two_move_from(p, i, j, len)) return false;
    }
    return any;
}

__global__ void __launch_bounds__(kThreads) extension_filter_kernel(const ExtArgs A) {
    __shared__ BaseSmem S;
    const int base = blockIdx.x / A.spans, span = blockIdx.x - base * A.spans;
    const int n = A.n;
    // this block's share of the base's bytes: its triples' pairs, and an equal part of part B
    uint8_t *const keep = A.keep + (size_t)base * (size_t)A.perBase;
    const int first = span * kSpan, last = min(first + kSpan, A.triples);
    const int restLen = A.perBase - 2 * A.triples;
    const int restFirst = (int)((long long)restLen * span / A.spans);
    const int restLast = (int)((long long)restLen * (span + 1) / A.spans);
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        uint8_t *const from = part == 0 ? keep + 2 * first : keep + 2 * A.triples + restFirst;
        uint8_t *const to = part == 0 ? keep + 2 * last : keep + 2 * A.triples + restLast;
        uint8_t *const lo = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(from) + 15) & ~uintptr_t(15));
        uint8_t *const hi = reinterpret_cast<uint8_t *>(reinterpret_cast<uintptr_t>(to) & ~uintptr_t(15));
        if (lo >= hi) {
            for (uint8_t *q = from + threadIdx.x; q < to; q += kThreads) *q = 0;
        } else {
            for (uint8_t *q = lo + 16 * threadIdx.x; q < hi; q += 16 * kThreads)
                *reinterpret_cast<uint4 *>(q) = make_uint4(0u, 0u, 0u, 0u);
            if (from + threadIdx.x < lo) from[threadIdx.x] = 0;
            if (hi + threadIdx.x < to) hi[threadIdx.x] = 0;
        }
    }
    load_base(S, A.spi + (size_t)base * 64, A.pi + (size_t)base * 64, n);
    if (__popcll(S.bad) > 3) return;  // three symbols cannot touch every bad cycle
    for (int t = first + (int)threadIdx.x; t < last; t += kThreads) {
        int a, b, c;
        decode_triple(t, n, A.triples, a, b, c);
        const unsigned long long touched = (1ull << S.cycle[a]) | (1ull << S.cycle[b]) | (1ull << S.cycle[c]);
        if (S.bad & ~touched) continue;
        const int o = cyclic3(S.index[a], S.index[b], S.index[c]) ? 0 : 1;
        S.list[atomicAdd(&S.survivors, 1)] =
            (uint32_t)a | ((uint32_t)b << 6) | ((uint32_t)c << 12) | ((uint32_t)o << 18);
    }
    __syncthreads();
    // (the barrier also orders the zeros above before the kept bytes below)
    for (int q = threadIdx.x; q < S.survivors; q += kThreads) {
        const uint32_t w = S.list[q];
        const int a = (int)(w & 63u), b = (int)((w >> 6) & 63u), c = (int)((w >> 12) & 63u), o = (int)(w >> 18);
        const int x1 = o == 0 ? b : c, x2 = o == 0 ? c : b;
        const int ca = S.cycle[a], cb = S.cycle[b], cc = S.cycle[c];
        const int symbols = S.len[a] + (cb != ca ? S.len[b] : 0) + (cc != ca && cc != cb ? S.len[c] : 0);
        if (!(symbols <= kPackedCycle ? walk_candidate<PackedCycle>(S, a, x1, x2, n)
                                      : walk_candidate<LongCycle>(S, a, x1, x2, n)))
            continue;
        // lexicographic index of (a, b, c): triples before a, pairs before b, then c
        const int ta = n - a, tb = n - b;
        const int t = A.triples - ta * (ta - 1) * (ta - 2) / 6 + (ta - 1) * (ta - 2) / 2 - tb * (tb - 1) / 2 + (c - b - 1);
        keep[2 * t + o] = 1;
    }
}

bool ok(cudaError_t e, std::string &err, const char *what) {
    if (e == cudaSuccess) return true;
    err = std::string(what) + ": CUDA error " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    return false;
}

int host_comb3(int n) { return n < 3 ? 0 : n * (n - 1) * (n - 2) / 6; }

}  // namespace

int extension_count(int n) { return 2 * host_comb3(n) + 2 * host_comb3(n + 3); }

int extension_filter_device(const uint8_t *spiDev, const uint8_t *piDev, int n, int count, uint8_t *keepDev,
                            cudaStream_t stream, std::string &err) {
    if (n < 3 || n + 3 > 63 || count < 0) {
        err = "tdp_extension_filter: n must be in 3..60";
        return -1;
    }
    if (count == 0) return 0;
    const int triples = host_comb3(n), spans = (triples + kSpan - 1) / kSpan;
    if ((long long)count * spans > 0x7FFFFFFFll) {
        err = "tdp_extension_filter: too many bases for one launch";
        return -1;
    }
    ExtArgs A{spiDev, piDev, n, extension_count(n), triples, spans, keepDev};
    extension_filter_kernel<<<count * spans, kThreads, 0, stream>>>(A);
    if (!ok(cudaGetLastError(), err, "extension filter launch")) return -3;
    return 0;
}

}  // namespace tdp
