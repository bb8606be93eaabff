// Permutation filter (replaces pi_filter_kernel / performGpuPiFilter, pi_filter.cu:38-260).
//
// Every pi with pi[0] = 0 over n symbols is visited in lexicographic order of
// pi[1..n-1] (the factoradic rank order of pi_filter.cu:38-53) and kept when
//   (1) the oriented triple is in cyclic order in pi           (pi_filter.cu:132-133),
//   (2) the cycle is NOT in cyclic order in pi reversed        (pi_filter.cu:135-142,
//       CommonOperations.isOriented, CommonOperations.java:443-445),
//   (3) unless skipped, the cycle admits no 2-move             (pi_filter.cu:86-115,
//       CommonOperations.java:406-431).
// B200 layout: for n <= 16 a thread decides 120 candidates at once as boolean functions of
// 128-bit words (below).  For larger n each thread walks kRanksPerThread consecutive ranks
// (one factoradic unrank, then next-permutation steps), so the O(n^2) divisions of the
// reference happen once per 16 candidates.  Hits are written in rank order: a counting pass stores per-thread hit
// counts and a block-exclusive prefix, one block scans the block totals, and a writing
// pass re-evaluates and stores rows at their final offsets.  The reference appends with
// one atomicAdd per hit in arbitrary order.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "pi_filter.h"

namespace tdp {

thread_local double gLastFilterKernelMs = 0.0;

namespace {

constexpr int kThreads = 256;
constexpr int kRanksPerThread = 16;
constexpr int kRanksPerBlock = kThreads * kRanksPerThread;
constexpr uint64_t kLaunchRanks = 1ull << 30;
constexpr uint64_t kLaunchGroups = 1ull << 22;  // of 120 ranks: 64 MB of group bits

struct FilterArgs {
    uint8_t cycle[64];
    uint8_t triple[64];
    uint8_t cycleIndex[64];
    unsigned long long fact[21];
    int cycleLen;
    int tripleLen;
    int n;
    int skip2Move;
    unsigned long long base;   // first rank of this launch
    unsigned long long total;  // (n-1)!
};

__device__ __forceinline__ bool cyclic_order(const uint8_t *index, const uint8_t *symbols, int count) {
    int leaps = 0;
    for (int i = 0; i < count; ++i) {
        const int next = (i + 1 == count) ? 0 : i + 1;
        if (index[symbols[i]] > index[symbols[next]]) {
            if (++leaps > 1) return false;
        }
    }
    return true;
}

__device__ __forceinline__ bool cyclic_order3(const uint8_t *index, int a, int b, int c) {
    const int ia = index[a], ib = index[b], ic = index[c];
    return ((ia > ib) + (ib > ic) + (ic > ia)) <= 1;
}

__device__ __forceinline__ int cycle_distance(const uint8_t *cycleIndex, int len, int a, int b) {
    const int ai = cycleIndex[a], bi = cycleIndex[b];
    return (bi >= ai) ? bi - ai : (len - ai) + bi;
}

__device__ bool has_2_move(const FilterArgs &A, const uint8_t *index) {
    const int len = A.cycleLen;
    const int before = len & 1;
    for (int i = 0; i < len - 2; ++i)
        for (int j = i + 1; j < len - 1; ++j)
            for (int k = j + 1; k < len; ++k) {
                const int a = A.cycle[i], b = A.cycle[j], c = A.cycle[k];
                if (!cyclic_order3(index, a, b, c)) continue;
                const int after = (cycle_distance(A.cycleIndex, len, a, b) & 1) +
                                  (cycle_distance(A.cycleIndex, len, b, c) & 1) +
                                  (cycle_distance(A.cycleIndex, len, c, a) & 1);
                if (after - before == 2) return true;
            }
    return false;
}

__device__ __forceinline__ void unrank(unsigned long long r, int n, const unsigned long long *fact, uint8_t *p) {
    uint8_t avail[64];
    for (int i = 0; i < n - 1; ++i) avail[i] = (uint8_t)(i + 1);
    p[0] = 0;
    for (int pos = 0; pos < n - 1; ++pos) {
        const unsigned long long f = fact[n - 2 - pos];
        const int choice = (int)(r / f);
        r -= (unsigned long long)choice * f;
        p[pos + 1] = avail[choice];
        for (int q = choice; q < n - 2 - pos; ++q) avail[q] = avail[q + 1];
    }
}

__device__ __forceinline__ void next_perm(uint8_t *p, int n) {
    int i = n - 2;
    while (i >= 1 && p[i] > p[i + 1]) --i;
    if (i < 1) return;
    int j = n - 1;
    while (p[j] < p[i]) --j;
    const uint8_t t = p[i];
    p[i] = p[j];
    p[j] = t;
    for (int l = i + 1, r = n - 1; l < r; ++l, --r) {
        const uint8_t u = p[l];
        p[l] = p[r];
        p[r] = u;
    }
}

__device__ __forceinline__ bool keep(const FilterArgs &A, const uint8_t *p, uint8_t *index, uint8_t *rindex) {
    const int n = A.n;
    for (int i = 0; i < n; ++i) index[p[i]] = (uint8_t)i;
    if (!cyclic_order(index, A.triple, A.tripleLen)) return false;
    for (int s = 0; s < n; ++s) rindex[s] = (uint8_t)((n - 1) - index[s]);
    if (cyclic_order(rindex, A.cycle, A.cycleLen)) return false;
    if (!A.skip2Move && has_2_move(A, index)) return false;
    return true;
}

// Block-wide exclusive scan of one value per thread; returns the prefix, total in *total.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned *total) {
    __shared__ unsigned warpSums[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warpSums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned s = (lane < kThreads / 32) ? warpSums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kThreads / 32) warpSums[lane] = s;
    }
    __syncthreads();
    const unsigned before = (warp > 0 ? warpSums[warp - 1] : 0u) + x - v;
    *total = warpSums[kThreads / 32 - 1];
    __syncthreads();
    return before;
}

__global__ void __launch_bounds__(kThreads) pi_filter_count_kernel(const FilterArgs A, unsigned *threadPrefix,
                                                                    unsigned *blockTotal) {
    uint8_t p[64], index[64], rindex[64];
    const unsigned long long first =
        A.base + ((unsigned long long)blockIdx.x * kThreads + threadIdx.x) * kRanksPerThread;
    unsigned hits = 0;
    if (first < A.total) {
        unrank(first, A.n, A.fact, p);
        const unsigned long long last = min(first + kRanksPerThread, A.total);
        for (unsigned long long r = first; r < last; ++r) {
            hits += keep(A, p, index, rindex) ? 1u : 0u;
            next_perm(p, A.n);
        }
    }
    unsigned total;
    const unsigned prefix = block_exclusive_scan(hits, &total);
    threadPrefix[(size_t)blockIdx.x * kThreads + threadIdx.x] = prefix;
    if (threadIdx.x == 0) blockTotal[blockIdx.x] = total;
}

// One block: exclusive scan of the block totals (64-bit running offset).
__global__ void __launch_bounds__(kThreads) pi_filter_scan_kernel(const unsigned *blockTotal,
                                                                   unsigned long long *blockOffset, int blocks,
                                                                   unsigned long long *grandTotal) {
    __shared__ unsigned long long running;
    if (threadIdx.x == 0) running = *grandTotal;
    __syncthreads();
    for (int base = 0; base < blocks; base += kThreads) {
        const int i = base + (int)threadIdx.x;
        const unsigned v = (i < blocks) ? blockTotal[i] : 0u;
        unsigned tileTotal;
        const unsigned prefix = block_exclusive_scan(v, &tileTotal);
        if (i < blocks) blockOffset[i] = running + prefix;
        __syncthreads();
        if (threadIdx.x == 0) running += tileTotal;
        __syncthreads();
    }
    if (threadIdx.x == 0) *grandTotal = running;
}

__global__ void __launch_bounds__(kThreads) pi_filter_write_kernel(const FilterArgs A, const unsigned *threadPrefix,
                                                                    const unsigned long long *blockOffset,
                                                                    uint8_t *out, unsigned long long maxRows) {
    uint8_t p[64], index[64], rindex[64];
    const unsigned long long first =
        A.base + ((unsigned long long)blockIdx.x * kThreads + threadIdx.x) * kRanksPerThread;
    if (first >= A.total) return;
    unsigned long long row = blockOffset[blockIdx.x] + threadPrefix[(size_t)blockIdx.x * kThreads + threadIdx.x];
    if (row >= maxRows) return;
    unrank(first, A.n, A.fact, p);
    const unsigned long long last = min(first + kRanksPerThread, A.total);
    for (unsigned long long r = first; r < last && row < maxRows; ++r) {
        if (keep(A, p, index, rindex)) {
            uint8_t *dst = out + row * (unsigned long long)A.n;
            for (int i = 0; i < A.n; ++i) dst[i] = p[i];
            ++row;
        }
        next_perm(p, A.n);
    }
}

// ---------------------------------------------------------------- packed path (n <= 16)
// With n <= 16 a whole pi fits in one 64-bit register as 4-bit symbols (nibble p = pi[p]),
// and so does its inverse.  A thread decides one group of candidates: those that share
// everything but their last t = min(5, n-1) positions, t! = 120 consecutive ranks for
// n >= 6, one bit each.  The code of a symbol is its position when it lies before the tail,
// else n-t plus its rank among the tail's symbols; whether x stands behind y is, for all of
// the group's candidates at once, one 128-bit word that depends on the two codes only
// (all, none, or the pairs of the t! arrangements), read from a table in shared memory.
// The predicates are boolean functions of those words:
//   (1) triple in cyclic order in pi: fewer than two descents around the triple;
//   (2) cycle oriented: the cycle is in cyclic order in reversed pi iff its positions have
//       at most one ascent around the cycle (reversal turns ascents into descents), so the
//       cycle is kept when it has two or more;
//   (3) 2-move: the cycle triples (i<j<k in cycle order) whose cycle-distance parities give
//       after - before == 2 do not depend on pi; the host lists them once (at most
//       C(16,3) = 560) and a candidate has a 2-move iff one listed triple is in cyclic order,
//       i.e. has fewer than two of three descents (one majority per word).
// The neighbours of a warp share most of their codes, so the table reads are broadcasts.
// Deciding one candidate at a time (next-permutation steps, 32 ranks per thread) cost some
// hundred instructions for each and twice, as the writing pass decided them again: n = 12
// with a 7-cycle took 1,057 us on the device and takes 51 us (count and write; 40 M
// candidates, bound by instruction issue), n = 9 took 117 us and takes 20 us (two launches'
// latency).  With the workspaces kept (below) the whole calls went from 2.3 ms to 91 us and
// from 0.8 ms to 46 us (repeated calls; the first on new inputs 140 and 73 us); with 831,600 rows
// (10 MB) the rest of a call, 0.55 ms, is their copy to the caller's pageable buffer.
constexpr int kPackedMaxN = 16;
constexpr int kTail = 5;
constexpr int kTailRanks = 120;
constexpr int kGroupThreads = 128;
constexpr int kMaxTwoMoveTriples = 560;

struct GroupArgs {
    unsigned long long base;   // first group of this launch
    unsigned groups;           // groups of this launch
    int cycleLen, tripleLen, n, tail, tailRanks, skip2Move, twoMoveCount;
    uint8_t cycle[16];
    uint8_t triple[16];
    uint32_t behind[kTail * kTail][4];     // bit r: the tail's x-th symbol stands behind its y-th in arrangement r
    uint32_t arrangement[kTailRanks];      // r-th arrangement of the tail, 4 bits per position
    uint16_t twoMove[kMaxTwoMoveTriples];  // a | b << 4 | c << 8
};

// Counters of one call, in front of its result rows (cleared before the first launch).
struct FilterHeader {
    unsigned long long hits;  // of the launches so far
    unsigned ticket;          // blocks of this launch that have counted
    unsigned pad[29];
};
static_assert(sizeof(FilterHeader) == 128, "rows follow on a line of their own");

__device__ __forceinline__ uint32_t nib(unsigned long long w, uint32_t i) { return (uint32_t)(w >> (4u * i)) & 15u; }

struct Bits {
    uint32_t w[4];
};

// The first candidate of a group (nibble p = symbol at code p) and the code of every symbol.
__device__ __forceinline__ void group_unrank(const GroupArgs &A, unsigned long long group, unsigned long long &seq,
                                             unsigned long long &code) {
    const int n = A.n, head = n - 1 - A.tail;  // positions between the fixed 0 and the tail
    // avail: symbols 1..n-1 as nibbles; those chosen for the head are taken out
    unsigned long long avail = 0xFEDCBA987654321ull & ((1ull << (4 * (n - 1))) - 1ull);
    seq = code = 0ull;
    if (head > 0) {
        // Lehmer digits, last head position first: radices 6, 7, ...  (head > 0 implies a tail of
        // 5, and the group number is below 15!/120, a sixth of it below 2^32)
        unsigned long long digits = group % 6u;
        unsigned r = (unsigned)(group / 6u);
#pragma unroll
        for (int k = 1; k < kPackedMaxN - 1 - kTail; ++k)
            if (k < head) {
                digits |= (unsigned long long)(r % (6u + k)) << (4 * k);
                r /= 6u + k;
            }
        for (int pos = 1; pos <= head; ++pos) {
            const uint32_t at = 4u * nib(digits, (uint32_t)(head - pos));
            const unsigned long long sym = (avail >> at) & 15ull;
            const unsigned long long low = (1ull << at) - 1ull;
            avail = (avail & low) | ((avail >> 4) & ~low);
            seq |= sym << (4 * pos);
            code |= (unsigned long long)pos << (4u * sym);
        }
    }
    for (int pos = head + 1; pos < n; ++pos) {
        const unsigned long long sym = avail & 15ull;
        avail >>= 4;
        seq |= sym << (4 * pos);
        code |= (unsigned long long)pos << (4u * sym);
    }
}

// Table of the block: entry 16 * x + y = arrangements with code x's symbol behind code y's.
__device__ __forceinline__ void behind_table(const GroupArgs &A, uint4 *table) {
    const int tail = A.tail, first = A.n - tail;
    for (int e = (int)threadIdx.x; e < 256; e += kGroupThreads) {
        const int x = e >> 4, y = e & 15;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (x >= first && y >= first) {
            if (x < A.n && y < A.n) {
                const uint32_t *b = A.behind[(x - first) * kTail + (y - first)];
                v = make_uint4(b[0], b[1], b[2], b[3]);
            }
        } else if (x > y) {
            v = make_uint4(~0u, ~0u, ~0u, ~0u);
        }
        table[e] = v;
    }
    __syncthreads();
}

__device__ __forceinline__ uint4 behind(const uint4 *table, unsigned long long code, uint32_t x, uint32_t y) {
    return table[16u * nib(code, x) + nib(code, y)];
}
// Adds d to a count that saturates at two.
__device__ __forceinline__ void count_two(Bits &one, Bits &two, const uint4 &d) {
    const uint32_t v[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        two.w[q] |= one.w[q] & v[q];
        one.w[q] |= v[q];
    }
}
__device__ __forceinline__ uint32_t majority(uint32_t a, uint32_t b, uint32_t c) {
    return (a & b) | (a & c) | (b & c);
}

// Kept candidates of a group, bit = rank in the group.  All lanes of a warp call it.
__device__ __forceinline__ Bits group_keep(const GroupArgs &A, const uint4 *table, unsigned long long code, bool live) {
    Bits keep, one = {}, two = {};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int left = A.tailRanks - 32 * q;
        keep.w[q] = !live || left <= 0 ? 0u : left >= 32 ? ~0u : (1u << left) - 1u;
    }
    for (int t = 0; t < A.tripleLen; ++t)
        count_two(one, two, behind(table, code, A.triple[t], A.triple[t + 1 == A.tripleLen ? 0 : t + 1]));
    Bits up1 = {}, up2 = {};
    for (int t = 0; t < A.cycleLen; ++t)
        count_two(up1, up2, behind(table, code, A.cycle[t + 1 == A.cycleLen ? 0 : t + 1], A.cycle[t]));
#pragma unroll
    for (int q = 0; q < 4; ++q) keep.w[q] &= ~two.w[q] & up2.w[q];
    if (A.skip2Move) return keep;
    for (int t = 0; t < A.twoMoveCount; ++t) {
        // every listed triple rejects about half of what is left: the warp is soon done
        if (!__any_sync(0xFFFFFFFFu, (keep.w[0] | keep.w[1] | keep.w[2] | keep.w[3]) != 0u)) break;
        const uint32_t w = A.twoMove[t];
        const uint32_t a = w & 15u, b = (w >> 4) & 15u, c = (w >> 8) & 15u;
        const uint4 ab = behind(table, code, a, b), bc = behind(table, code, b, c), ca = behind(table, code, c, a);
        keep.w[0] &= majority(ab.x, bc.x, ca.x);
        keep.w[1] &= majority(ab.y, bc.y, ca.y);
        keep.w[2] &= majority(ab.z, bc.z, ca.z);
        keep.w[3] &= majority(ab.w, bc.w, ca.w);
    }
    return keep;
}

// Exclusive scan of one value per thread over the block; the total in *total.
__device__ __forceinline__ unsigned group_scan(unsigned v, unsigned *total) {
    __shared__ unsigned warpSums[kGroupThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // the previous scan's sums have been read
    if (lane == 31) warpSums[warp] = x;
    __syncthreads();
    unsigned before = 0u, sum = 0u;
#pragma unroll
    for (int q = 0; q < kGroupThreads / 32; ++q) {
        if (q < warp) before += warpSums[q];
        sum += warpSums[q];
    }
    *total = sum;
    return before + x - v;
}

// Decides every group of the launch and counts its hits; the last block to finish turns the
// block totals into row offsets and adds the launch's hits to the header.
__global__ void __launch_bounds__(kGroupThreads) group_count_kernel(const __grid_constant__ GroupArgs A, Bits *keepOf,
                                                                     unsigned *blockTotal,
                                                                     unsigned long long *blockOffset,
                                                                     FilterHeader *header) {
    __shared__ uint4 table[256];
    __shared__ bool last;
    behind_table(A, table);
    const unsigned g = blockIdx.x * kGroupThreads + threadIdx.x;
    const bool live = g < A.groups;
    unsigned long long seq, code;
    group_unrank(A, A.base + (live ? g : 0u), seq, code);
    const Bits keep = group_keep(A, table, code, live);
    if (live && keepOf) keepOf[g] = keep;
    unsigned total;
    group_scan(__popc(keep.w[0]) + __popc(keep.w[1]) + __popc(keep.w[2]) + __popc(keep.w[3]), &total);
    if (threadIdx.x == 0) {
        blockTotal[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(&header->ticket, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    unsigned long long running = header->hits;
    constexpr unsigned kPer = 16;
    for (unsigned at = 0; at < gridDim.x; at += kPer * kGroupThreads) {
        const unsigned first = at + threadIdx.x * kPer;
        unsigned v[kPer], sum = 0u;
#pragma unroll
        for (unsigned q = 0; q < kPer; ++q) {
            v[q] = first + q < gridDim.x ? __ldcg(blockTotal + first + q) : 0u;
            sum += v[q];
        }
        unsigned tile;
        unsigned long long off = running + group_scan(sum, &tile);
#pragma unroll
        for (unsigned q = 0; q < kPer; ++q) {
            if (first + q < gridDim.x) blockOffset[first + q] = off;
            off += v[q];
        }
        running += tile;
    }
    __syncthreads();  // every thread has read header->hits
    if (threadIdx.x == 0) {
        header->hits = running;
        header->ticket = 0u;
    }
}

// Position of the h-th set bit of w (h < popc(w)).
__device__ __forceinline__ uint32_t nth_bit(uint32_t w, uint32_t h) {
    uint32_t at = 0u;
#pragma unroll
    for (uint32_t width = 16u; width; width >>= 1) {
        const uint32_t low = (uint32_t)__popc((w >> at) & ((1u << width) - 1u));
        if (h >= low) {
            h -= low;
            at += width;
        }
    }
    return at;
}

// Writes the kept candidates' rows in rank order.  The lanes of a warp share out the hits of
// its 32 groups, one row each, stage 32 rows in shared memory and store them as words.
__global__ void __launch_bounds__(kGroupThreads) group_write_kernel(const __grid_constant__ GroupArgs A,
                                                                     const Bits *keepOf,
                                                                     const unsigned long long *blockOffset,
                                                                     uint8_t *out, unsigned long long maxRows) {
    __shared__ uint32_t arrangement[kTailRanks];
    __shared__ uint4 keepShared[kGroupThreads];
    __shared__ unsigned long long seqShared[kGroupThreads];
    __shared__ __align__(16) uint8_t stage[kGroupThreads / 32][32 * kPackedMaxN + 16];
    const unsigned long long blockRow = blockOffset[blockIdx.x];
    if (blockRow >= maxRows) return;
    const int lane = (int)(threadIdx.x & 31u), n = A.n, head = n - A.tail;
    const unsigned g = blockIdx.x * kGroupThreads + threadIdx.x;
    Bits keep = {};
    if (g < A.groups) keep = keepOf[g];
    const unsigned c0 = __popc(keep.w[0]), c1 = c0 + __popc(keep.w[1]), c2 = c1 + __popc(keep.w[2]);
    const unsigned mine = c2 + __popc(keep.w[3]);
    unsigned blockHits;
    const unsigned prefix = group_scan(mine, &blockHits);
    if (blockHits == 0u) return;
    for (int r = (int)threadIdx.x; r < A.tailRanks; r += kGroupThreads) arrangement[r] = A.arrangement[r];
    unsigned long long seq = 0ull, code;
    if (mine) group_unrank(A, A.base + g, seq, code);
    keepShared[threadIdx.x] = make_uint4(keep.w[0], keep.w[1], keep.w[2], keep.w[3]);
    seqShared[threadIdx.x] = seq;
    __syncthreads();
    // hits of the warp's groups before this lane's, and of all of them
    const unsigned warpFirst = __shfl_sync(0xFFFFFFFFu, prefix, 0);
    const unsigned before = prefix - warpFirst;
    const unsigned warpHits = __shfl_sync(0xFFFFFFFFu, before + mine, 31);
    const unsigned long long warpRow = blockRow + warpFirst;
    if (warpRow >= maxRows) return;
    const unsigned rows = (unsigned)min((unsigned long long)warpHits, maxRows - warpRow);
    uint8_t *const buf = stage[threadIdx.x >> 5];
    for (unsigned from = 0; from < rows; from += 32u) {
        const unsigned count = min(32u, rows - from);
        uint8_t *const dst = out + (warpRow + from) * (unsigned long long)n;
        const unsigned shift = (unsigned)(reinterpret_cast<uintptr_t>(dst) & 3u);  // dst - shift is a word address
        const unsigned h = from + (unsigned)lane;
        // the last lane whose first hit is not behind h owns hit h (groups without hits share their
        // successor's prefix, so the last one is the owner)
        int owner = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1) {
            const unsigned b = __shfl_sync(0xFFFFFFFFu, before, owner + step);
            if (b <= h) owner += step;
        }
        unsigned at = h - __shfl_sync(0xFFFFFFFFu, before, owner);
        if ((unsigned)lane < count) {
            const int slot = (int)(threadIdx.x & ~31u) + owner;
            const uint4 k4 = keepShared[slot];
            const unsigned long long first = seqShared[slot];
            const unsigned p0 = __popc(k4.x), p1 = __popc(k4.y), p2 = __popc(k4.z);
            uint32_t w = k4.x, r = 0u;
            if (at >= p0) {
                at -= p0, w = k4.y, r = 32u;
                if (at >= p1) {
                    at -= p1, w = k4.z, r = 64u;
                    if (at >= p2) at -= p2, w = k4.w, r = 96u;
                }
            }
            r += nth_bit(w, at);
            const uint32_t order = arrangement[r];
            uint8_t *const row = buf + shift + lane * n;
            for (int p = 0; p < head; ++p) row[p] = (uint8_t)nib(first, (uint32_t)p);
            for (int p = head; p < n; ++p) {
                const uint32_t from4 = (uint32_t)head + ((order >> (4 * (p - head))) & 15u);
                row[p] = (uint8_t)nib(first, from4);
            }
        }
        __syncwarp();
        const unsigned bytes = count * (unsigned)n, end = shift + bytes;
        const unsigned firstWord = shift ? 4u : 0u, endWord = end & ~3u;
        if (shift) {  // bytes up to the first word boundary
            if ((unsigned)lane >= shift && (unsigned)lane < min(4u, end)) dst[lane - shift] = buf[lane];
        }
        for (unsigned o = firstWord + 4u * lane; o < endWord; o += 128u)
            *reinterpret_cast<uint32_t *>(dst - shift + o) = *reinterpret_cast<const uint32_t *>(buf + o);
        const unsigned tailFrom = max(endWord, firstWord);
        if (tailFrom + lane < end) dst[tailFrom - shift + lane] = buf[tailFrom + lane];
        __syncwarp();
    }
}

// Fills the tail tables of A: its t! arrangements in lexicographic order.
void tail_tables(GroupArgs &A) {
    uint8_t p[kTail];
    for (int i = 0; i < A.tail; ++i) p[i] = (uint8_t)i;
    int r = 0;
    do {
        for (int i = 0; i < A.tail; ++i) A.arrangement[r] |= (uint32_t)p[i] << (4 * i);
        for (int i = 0; i < A.tail; ++i)
            for (int j = 0; j < i; ++j) A.behind[p[i] * kTail + p[j]][r >> 5] |= 1u << (r & 31);
        ++r;
    } while (std::next_permutation(p, p + A.tail));
    A.tailRanks = r;
}

// The host half of the packed path: the pi-independent 2-move triple list
// (pi_filter.cu:86-115 restated: cycle positions i<j<k, cycle distances a->b, b->c, c->a).
int two_move_triples(const uint8_t *cycle, int len, uint16_t *out) {
    uint8_t index[64] = {};
    for (int i = 0; i < len; ++i) index[cycle[i]] = (uint8_t)i;
    auto dist = [&](int a, int b) {
        const int ai = index[a], bi = index[b];
        return (bi >= ai) ? bi - ai : (len - ai) + bi;
    };
    const int before = len & 1;
    int count = 0;
    for (int i = 0; i < len - 2; ++i)
        for (int j = i + 1; j < len - 1; ++j)
            for (int k = j + 1; k < len; ++k) {
                const int a = cycle[i], b = cycle[j], c = cycle[k];
                const int after = (dist(a, b) & 1) + (dist(b, c) & 1) + (dist(c, a) & 1);
                if (after - before == 2) out[count++] = (uint16_t)(a | (b << 4) | (c << 8));
            }
    return count;
}

// ---------------------------------------------------------------- allocation-free variant
// Scratch of tdp_pi_filter_noalloc, for callers that cannot allocate device memory: slot 0
// holds the hit total, slots [1, 1+B) the block offsets and [1+B, 1+2B) the block totals,
// B = number of 4096-rank blocks of 11! candidates (n <= 12).  Every GPU that loads the
// library keeps these 156 KB until the process exits.  In host code the symbol is only a
// stand-in: the device address comes from cudaGetSymbolAddress (noalloc_scratch below).
constexpr int kNoAllocMaxN = 12;
constexpr unsigned long long kNoAllocMaxRanks = 39916800ull;  // 11!
constexpr int kNoAllocMaxBlocks = (int)((kNoAllocMaxRanks + kRanksPerBlock - 1) / kRanksPerBlock);
static __device__ __align__(256) unsigned long long gNoAllocScratch[1 + 2 * kNoAllocMaxBlocks];

// Count pass without per-thread scratch: block totals only.
__global__ void __launch_bounds__(kThreads) noalloc_count_kernel(const FilterArgs A, unsigned long long *scratch,
                                                                  int blocks) {
    uint8_t p[64], index[64], rindex[64];
    const unsigned long long first = ((unsigned long long)blockIdx.x * kThreads + threadIdx.x) * kRanksPerThread;
    unsigned hits = 0;
    if (first < A.total) {
        unrank(first, A.n, A.fact, p);
        const unsigned long long last = min(first + kRanksPerThread, A.total);
        for (unsigned long long r = first; r < last; ++r) {
            hits += keep(A, p, index, rindex) ? 1u : 0u;
            next_perm(p, A.n);
        }
    }
    unsigned total;
    block_exclusive_scan(hits, &total);
    if (threadIdx.x == 0) scratch[1 + blocks + blockIdx.x] = total;
}

// One block: block offsets from the block totals; the hit total goes to scratch[0].
__global__ void __launch_bounds__(kThreads) noalloc_scan_kernel(unsigned long long *scratch, int blocks) {
    __shared__ unsigned long long running;
    if (threadIdx.x == 0) running = 0ull;
    __syncthreads();
    for (int base = 0; base < blocks; base += kThreads) {
        const int i = base + (int)threadIdx.x;
        const unsigned v = (i < blocks) ? (unsigned)scratch[1 + blocks + i] : 0u;
        unsigned tileTotal;
        const unsigned prefix = block_exclusive_scan(v, &tileTotal);
        if (i < blocks) scratch[1 + i] = running + prefix;
        __syncthreads();
        if (threadIdx.x == 0) running += tileTotal;
        __syncthreads();
    }
    if (threadIdx.x == 0) scratch[0] = running;
}

// Write pass: each thread recounts its ranks to find its offset inside the block, then
// re-walks them and stores the kept rows.
__global__ void __launch_bounds__(kThreads) noalloc_write_kernel(const FilterArgs A, const unsigned long long *scratch,
                                                                  uint8_t *out, unsigned long long maxRows) {
    uint8_t p[64], index[64], rindex[64];
    const unsigned long long first = ((unsigned long long)blockIdx.x * kThreads + threadIdx.x) * kRanksPerThread;
    const unsigned long long last = min(first + kRanksPerThread, A.total);
    unsigned hits = 0;
    if (first < A.total) {
        unrank(first, A.n, A.fact, p);
        for (unsigned long long r = first; r < last; ++r) {
            hits += keep(A, p, index, rindex) ? 1u : 0u;
            next_perm(p, A.n);
        }
    }
    unsigned total;
    const unsigned prefix = block_exclusive_scan(hits, &total);
    if (first >= A.total || hits == 0) return;
    unsigned long long row = scratch[1 + blockIdx.x] + prefix;
    if (row >= maxRows) return;
    unrank(first, A.n, A.fact, p);
    for (unsigned long long r = first; r < last && row < maxRows; ++r) {
        if (keep(A, p, index, rindex)) {
            uint8_t *dst = out + row * (unsigned long long)A.n;
            for (int i = 0; i < A.n; ++i) dst[i] = p[i];
            ++row;
        }
        next_perm(p, A.n);
    }
}

// Device address of gNoAllocScratch for the current device.  It is looked up
// (cudaGetSymbolAddress, with that device current) on the first call on a device and cached
// together with the device's current context, and looked up again when that context has
// changed (after cudaDeviceReset the old address is stale).
unsigned long long *noalloc_scratch(std::string &err) {
    using CtxGetCurrent = int (*)(void **);
    static std::mutex mu;
    static CtxGetCurrent ctxGetCurrent = nullptr;
    static void *ctxOf[64] = {};
    static unsigned long long *addr[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        err = "tdp_pi_filter_noalloc: no current CUDA device";
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!ctxGetCurrent) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            err = "tdp_pi_filter_noalloc: cuCtxGetCurrent is not available";
            return nullptr;
        }
        ctxGetCurrent = reinterpret_cast<CtxGetCurrent>(fn);
    }
    void *ctx = nullptr;
    if (!addr[dev] || ctxGetCurrent(&ctx) != 0 || ctx != ctxOf[dev]) {
        void *ptr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&ptr, gNoAllocScratch);
        if (e != cudaSuccess || !ptr) {
            err = std::string("tdp_pi_filter_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e);
            return nullptr;
        }
        // the runtime has made the device's primary context current by now
        ctx = nullptr;
        if (ctxGetCurrent(&ctx) != 0) ctx = nullptr;
        ctxOf[dev] = ctx;
        addr[dev] = static_cast<unsigned long long *>(ptr);
    }
    return addr[dev];
}

bool ok(cudaError_t e, std::string &err, const char *what) {
    if (e == cudaSuccess) return true;
    err = std::string(what) + ": CUDA error " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    return false;
}

// Device buffers, a pinned staging buffer and events of one call.  Allocating and freeing them
// took 0.5 ms and more per call (n = 9: 0.9 ms of which the kernels were 30 us), so a finished
// call leaves its workspace for the next: at most kIdleWorkspaces lie idle, of at most kIdleBytes
// together (n = 12 with 2^20 rows takes 18 MB), and tdp_destroy_slots frees them, as does a call
// that would otherwise run out of memory.  A call takes one out of the pool for itself, so
// concurrent calls never share one.  A workspace belongs to the context it was made in
// (cuCtxGetId: a device that was reset has another), and serves only calls in that context.
constexpr size_t kIdleBytes = 96u << 20;
constexpr size_t kIdleWorkspaces = 8;
constexpr size_t kStageBytes = 128u << 10;

struct Workspace {
    void *scratch = nullptr, *rows = nullptr;
    size_t scratchBytes = 0, rowsBytes = 0;
    uint8_t *stage = nullptr;  // pinned
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    unsigned long long context = 0;

    void release() {
        cudaFree(scratch);
        cudaFree(rows);
        if (stage) cudaFreeHost(stage);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        *this = Workspace();
    }
};

std::mutex gIdleMutex;
std::vector<Workspace> gIdle;

// Id of the calling thread's current context, 0 when there is none (or it cannot be asked).
unsigned long long current_context() {
    using CtxGetId = int (*)(void *, unsigned long long *);
    static const CtxGetId getId = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<CtxGetId>(fn);
    }();
    unsigned long long id = 0;
    return getId && getId(nullptr, &id) == 0 ? id : 0;
}

// A workspace for one call: an idle one of this context, else an empty one.  Goes back to the
// pool when the call ends well, and is freed otherwise.
struct WorkspaceLease {
    Workspace ws;
    bool finished = false;

    WorkspaceLease() {
        const unsigned long long context = current_context();
        std::lock_guard<std::mutex> lock(gIdleMutex);
        gIdle.reserve(kIdleWorkspaces);  // the destructor does not allocate
        if (!context) return;
        for (size_t i = 0; i < gIdle.size(); ++i)
            if (gIdle[i].context == context) {
                ws = gIdle[i];
                gIdle.erase(gIdle.begin() + (std::ptrdiff_t)i);
                return;
            }
    }
    ~WorkspaceLease() {
        if (finished && ws.scratchBytes + ws.rowsBytes <= kIdleBytes) {
            ws.context = current_context();
            std::lock_guard<std::mutex> lock(gIdleMutex);
            size_t bytes = ws.scratchBytes + ws.rowsBytes;
            for (const Workspace &idle : gIdle) bytes += idle.scratchBytes + idle.rowsBytes;
            if (ws.context && gIdle.size() < kIdleWorkspaces && bytes <= kIdleBytes) {
                gIdle.push_back(ws);
                return;
            }
        }
        ws.release();
    }
    WorkspaceLease(const WorkspaceLease &) = delete;
    WorkspaceLease &operator=(const WorkspaceLease &) = delete;
};

cudaError_t reserve(void *&ptr, size_t &have, size_t bytes) {
    if (have >= bytes) return cudaSuccess;
    cudaFree(ptr);
    ptr = nullptr;
    have = 0;
    cudaError_t e = cudaMalloc(&ptr, bytes);
    if (e == cudaErrorMemoryAllocation) {
        // what idle workspaces hold must not make a call fail that fits without them
        cudaGetLastError();
        pi_filter_release();
        e = cudaMalloc(&ptr, bytes);
    }
    if (e == cudaSuccess) have = bytes;
    else cudaGetLastError();  // reported by this call, not by the next launch's check
    return e;
}

}  // namespace

void pi_filter_release() {
    std::lock_guard<std::mutex> lock(gIdleMutex);
    if (gIdle.empty()) return;
    const unsigned long long context = current_context();
    int original = -1;
    if (cudaGetDevice(&original) != cudaSuccess) original = -1;
    for (Workspace &ws : gIdle) {
        // events and memory are freed in their own context; those of a context that is gone went with it
        cudaPointerAttributes at;
        if (ws.context != context) {
            if (cudaPointerGetAttributes(&at, ws.rows) != cudaSuccess || at.type != cudaMemoryTypeDevice) {
                cudaGetLastError();
                continue;
            }
            cudaSetDevice(at.device);
        }
        if (ws.context == current_context()) ws.release();
        if (original >= 0) cudaSetDevice(original);
    }
    gIdle.clear();
}

int64_t pi_filter_run(const uint8_t *cycle, int cycleLen, const uint8_t *triple, int tripleLen, int n,
                      int skip2Move, uint8_t *out, int64_t maxRows, double timeLimitS, std::string &err) {
    if (n > 63) {
        err = "n exceeds PI_FILTER_MAX_N";
        return -1;
    }
    if (n < 1) {
        err = "n must be at least 1";
        return -1;
    }
    if (n > 21) {
        err = "pi filter: (n-1)! does not fit in 64 bits for n > 21";
        return -1;
    }
    if (cycleLen < 0 || cycleLen > 63 || tripleLen < 0 || tripleLen > 63 || maxRows < 0) {
        err = "pi filter: invalid cycle/triple length or row limit";
        return -1;
    }
    for (int i = 0; i < cycleLen; ++i)
        if (cycle[i] >= n) {
            err = "pi filter: cycle symbol out of range";
            return -1;
        }
    for (int i = 0; i < tripleLen; ++i)
        if (triple[i] >= n) {
            err = "pi filter: triple symbol out of range";
            return -1;
        }
    FilterArgs A;
    std::memset(&A, 0, sizeof(A));
    std::memcpy(A.cycle, cycle, cycleLen);
    std::memcpy(A.triple, triple, tripleLen);
    for (int i = 0; i < cycleLen; ++i) A.cycleIndex[cycle[i]] = (uint8_t)i;
    A.fact[0] = 1;
    for (int i = 1; i < 21; ++i) A.fact[i] = A.fact[i - 1] * (unsigned long long)i;
    A.cycleLen = cycleLen;
    A.tripleLen = tripleLen;
    A.n = n;
    A.skip2Move = skip2Move ? 1 : 0;
    A.total = A.fact[n - 1 > 0 ? n - 1 : 0];

    // n <= 16 (with cycle and triple of at most 16 symbols) takes the packed-register kernels,
    // whose units are groups of t! ranks
    const bool packed = n <= kPackedMaxN && cycleLen <= 16 && tripleLen <= 16;
    GroupArgs G;
    std::memset(&G, 0, sizeof(G));
    if (packed) {
        std::memcpy(G.cycle, cycle, cycleLen);
        std::memcpy(G.triple, triple, tripleLen);
        G.cycleLen = cycleLen;
        G.tripleLen = tripleLen;
        G.n = n;
        G.tail = std::min(kTail, n - 1);
        G.skip2Move = A.skip2Move;
        G.twoMoveCount = two_move_triples(cycle, cycleLen, G.twoMove);
        tail_tables(G);
    }
    const uint64_t unitRanks = packed ? (uint64_t)G.tailRanks : 1;
    const uint64_t launchUnits = packed ? kLaunchGroups : kLaunchRanks;
    const uint64_t units = A.total / unitRanks;  // the t! of the packed path divides (n-1)!
    const uint64_t unitsPerBlock = packed ? kGroupThreads : kRanksPerBlock;
    const size_t maxBlocks = (size_t)((std::min(launchUnits, units) + unitsPerBlock - 1) / unitsPerBlock);
    // scratch: block offsets, block totals, then the groups' bits or the threads' prefixes
    const size_t offsetBytes = (maxBlocks * sizeof(unsigned long long) + 127) & ~(size_t)127;
    const size_t totalBytes = (maxBlocks * sizeof(unsigned) + 127) & ~(size_t)127;
    const size_t unitBytes = packed ? maxBlocks * kGroupThreads * sizeof(Bits) : maxBlocks * kThreads * sizeof(unsigned);
    // no call has more rows than candidates
    const uint64_t maxRowsHere = std::min<uint64_t>((uint64_t)maxRows, A.total);
    const size_t rowBytes = (size_t)maxRowsHere * (size_t)n;

    WorkspaceLease lease;
    Workspace &ws = lease.ws;
    if (!ok(reserve(ws.scratch, ws.scratchBytes, offsetBytes + totalBytes + unitBytes), err, "cudaMalloc")) return -3;
    if (!ok(reserve(ws.rows, ws.rowsBytes, sizeof(FilterHeader) + rowBytes), err, "cudaMalloc(rows)")) return -4;
    if ((!ws.stage && !ok(cudaHostAlloc(&ws.stage, kStageBytes, cudaHostAllocPortable), err, "cudaHostAlloc")) ||
        (!ws.e0 && !ok(cudaEventCreate(&ws.e0), err, "cudaEventCreate")) ||
        (!ws.e1 && !ok(cudaEventCreate(&ws.e1), err, "cudaEventCreate")))
        return -3;
    FilterHeader *const header = static_cast<FilterHeader *>(ws.rows);
    uint8_t *const rows = static_cast<uint8_t *>(ws.rows) + sizeof(FilterHeader);
    unsigned long long *const offsets = static_cast<unsigned long long *>(ws.scratch);
    unsigned *const totals = reinterpret_cast<unsigned *>(static_cast<uint8_t *>(ws.scratch) + offsetBytes);
    void *const perUnit = static_cast<uint8_t *>(ws.scratch) + offsetBytes + totalBytes;
    if (!ok(cudaMemsetAsync(header, 0, sizeof(FilterHeader)), err, "cudaMemset")) return -3;

    float kernelMs = 0.f;
    const auto start = std::chrono::steady_clock::now();
    // header and the first rows come back in one copy
    const size_t staged = sizeof(FilterHeader) + std::min(out ? rowBytes : 0, kStageBytes - sizeof(FilterHeader));
    for (uint64_t base = 0; base < units; base += launchUnits) {
        const uint64_t here = std::min<uint64_t>(launchUnits, units - base);
        const int blocks = (int)((here + unitsPerBlock - 1) / unitsPerBlock);
        cudaEventRecord(ws.e0);
        if (packed) {
            G.base = base;
            G.groups = (unsigned)here;
            Bits *const keepOf = maxRowsHere > 0 ? static_cast<Bits *>(perUnit) : nullptr;
            group_count_kernel<<<blocks, kGroupThreads>>>(G, keepOf, totals, offsets, header);
            if (maxRowsHere > 0)
                group_write_kernel<<<blocks, kGroupThreads>>>(G, keepOf, offsets, rows, maxRowsHere);
        } else {
            A.base = base;
            unsigned *const prefix = static_cast<unsigned *>(perUnit);
            pi_filter_count_kernel<<<blocks, kThreads>>>(A, prefix, totals);
            pi_filter_scan_kernel<<<1, kThreads>>>(totals, offsets, blocks, &header->hits);
            if (maxRowsHere > 0)
                pi_filter_write_kernel<<<blocks, kThreads>>>(A, prefix, offsets, rows, maxRowsHere);
        }
        cudaEventRecord(ws.e1);
        if (!ok(cudaGetLastError(), err, "pi filter launch")) return -3;
        const bool last = base + launchUnits >= units;
        if (last && !ok(cudaMemcpyAsync(ws.stage, ws.rows, staged, cudaMemcpyDeviceToHost), err, "read rows"))
            return -3;
        if (!ok(cudaStreamSynchronize(nullptr), err, "pi filter")) return -3;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ws.e0, ws.e1);
        kernelMs += ms;
        const double elapsed = std::chrono::duration<double>(std::chrono::steady_clock::now() - start).count();
        if (!last && elapsed > timeLimitS) {
            err = "pi filter: time limit exceeded";
            lease.finished = true;
            return -5;
        }
    }
    gLastFilterKernelMs = kernelMs;
    unsigned long long hits;
    std::memcpy(&hits, ws.stage, sizeof(hits));
    const size_t keptBytes = (size_t)std::min<uint64_t>(hits, maxRowsHere) * (size_t)n;
    if (keptBytes > 0 && out) {
        const size_t first = std::min(keptBytes, staged - sizeof(FilterHeader));
        std::memcpy(out, ws.stage + sizeof(FilterHeader), first);
        if (keptBytes > first &&
            !ok(cudaMemcpy(out + first, rows + first, keptBytes - first, cudaMemcpyDeviceToHost), err, "read rows"))
            return -3;
    }
    lease.finished = true;
    return (int64_t)hits;
}

int64_t pi_filter_noalloc_run(const uint8_t *cycle, int cycleLen, const uint8_t *triple, int tripleLen, int n,
                              int skip2Move, uint8_t *outDevice, int64_t maxRows, cudaStream_t stream,
                              std::string &err) {
    if (n < 1 || n > kNoAllocMaxN) {
        err = "tdp_pi_filter_noalloc: n must be in 1..12 (its static scratch covers (n-1)! <= 11! candidates); "
              "use tdp_pi_filter for larger n";
        return -1;
    }
    if (cycleLen < 0 || cycleLen > 63 || tripleLen < 0 || tripleLen > 63 || maxRows < 0 ||
        (maxRows > 0 && !outDevice) || (cycleLen > 0 && !cycle) || (tripleLen > 0 && !triple)) {
        err = "tdp_pi_filter_noalloc: invalid cycle/triple length, row limit or output buffer";
        return -1;
    }
    for (int i = 0; i < cycleLen; ++i)
        if (cycle[i] >= n) {
            err = "tdp_pi_filter_noalloc: cycle symbol out of range";
            return -1;
        }
    for (int i = 0; i < tripleLen; ++i)
        if (triple[i] >= n) {
            err = "tdp_pi_filter_noalloc: triple symbol out of range";
            return -1;
        }
    unsigned long long *scratch = noalloc_scratch(err);
    if (!scratch) return -3;
    FilterArgs A;
    std::memset(&A, 0, sizeof(A));
    std::memcpy(A.cycle, cycle, cycleLen);
    std::memcpy(A.triple, triple, tripleLen);
    for (int i = 0; i < cycleLen; ++i) A.cycleIndex[cycle[i]] = (uint8_t)i;
    A.fact[0] = 1;
    for (int i = 1; i < 21; ++i) A.fact[i] = A.fact[i - 1] * (unsigned long long)i;
    A.cycleLen = cycleLen;
    A.tripleLen = tripleLen;
    A.n = n;
    A.skip2Move = skip2Move ? 1 : 0;
    A.total = A.fact[n - 1 > 0 ? n - 1 : 0];
    A.base = 0;
    const int blocks = (int)((A.total + kRanksPerBlock - 1) / kRanksPerBlock);
    // The scratch keeps the previous call's contents; nothing needs clearing: the count pass
    // writes every block total the scan reads, and the scan writes every offset the write
    // pass reads and the hit total.
    noalloc_count_kernel<<<blocks, kThreads, 0, stream>>>(A, scratch, blocks);
    noalloc_scan_kernel<<<1, kThreads, 0, stream>>>(scratch, blocks);
    if (maxRows > 0)
        noalloc_write_kernel<<<blocks, kThreads, 0, stream>>>(A, scratch, outDevice, (unsigned long long)maxRows);
    if (!ok(cudaGetLastError(), err, "tdp_pi_filter_noalloc launch")) return -3;
    unsigned long long hits = 0;
    if (!ok(cudaMemcpyAsync(&hits, scratch, sizeof(hits), cudaMemcpyDeviceToHost, stream), err,
            "tdp_pi_filter_noalloc read") ||
        !ok(cudaStreamSynchronize(stream), err, "tdp_pi_filter_noalloc"))
        return -3;
    return (int64_t)hits;
}

}  // namespace tdp
