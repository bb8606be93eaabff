// Device generator of the extend step's one-3-cycle insertions (Extensions.java:95-141,
// Type 1 and Type 2 extensions of SortOrExtend's proof generator).
//
// A configuration is spi over n symbols with pi = (0 1 ... n-1).  An extension inserts a new
// unoriented 3-cycle before old positions a <= b <= c (not a = b = c): old position p moves
// to p + [a <= p] + [b <= p] + [c <= p], the new symbols sit at a, b + 1 and c + 2, and the
// new cycle runs from the largest of them downwards, as Configuration.ofSignature builds an
// unoriented cycle (Configuration.java:106-145).  The old cycles keep their order, relabelled.
// The reference produces
//   Type 1 (the configuration has open gates): for every open gate g and every b <= c, the
//     insertion at {g, b, c} (Extensions.java:95-116);
//   Type 2 (no open gate): every insertion (Extensions.java:118-141);
// so as a set Type 1 is every insertion whose positions include an open gate.  Open gates
// follow CommonOperations.getOpenGates (CommonOperations.java:501-546): symbol a with
// b = spi(a) is closed when an edge (c, spi(c)) of another cycle makes a, c, b, spi(c) cyclic
// in pi^-1, or a c of a's own cycle makes a, b, c cyclic in pi.
//
// Layout: slot e of configuration r enumerates the multisets a <= b <= c over [0, maxN) in
// lexicographic order (C(maxN + 2, 3) slots per configuration); flag[e] = 1 (Type 1),
// 2 (Type 2) or 0 (not an extension of this configuration), and the extended spi goes to a
// 64-byte row.
//
// One launch.  A block takes one configuration, or a share of a large one; it finds the open
// gates itself (n^2 pair tests over the block), so no gate pass runs before.  Rows with the
// same a are consecutive; a warp walks a range of them, four lanes per row with 16 bytes each in
// four registers (two lanes when a row has at most 32 symbols: the rest is zeros).
// Inserting one symbol before position z moves the bytes past z up by one and adds 1 to every
// value >= z; that is a byte select between a word and its one-byte shift, and one add, on four
// symbols at a time (values stay below 64, so a byte never carries into the next).  The
// insertion at a is shared by the rows of a.  A row leaves as four 16-byte stores, consecutive
// rows from one warp.  Flags are written slot-parallel, one byte per thread.
// Bound: the integer pipe (each step about 120 instructions for 8 or 16 rows, and a block's
// set-up), then the rows' stores.  500 configurations of 3..8 3-cycles (max_n 24, 36.6 MB written), one B200:
// 138 us per call with one thread storing a row byte by byte after a gate pass, 31 us in this
// form.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <type_traits>

#include "../../include/tdp1375.h"

namespace tdp {
namespace {

constexpr int kMaxIn = 60;  // n + 3 <= 63
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kSlotsPerBlock = 1024;  // a block's share (768: 30.9 us, 1,536: 30.8, 3,072: 35.6 at the sizes above)

__device__ __forceinline__ bool cyclic_positions3(int a, int b, int c) {
    return (a > b) + (b > c) + (c > a) <= 1;
}
__device__ __forceinline__ bool cyclic_positions4(int a, int b, int c, int d) {
    return (a > b) + (b > c) + (c > d) + (d > a) <= 1;
}

// Bytes at positions >= z of the word whose first byte is position `base` (z8 = 8 z; the
// funnel shift clamps at 32, i.e. to no byte).
__device__ __forceinline__ uint32_t bytes_from(int z8, int base) {
    return __funnelshift_lc(0u, 0xFFFFFFFFu, (uint32_t)max(z8 - 8 * base, 0));
}

// Inserts a symbol before position z: bytes past z move up by one, values >= z grow by 1, the
// byte at z becomes `value` (value < z).  `below` is the word before row[0] (its last byte
// moves in).  128 - z + v sets a byte's top bit when v >= z; v and z stay below 64.
__device__ __forceinline__ void insert_symbol(const uint32_t (&row)[4], uint32_t below, int z, int value, int base,
                                              uint32_t (&out)[4]) {
    const uint32_t k4 = (uint32_t)(128 - z) * 0x01010101u, v4 = (uint32_t)value * 0x01010101u;
    uint32_t gePrev = bytes_from(8 * z, base - 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t up = __funnelshift_l(i == 0 ? below : row[i == 0 ? 0 : i - 1], row[i], 8);
        const uint32_t ge = bytes_from(8 * z, base + 4 * i), gt = __funnelshift_l(gePrev, ge, 8);
        gePrev = ge;
        uint32_t w = (v4 & ge) | (row[i] & ~ge);
        w = (up & gt) | (w & ~gt);
        out[i] = w + (((w + k4) & 0x80808080u) >> 7);
    }
}

// The largest m with C(m, 2) <= v.
__device__ __forceinline__ int pair_root(int v) {
    int m = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)v)) * 0.5f);
    if (m * (m - 1) / 2 > v) --m;
    if ((m + 1) * m / 2 <= v) ++m;
    return m;
}

// Lexicographic index u of b <= c over the n - a symbols a..n-1; the index from the end is one
// of pairs among the symbols after b, shifted by one.
__device__ __forceinline__ void decode_pair(int u, int a, int n, int &b, int &c) {
    const int left = (n - a) * (n - a + 1) / 2 - 1 - u;
    const int m = pair_root(left);
    b = n - m;
    c = n - 1 - (left - m * (m - 1) / 2);
}

// A block's share of a configuration's flags and rows: slots over [0, maxN), rows of n + 3
// symbols.  gate: its open gates.
template <int kLanes, bool kAligned>
__device__ __forceinline__ void write_slots(const uint8_t *s, int n, int maxN, int part, int parts,
                                            unsigned long long gate, unsigned long long symbols, uint8_t *flags,
                                            uint8_t *out) {
    constexpr int kRows = 32 / kLanes;  // rows per warp step
    const int t = threadIdx.x, lane = t & 31;
    const uint8_t type = gate == 0ull ? 2 : 1;
    // an open gate among a, b, c makes a Type 1 extension; without open gates every symbol counts
    using Mask = std::conditional_t<kLanes == 2, uint32_t, unsigned long long>;  // n <= 29 symbols, or more
    const Mask useful = (Mask)(gate == 0ull ? symbols : gate);
    auto is_extension = [&](int a, int b, int c) -> bool {
        return c < n && a != c && (((useful >> a) | (useful >> b) | (useful >> c)) & 1u);
    };

    // flags of this block's share of the slots
    const int slots = (maxN + 2) * (maxN + 1) * maxN / 6;
    const int slotLast = min((part + 1) * kSlotsPerBlock, slots);
    for (int e = part * kSlotsPerBlock + t; e < slotLast; e += kThreads) {
        // counted from the end, a multiset with m symbols after its first has C(m + 2, 3) before it
        const int left = slots - 1 - e;
        int lo = 0, hi = maxN - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if ((m + 2) * (m + 1) * m / 6 <= left) lo = m;
            else hi = m - 1;
        }
        const int a = maxN - 1 - lo, rest = left - (lo + 2) * (lo + 1) * lo / 6;
        const int m = pair_root(rest);
        flags[e] = is_extension(a, maxN - m, maxN - 1 - (rest - m * (m - 1) / 2)) ? type : (uint8_t)0;
    }

    // rows: those of first position a number R(a) = C(live - a + 1, 2), in steps of kRows
    const int live = min(n, maxN);
    auto rows_of = [&](int a) -> int { return (live - a) * (live - a + 1) / 2; };
    // a prefix sum over a (one per lane; n <= 60 takes two rounds) finds this warp's first step
    const int share = part * kWarps + (t >> 5), shares = parts * kWarps;
    int steps = 0, before[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int sum = lane + 32 * h < live ? (rows_of(lane + 32 * h) + kRows - 1) / kRows : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, sum, o);
            if (lane >= o) sum += y;
        }
        before[h] = steps + sum;  // steps of all first positions up to this one
        steps = __shfl_sync(0xFFFFFFFFu, before[h], 31);
    }
    int step = steps * share / shares;
    int todo = steps * (share + 1) / shares - step;
    int a = __popc(__ballot_sync(0xFFFFFFFFu, before[0] <= step));
    if (a == 32) a += __popc(__ballot_sync(0xFFFFFFFFu, before[1] <= step));
    if (a > 0) step -= __shfl_sync(0xFFFFFFFFu, a > 32 ? before[1] : before[0], (a - 1) & 31);
    const int j = lane % kLanes, base = 16 * j, group = lane / kLanes;
    uint32_t src[4], one[4], xByte[4], keep[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        src[i] = reinterpret_cast<const uint32_t *>(s)[4 * j + i];
        keep[i] = ~bytes_from(8 * (n + 3), base + 4 * i);
    }
    int oneOf = -1, slotA = 0;
    for (; todo > 0; --todo) {
        if (oneOf != a) {
            uint32_t below = __shfl_up_sync(0xFFFFFFFFu, src[3], 1);
            insert_symbol(src, j == 0 ? 0u : below, a, 0, base, one);
            if (a == 0 && j == 0) one[0] -= 1u;  // x's byte stays 0 (0 >= z = 0 added 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) xByte[i] = (a - base) >> 2 == i ? 1u << ((a & 3) * 8) : 0u;
            oneOf = a;
            slotA = slots - (maxN - a + 2) * (maxN - a + 1) * (maxN - a) / 6;
        }
        const int u = step * kRows + group, rows = rows_of(a);
        int b, c;
        decode_pair(min(u, rows - 1), a, live, b, c);
        // x = a (its value z = c + 2 follows), y = b + 1 with value x, z with value y
        uint32_t two[4], w[4];
        uint32_t below = __shfl_up_sync(0xFFFFFFFFu, one[3], 1);
        insert_symbol(one, j == 0 ? 0u : below, b + 1, a, base, two);
        below = __shfl_up_sync(0xFFFFFFFFu, two[3], 1);
        insert_symbol(two, j == 0 ? 0u : below, c + 2, b + 1, base, w);
        if (u < rows && is_extension(a, b, c)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = (w[i] + xByte[i] * (uint32_t)(c + 2)) & keep[i];
            // slot of (a, b, c): after (a, b', .) for the b' of a..b-1, maxN - b' slots each
            const int slot = slotA + (b - a) * maxN - (b - a) * (a + b - 1) / 2 + (c - b);
            uint8_t *const dst = out + (size_t)slot * 64 + base;
            if (kAligned) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                if (kLanes == 2) *reinterpret_cast<uint4 *>(dst + 32) = make_uint4(0u, 0u, 0u, 0u);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    dst[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
                    if (kLanes == 2) dst[32 + i] = 0;
                }
            }
        }
        if (++step == (rows + kRows - 1) / kRows) {
            step = 0;
            ++a;
        }
    }
}

template <bool kAligned>
__global__ void __launch_bounds__(kThreads) insertion_kernel(const uint8_t *spi, const uint8_t *nArr, int maxN,
                                                             int parts, unsigned long long *gates, uint8_t *flags,
                                                             uint8_t *out) {
    __shared__ __align__(16) uint8_t s[64];
    __shared__ uint8_t leader[64];
    __shared__ uint32_t closed[2];
    const int r = blockIdx.x / parts, part = blockIdx.x - r * parts;
    const int t = threadIdx.x;
    const int n = min((int)nArr[r], 64);
    if (t < 64) s[t] = t < n ? spi[(size_t)r * 64 + t] & 63 : 0;
    if (t < 2) closed[t] = 0u;
    __syncthreads();
    if (t < n) {
        // cycle leader (least symbol), by walking the cycle (bounded by n)
        int m = t, cur = s[t];
        for (int it = 0; it < n && cur != t; ++it) {
            m = min(m, cur);
            cur = s[cur];
        }
        leader[t] = (uint8_t)m;
        // a fixed point is no gate
        if (s[t] == t) atomicOr(&closed[t >> 5], 1u << (t & 31));
    }
    __syncthreads();
    // four threads per symbol a, each a quarter of the symbols c
    for (int a = t >> 2, c = t & 3; a < n && c < n; c += 4) {
        const int b = s[a], d = s[c];
        if (d == c || b == a) continue;
        bool close;
        if (leader[c] != leader[a]) {
            // another cycle's edge (c, d): a, c, b, d cyclic in pi^-1
            close = cyclic_positions4(n - 1 - a, n - 1 - c, n - 1 - b, n - 1 - d);
        } else {
            close = c != a && c != b && cyclic_positions3(a, b, c);
        }
        if (close) {
            atomicOr(&closed[a >> 5], 1u << (a & 31));
            break;
        }
    }
    __syncthreads();
    const unsigned long long symbols = n >= 64 ? ~0ull : (1ull << n) - 1ull;
    const unsigned long long gate = ~((unsigned long long)closed[0] | ((unsigned long long)closed[1] << 32)) & symbols;
    if (part == 0 && t == 0) gates[r] = gate;
    const size_t slots = (size_t)((maxN + 2) * (maxN + 1) * maxN / 6);
    flags += r * slots;
    out += r * slots * 64;
    if (n + 3 <= 32)
        write_slots<2, kAligned>(s, n, maxN, part, parts, gate, symbols, flags, out);
    else
        write_slots<4, kAligned>(s, n, maxN, part, parts, gate, symbols, flags, out);
}

thread_local std::string gError;

}  // namespace
}  // namespace tdp

extern "C" const char *tdp_insertion_extensions_error(void) { return tdp::gError.c_str(); }

extern "C" int64_t tdp_insertion_extension_slots(int max_n) {
    if (max_n < 0) return 0;
    return (int64_t)(max_n + 2) * (max_n + 1) * max_n / 6;
}

extern "C" int tdp_insertion_extensions_device(const uint8_t *spi, const uint8_t *n, int count, int max_n,
                                               uint64_t *gates, uint8_t *flags, uint8_t *out, void *stream) {
    if (count < 0 || max_n < 1 || max_n > tdp::kMaxIn || (count > 0 && (!spi || !n || !gates || !flags || !out))) {
        tdp::gError = "tdp_insertion_extensions_device: need 1 <= max_n <= 60 and device buffers";
        return TDP_ERR_ARGUMENT;
    }
    if (count == 0) return 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int parts = (int)((tdp_insertion_extension_slots(max_n) + tdp::kSlotsPerBlock - 1) / tdp::kSlotsPerBlock);
    if ((long long)count * parts > 0x7FFFFFFFll) {
        tdp::gError = "tdp_insertion_extensions_device: too many configurations for one launch";
        return TDP_ERR_ARGUMENT;
    }
    // 16-byte row stores need an aligned buffer; any other address is stored byte by byte
    auto *const kernel = (reinterpret_cast<uintptr_t>(out) & 15u) == 0 ? tdp::insertion_kernel<true>
                                                                         : tdp::insertion_kernel<false>;
    kernel<<<count * parts, tdp::kThreads, 0, s>>>(spi, n, max_n, parts, reinterpret_cast<unsigned long long *>(gates),
                                                   flags, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        tdp::gError = std::string("tdp_insertion_extensions_device: ") + cudaGetErrorString(e);
        return TDP_ERR_CUDA;
    }
    return 0;
}
