// Batched canonical form of configurations: Configuration.getCanonical / hashCode
// (Configuration.java:56-104, 147-195, 241-245, 290-303), one warp per configuration.
//
// A configuration is spi over symbols 0..n-1 (n <= 63), every symbol in a cycle of length
// >= 2, with pi = (0 1 ... n-1) (CANONICAL_PI).  Its 2n equivalent signatures are, for every
// start symbol r of pi, the signature under pi started at r (variant 2r) and the signature
// of the mirrored configuration (variant 2r+1: spi conjugated by the involution that swaps
// the symbols at pi positions i and n-1-i, then inverted).  The canonical signature is the
// one with the least hash (CRC32 of the big-endian float bytes, as a signed int), ties
// broken lexicographically, scanning the variants in the reference's order; the
// configuration's hash code is that hash.
//
// One warp per row, lanes over variants.  What makes a lane's walk along its variant cheap:
//  * whether a cycle is oriented (more than one leap of pi^-1 positions) is the same in every
//    variant: with d = (pos(succ) - pos(s)) mod n, the descents around a cycle number
//    sum(d) / n, and neither a rotation of pi nor the mirror changes a d.  So the cycle tables
//    (cycle number, steps t from the least symbol, length, orientation) are built once per row.
//  * the walk needs no positions: the label of a cycle is the count of cycles met before it,
//    plus one, and the index of an oriented symbol is t minus the t of the cycle's first symbol
//    met (modulo its length; the mirror runs t backwards).  Each lane keeps (label, first t)
//    per cycle in its own column of shared memory.
//  * the CRC32 takes a whole float per step: crc' is linear in crc ^ value, so it is the xor of
//    seven table entries selected by 5-bit windows.  A window's table has 32 words, one per
//    bank, so the lookups of a warp never conflict (a byte table costs about 3.5 wavefronts per
//    lookup, and four of them in series per float).
// The least hash is reduced over lanes and groups of 32 variants.  Only the winner's row is
// written out, built position-parallel; variants that tie with it on the hash (mostly
// symmetric configurations, with equal rows) are built and compared the same way, in variant
// order.
// Bound: instruction issue (about 45 instructions per variant and position) and the shared
// memory pipe (11 wavefronts); HBM moves 329 bytes per row.  250,000 rows of 3..10 3-cycles
// on one B200: 2,780 us with lanes over positions, shared-memory atomics per variant and a byte
// table per CRC (1,719 M warp instructions), 713 us in this form (590 M).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>

#include "canonical.h"

namespace tdp {
namespace {

constexpr int kWarps = 8;   // warps (configurations) per block
constexpr int kMaxN = 63;   // two symbols per lane in the position-parallel parts; at most 31 cycles
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t kPoly = 0xEDB88320u;  // reflected CRC-32 polynomial (java.util.zip.CRC32)

struct CanonArgs {
    const uint8_t *spi;  // rows of 64 bytes: successor array
    const uint8_t *n;    // per-row symbol count
    int count;
    float *sig;          // rows of 64 floats: canonical signature
    int32_t *hash;
    int32_t *variant;
};

// A symbol's word: cycle number << 7 (the byte offset of its row in WarpSmem::met), t, length
// and orientation; t, length and the orientation bit are 0 on unoriented cycles.
constexpr uint32_t kCycleOffset = 31u << 7;
constexpr int kTShift = 12, kLenShift = 18, kOrientedShift = 24;

struct WarpSmem {
    uint32_t met[32][32];      // [cycle][lane]: float bits of the label | first t; 0 = not met
    uint32_t word[2][2 * 64];  // [mirror][symbol], two periods: no wrap along a walk
    uint8_t spi[64];
    float best[64];
    int firstPos[32], anchor[32];
};

// The signature value of one symbol: label plus index/100 (index 0 on unoriented cycles), the
// same two single-precision operations as Java's label + (float) index / 100.
__device__ __forceinline__ float value_of(const float *hundredth, uint32_t w, uint32_t met) {
    int idx = (int)((w >> kTShift) & 63u) - (int)(met & 63u);
    if (idx < 0) idx += (int)((w >> kLenShift) & 63u);
    return __fadd_rn(__uint_as_float(met & ~63u), hundredth[idx + (int)(w >> kOrientedShift)]);
}

// The row of one variant, lanes over positions: value at positions lane and lane + 32.
__device__ __forceinline__ void build_row(WarpSmem &S, const float *hundredth, int variant, int n, int lane,
                                          float (&value)[2]) {
    const int r = variant >> 1, mirror = variant & 1;
    S.firstPos[lane] = 127;
    __syncwarp();
    uint32_t w[2];
    int cycle[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = lane + 32 * h;
        w[h] = 0u, cycle[h] = 0;
        if (p < n) {
            w[h] = S.word[mirror][mirror ? r + n - 1 - p : r + p];
            cycle[h] = (int)((w[h] & kCycleOffset) >> 7);
            atomicMin(&S.firstPos[cycle[h]], p);
        }
    }
    __syncwarp();
    bool first[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int p = lane + 32 * h;
        first[h] = p < n && S.firstPos[cycle[h]] == p;
        if (first[h]) S.anchor[cycle[h]] = (int)((w[h] >> kTShift) & 63u);
    }
    const uint64_t firsts =
        (uint64_t)__ballot_sync(kFull, first[0]) | ((uint64_t)__ballot_sync(kFull, first[1]) << 32);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        value[h] = 0.f;
        if (lane + 32 * h < n) {
            const int fp = S.firstPos[cycle[h]];
            const int label = __popcll(firsts & ((2ull << fp) - 1ull));
            value[h] = value_of(hundredth, w[h],
                                __float_as_uint(__int2float_rn(label)) | (uint32_t)S.anchor[cycle[h]]);
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kWarps * 32) canonical_kernel(const CanonArgs A) {
    __shared__ uint32_t crc5[7][32];    // crc5[k][e]: 32 CRC steps on e << 5k
    __shared__ float hundredth[64];     // i / 100, and 0 for unoriented symbols
    __shared__ WarpSmem smem[kWarps];
    for (int i = threadIdx.x; i < 7 * 32; i += blockDim.x) {
        uint32_t c = (i >> 5) < 6 ? (uint32_t)(i & 31) << (5 * (i >> 5)) : (uint32_t)(i & 3) << 30;
        for (int k = 0; k < 32; ++k) c = (c >> 1) ^ (kPoly & (0u - (c & 1u)));
        crc5[i >> 5][i & 31] = c;
    }
    if (threadIdx.x < 64) hundredth[threadIdx.x] = __fdiv_rn(__int2float_rn((int)threadIdx.x), 100.0f);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    WarpSmem &S = smem[threadIdx.x >> 5];
    for (int row = blockIdx.x * kWarps + (threadIdx.x >> 5); row < A.count; row += gridDim.x * kWarps) {
        const int n = A.n[row];
        const uint8_t *src = A.spi + (size_t)row * 64;
        // validity: 2 <= n <= 63, spi a permutation of 0..n-1 without fixed points; a bad row
        // gets variant -1, hash 0 and a zero signature
        bool bad = n < 2 || n > kMaxN;
        uint32_t seen[2] = {0u, 0u};
        if (!bad) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int x = lane + 32 * h;
                if (x < n) {
                    const int s = src[x];
                    bad |= s >= n || s == x;
                    seen[(s >> 5) & 1] |= 1u << (s & 31);
                    S.spi[x] = (uint8_t)s;
                }
            }
        }
        const int distinct = __popc(__reduce_or_sync(kFull, seen[0])) + __popc(__reduce_or_sync(kFull, seen[1]));
        float *dst = A.sig + (size_t)row * 64;
        if (__any_sync(kFull, bad || distinct != n)) {
            dst[lane] = 0.f;
            dst[lane + 32] = 0.f;
            if (lane == 0) {
                A.hash[row] = 0;
                A.variant[row] = -1;
            }
            __syncwarp();
            continue;
        }
        __syncwarp();
        // cycle tables: each lane walks the cycles of its symbols (length <= n)
        int least[2], t[2], len[2], ascents[2];
        bool leads[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int x = lane + 32 * h;
            least[h] = x, t[h] = 0, len[h] = 1, ascents[h] = 0;
            if (x < n) {
                int at = 0, prev = x;
                for (int y = S.spi[x]; y != x && len[h] <= kMaxN; y = S.spi[y]) {
                    if (y < least[h]) least[h] = y, at = len[h];
                    ascents[h] += prev < y ? 1 : 0;
                    prev = y;
                    ++len[h];
                }
                ascents[h] += prev < x ? 1 : 0;
                t[h] = at == 0 ? 0 : len[h] - at;
            }
            leads[h] = x < n && least[h] == x;
        }
        const uint64_t leaders =
            (uint64_t)__ballot_sync(kFull, leads[0]) | ((uint64_t)__ballot_sync(kFull, leads[1]) << 32);
        const int cycles = __popcll(leaders);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int x = lane + 32 * h;
            if (x < n) {
                const uint32_t cycle = (uint32_t)__popcll(leaders & ((1ull << least[h]) - 1ull)) << 7;
                uint32_t fwd = cycle, mir = cycle;
                if (ascents[h] > 1) {
                    const uint32_t rest = ((uint32_t)len[h] << kLenShift) | (1u << kOrientedShift);
                    fwd |= rest | ((uint32_t)t[h] << kTShift);
                    // the mirror runs spi's cycle backwards
                    mir |= rest | ((uint32_t)(t[h] == 0 ? 0 : len[h] - t[h]) << kTShift);
                }
                S.word[0][x] = S.word[0][x + n] = fwd;
                S.word[1][x] = S.word[1][x + n] = mir;
            }
        }
        __syncwarp();
        // slot u < n: pi started at u; slot n + u: its mirror.  Slots go to lanes 32 at a time.
        int32_t hash[4];
        const int groups = (2 * n + 31) >> 5;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            hash[g] = INT32_MAX;
            const int u = lane + 32 * g;
            if (g < groups && u < 2 * n) {
                const bool mirror = u >= n;
                const int r = mirror ? u - n : u;
                const uint32_t *w = mirror ? &S.word[1][r + n - 1] : &S.word[0][r];
                const int dir = mirror ? -1 : 1;
                char *const met = reinterpret_cast<char *>(&S.met[0][lane]);
                for (int c = 0; c < cycles; ++c) *reinterpret_cast<uint32_t *>(met + (c << 7)) = 0u;
                float labels = 0.f;
                uint32_t crc = 0xFFFFFFFFu;
#pragma unroll 2
                for (int p = 0; p < n; ++p, w += dir) {
                    const uint32_t sym = *w;
                    uint32_t *const m = reinterpret_cast<uint32_t *>(met + (sym & kCycleOffset));
                    uint32_t e = *m;
                    if (e == 0u) {
                        labels = __fadd_rn(labels, 1.0f);
                        e = __float_as_uint(labels) | ((sym >> kTShift) & 63u);
                        *m = e;
                    }
                    const uint32_t x =
                        crc ^ __byte_perm(__float_as_uint(value_of(hundredth, sym, e)), 0u, 0x0123);
                    crc = crc5[0][x & 31u] ^ crc5[1][(x >> 5) & 31u] ^ crc5[2][(x >> 10) & 31u] ^
                          crc5[3][(x >> 15) & 31u] ^ crc5[4][(x >> 20) & 31u] ^ crc5[5][(x >> 25) & 31u] ^
                          crc5[6][x >> 30];
                }
                hash[g] = (int32_t)(crc ^ 0xFFFFFFFFu);
            }
        }
        // Configuration.getCanonical: the least hash, ties by Arrays.compare, then by variant
        int32_t least32 = min(min(hash[0], hash[1]), min(hash[2], hash[3]));
        least32 = __reduce_min_sync(kFull, least32);
        int bestV = -1;
        for (int from = 0;;) {
            // the first variant >= from with the least hash
            int v = INT32_MAX;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int u = lane + 32 * g;
                if (u < 2 * n && hash[g] == least32) {
                    const int mine = u >= n ? 2 * (u - n) + 1 : 2 * u;
                    if (mine >= from) v = min(v, mine);
                }
            }
            v = __reduce_min_sync(kFull, v);
            if (v == INT32_MAX) break;
            float value[2];
            build_row(S, hundredth, v, n, lane, value);
            bool take = bestV < 0;
            if (!take) {
                const bool d0 = lane < n && value[0] != S.best[lane];
                const bool d1 = lane + 32 < n && value[1] != S.best[lane + 32];
                const unsigned b0 = __ballot_sync(kFull, d0), b1 = __ballot_sync(kFull, d1);
                if (b0 | b1) {  // the least differing position decides
                    const bool less = b0 ? value[0] < S.best[lane] : value[1] < S.best[lane + 32];
                    take = __shfl_sync(kFull, (int)less, __ffs(b0 ? b0 : b1) - 1) != 0;
                }
                __syncwarp();
            }
            if (take) {
                bestV = v;
                S.best[lane] = value[0];
                S.best[lane + 32] = value[1];
            }
            __syncwarp();
            from = v + 1;
        }
        dst[lane] = S.best[lane];
        dst[lane + 32] = S.best[lane + 32];
        if (lane == 0) {
            A.hash[row] = least32;
            A.variant[row] = bestV;
        }
        __syncwarp();
    }
}

bool ok(cudaError_t e, std::string &err, const char *what) {
    if (e == cudaSuccess) return true;
    err = std::string(what) + ": CUDA error " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")";
    return false;
}

}  // namespace

int canonical_validate(const uint8_t *spi, const uint8_t *n, int count, std::string &err) {
    for (int r = 0; r < count; ++r) {
        const int m = n[r];
        if (m < 2 || m > kMaxN) {
            err = "tdp_canonical: row " + std::to_string(r) + ": n must be in 2..63";
            return -1;
        }
        uint64_t seen = 0;
        const uint8_t *s = spi + (size_t)r * 64;
        for (int x = 0; x < m; ++x) {
            if (s[x] >= m || ((seen >> s[x]) & 1ull) || s[x] == x) {
                err = "tdp_canonical: row " + std::to_string(r) +
                      ": spi must be a permutation of 0..n-1 without fixed points";
                return -1;
            }
            seen |= 1ull << s[x];
        }
    }
    return 0;
}

int canonical_device(const uint8_t *spiDev, const uint8_t *nDev, int count, float *sigDev, int32_t *hashDev,
                     int32_t *variantDev, cudaStream_t stream, std::string &err) {
    if (count < 0) {
        err = "tdp_canonical: count must be >= 0";
        return -1;
    }
    if (count == 0) return 0;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = (int)std::min<long long>(((long long)count + kWarps - 1) / kWarps, (long long)sms * 16 / kWarps * 4);
    CanonArgs A{spiDev, nDev, count, sigDev, hashDev, variantDev};
    canonical_kernel<<<blocks, kWarps * 32, 0, stream>>>(A);
    if (!ok(cudaGetLastError(), err, "canonical launch")) return -3;
    return 0;
}

}  // namespace tdp
