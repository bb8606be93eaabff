// Element-wise and row kernels of the move-ordering MLP (features, loss, optimiser, order).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <string>

#include "mlp.h"
#include "tdp_math.cuh"

namespace tdp {
namespace mlp {
namespace {

// Lexicographic index of (i<j<k) among the triples of 32 positions.
__host__ __device__ __forceinline__ int lex32(int i, int j, int k) {
    // triples before first index i, then before second index j (given i), then k
    int idx = 0;
    for (int a = 0; a < i; ++a) idx += (31 - a) * (30 - a) / 2;
    for (int b = i + 1; b < j; ++b) idx += 31 - b;
    return idx + (k - j - 1);
}

__global__ void features_kernel(const uint8_t *spi, const uint8_t *pi, const uint8_t *nArr, int rowStride,
                                int nStride, int count, __nv_bfloat16 *X) {
    const int s = blockIdx.x;
    if (s >= count) return;
    __shared__ uint8_t sp[32], pp[32], pos[32];
    __shared__ int hist[64];
    const int n = min((int)nArr[(size_t)s * nStride], 32);
    const int t = threadIdx.x;
    if (t < 32) {
        sp[t] = t < n ? spi[(size_t)s * rowStride + t] : (uint8_t)t;
        pp[t] = t < n ? pi[(size_t)s * rowStride + t] : (uint8_t)t;
    }
    if (t < 64) hist[t] = 0;
    __syncthreads();
    if (t < 32) pos[pp[t]] = (uint8_t)t;
    __syncthreads();
    // adjacency in pi-position coordinates: row i = position of x, column j = position of spi(x)
    for (int e = t; e < 1024; e += blockDim.x) {
        const int i = e >> 5, j = e & 31;
        float v = 0.f;
        if (i < n && j < n && pos[sp[pp[i]]] == j) v = 1.f;
        X[(size_t)s * kFeatures + e] = __float2bfloat16_rn(v);
    }
    if (t < n) {
        // cycle length of symbol t, counted once at the cycle's smallest symbol
        int len = 1, m = t, cur = sp[t];
        while (cur != t && len < 64) {
            m = min(m, (int)cur);
            cur = sp[cur];
            ++len;
        }
        if (m == t) atomicAdd(&hist[len - 1], 1);
    }
    __syncthreads();
    if (t < 64) X[(size_t)s * kFeatures + 1024 + t] = __float2bfloat16_rn((float)hist[t]);
}

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// The largest position k of every triple (i < j < k) of 32, in lexicographic order: column c of
// the logits is valid for a state of n symbols when kLast[c] < n.
struct LastTable {
    alignas(4) uint8_t k[kTriples];
    constexpr LastTable() : k() {
        int c = 0;
        for (int i = 0; i < 30; ++i)
            for (int j = i + 1; j < 31; ++j)
                for (int l = j + 1; l < 32; ++l) k[c++] = (uint8_t)l;
    }
};
__device__ const LastTable kLast = LastTable();

// One block of 128 threads per row; a thread owns the column pairs 2 threadIdx.x + 256 t and
// keeps them in registers, so the row is read once and each exponential is taken once.  The sum
// is that of 256 strided columns' sums, added within groups of 32 and then across the eight
// groups, in one fixed order.  Bound: the row's bytes (20 KB in, 10 KB out) and the divisions;
// the largest position of a column comes from a table (the decode of c into (i, j, k) in all
// three passes over the row was the whole cost before).  4,096 rows on one B200: 255 us with
// the decodes, 61 us with the table and one column per thread, 56 us in pairs.  top1 (or
// null) receives 1 where the row's greatest logit, over all triples, is the target's.
constexpr int kXentThreads = 128;
constexpr int kXentPer = kTriplesPadded / 256;  // column pairs per thread
static_assert(kTriples % 2 == 0 && kTriplesPadded % 256 == 0, "column pairs");

template <bool kTop1>
__global__ void __launch_bounds__(kXentThreads, 6) softmax_xent_kernel(const float *logits, int ld, const uint8_t *nArr,
                                                                    const int32_t *target, int rows,
                                                                    __nv_bfloat16 *dlogits, float *loss, float *top1) {
    const int r = blockIdx.x;
    if (r >= rows) return;
    const int n = nArr[r];
    __shared__ float red[8];
    const float *row = logits + (size_t)r * ld;
    const bool paired = ld % 2 == 0 && (reinterpret_cast<uintptr_t>(logits) & 7u) == 0 &&
                        (reinterpret_cast<uintptr_t>(dlogits) & 3u) == 0;
    float2 x[kXentPer];
    unsigned long long valid = 0ull;  // bits 2t, 2t + 1: the pair's columns
    float mx = -FLT_MAX;
#pragma unroll
    for (int t = 0; t < kXentPer; ++t) {
        const int c = 2 * (int)threadIdx.x + 256 * t;
        x[t] = make_float2(0.f, 0.f);
        if (c < kTriples) {
            if (paired) x[t] = *reinterpret_cast<const float2 *>(row + c);
            else x[t] = make_float2(row[c], row[c + 1]);
            const uint32_t last = *reinterpret_cast<const uint16_t *>(kLast.k + c);
            if ((int)(last & 0xFFu) < n) valid |= 1ull << (2 * t), mx = fmaxf(mx, x[t].x);
            if ((int)(last >> 8) < n) valid |= 2ull << (2 * t), mx = fmaxf(mx, x[t].y);
        }
    }
    const int tgt = target[r];
    // some logit ranks before the target's (greater, or equal and earlier); a target that is no
    // triple is never the greatest
    bool beaten = tgt < 0 || tgt >= kTriples;
    if (kTop1 && !beaten) {
        const float tv = row[tgt];
        const bool isNan = tv != tv;  // a NaN ranks as the greatest
#pragma unroll
        for (int t = 0; t < kXentPer; ++t) {
            const int c = 2 * (int)threadIdx.x + 256 * t;
            if (c < kTriples) {
                if (!isNan) {
                    beaten |= !(x[t].x <= tv) || (x[t].x == tv && c < tgt);
                    beaten |= !(x[t].y <= tv) || (x[t].y == tv && c + 1 < tgt);
                } else {
                    beaten |= (x[t].x != x[t].x && c < tgt) || (x[t].y != x[t].y && c + 1 < tgt);
                }
            }
        }
    }
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    beaten = __syncthreads_or(beaten);
    float2 part = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kXentPer; ++t) {
        x[t].x = __expf(x[t].x - mx);
        x[t].y = __expf(x[t].y - mx);
        if ((valid >> (2 * t)) & 1ull) part.x += x[t].x;
        if ((valid >> (2 * t)) & 2ull) part.y += x[t].y;
    }
    // a group of 32 columns is 16 lanes of pairs; its halving tree ends inside the pair
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        part.x += __shfl_xor_sync(0xFFFFFFFFu, part.x, o);
        part.y += __shfl_xor_sync(0xFFFFFFFFu, part.y, o);
    }
    if ((threadIdx.x & 15) == 0) red[threadIdx.x >> 4] = part.x + part.y;
    __syncthreads();
    // the eight groups' sums, halved as eight lanes of a warp would
    const float sum = ((red[0] + red[4]) + (red[2] + red[6])) + ((red[1] + red[5]) + (red[3] + red[7]));
    const float inv = 1.f / (float)rows;
#pragma unroll
    for (int t = 0; t < kXentPer; ++t) {
        const int c = 2 * (int)threadIdx.x + 256 * t;
        float2 g = make_float2(0.f, 0.f);
        if ((valid >> (2 * t)) & 1ull) g.x = x[t].x / sum - (c == tgt ? 1.f : 0.f);
        if ((valid >> (2 * t)) & 2ull) g.y = x[t].y / sum - (c + 1 == tgt ? 1.f : 0.f);
        __nv_bfloat16 *const dst = dlogits + (size_t)r * ld + c;
        if (paired && c + 1 < ld) {
            *reinterpret_cast<__nv_bfloat162 *>(dst) = __floats2bfloat162_rn(g.x * inv, g.y * inv);
        } else {
            if (c < ld) dst[0] = __float2bfloat16_rn(g.x * inv);
            if (c + 1 < ld) dst[1] = __float2bfloat16_rn(g.y * inv);
        }
    }
    for (int c = (int)threadIdx.x + kTriplesPadded; c < ld; c += kXentThreads)
        dlogits[(size_t)r * ld + c] = __float2bfloat16_rn(0.f);
    if (threadIdx.x == 0) {
        loss[r] = -(row[tgt] - mx - __logf(sum));
        if (kTop1) top1[r] = beaten ? 0.f : 1.f;
    }
}

__global__ void transpose_kernel(const __nv_bfloat16 *in, int rows, int cols, __nv_bfloat16 *out) {
    __shared__ __nv_bfloat16 tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int r = by + y, c = bx + threadIdx.x;
        if (r < rows && c < cols) tile[y][threadIdx.x] = in[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        const int r = bx + y, c = by + threadIdx.x;  // out is cols x rows
        if (r < cols && c < rows) out[(size_t)r * rows + c] = tile[threadIdx.x][y];
    }
}

__global__ void relu_backward_kernel(__nv_bfloat16 *grad, const __nv_bfloat16 *act, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        if (__bfloat162float(act[i]) <= 0.f) grad[i] = __float2bfloat16_rn(0.f);
}

// 32 columns per block, 32 rows at a time, then a reduction over the rows' warps.
__global__ void __launch_bounds__(1024) column_sums_kernel(const __nv_bfloat16 *grad, int rows, int cols, float *out) {
    __shared__ float part[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + x;
    float s = 0.f;
    if (c < cols)
        for (int r = y; r < rows; r += 32) s += __bfloat162float(grad[(size_t)r * cols + c]);
    part[y][x] = s;
    __syncthreads();
    const float v = warp_sum(part[x][y]);
    if (x == 0 && blockIdx.x * 32 + y < cols) out[blockIdx.x * 32 + y] = v;
}

// Bias gradients of one training step, all layers in one launch: partial column sums over spans
// of kSumRows rows.  A block takes 256 columns (32 threads of 8) and 8 rows at a time.
constexpr int kSumRows = 64;

struct ColumnSumArgs {
    const __nv_bfloat16 *grad[4];
    float *partials[4];  // [spans x cols]
    int cols[4], firstBlock[4];
    int rows;
};

__global__ void __launch_bounds__(256) column_partials_kernel(const __grid_constant__ ColumnSumArgs A) {
    __shared__ float part[8][256 + 8];
    int layer = 3;
    while (layer > 0 && (int)blockIdx.x < A.firstBlock[layer]) --layer;
    const int cols = A.cols[layer], x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int c = ((int)blockIdx.x - A.firstBlock[layer]) * 256 + x * 8;
    float s[8] = {};
    const int last = min((int)(blockIdx.y + 1) * kSumRows, A.rows);
#pragma unroll 4
    for (int r = (int)blockIdx.y * kSumRows + y; r < last; r += 8) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(A.grad[layer] + (size_t)r * cols + c));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            s[2 * j] += __uint_as_float(w[j] << 16);
            s[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) part[y][x * 8 + j] = s[j];
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) sum += part[q][threadIdx.x];
    A.partials[layer][(size_t)blockIdx.y * cols + ((int)blockIdx.x - A.firstBlock[layer]) * 256 + threadIdx.x] = sum;
}

__global__ void adam_kernel(float *master, __nv_bfloat16 *weight, const float *grad, float *m, float *v, size_t count,
                            float lr, float b1, float b2, float eps, float c1, float c2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const float g = grad[i];
        const float mi = b1 * m[i] + (1.f - b1) * g;
        const float vi = b2 * v[i] + (1.f - b2) * g * g;
        m[i] = mi;
        v[i] = vi;
        const float w = master[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        master[i] = w;
        weight[i] = __float2bfloat16_rn(w);
    }
}

// One Adam step of all weights and biases in one launch, four elements per thread.  The gradient
// is the sum of its partial products (spans of rows), added here so it never makes a pass of
// its own.  Block 0 reduces the rows' losses and top-1 hits to their means; the biases, whose
// sums have the most parts, come next, so the long chains start first.
struct AdamSegment {
    float *master;
    __nv_bfloat16 *weight;  // null for a bias
    const float *partials;  // [splits x count]
    float *m, *v;
    int splits, count, zeroFrom, firstBlock;  // elements from zeroFrom on are padding: weight 0
};
struct AdamArgs {
    AdamSegment seg[8];
    float lr, b1, b2, eps, c1, c2;
    const float *loss, *top1;
    float *means;
    int rows;
};
constexpr int kAdamPerBlock = 1024;

__global__ void __launch_bounds__(256) adam_step_kernel(const __grid_constant__ AdamArgs A) {
    if (blockIdx.x == 0) {
        __shared__ float sums[2][8];
        float l = 0.f, h = 0.f;
        for (int r = threadIdx.x; r < A.rows; r += 256) l += A.loss[r], h += A.top1[r];
        l = warp_sum(l);
        h = warp_sum(h);
        if ((threadIdx.x & 31) == 0) sums[0][threadIdx.x >> 5] = l, sums[1][threadIdx.x >> 5] = h;
        __syncthreads();
        if (threadIdx.x < 2) {
            float s = 0.f;
            for (int w = 0; w < 8; ++w) s += sums[threadIdx.x][w];
            A.means[threadIdx.x] = s / (float)A.rows;
        }
        return;
    }
    int k = 7;
    while (k > 0 && (int)blockIdx.x < A.seg[k].firstBlock) --k;
    const AdamSegment &S = A.seg[k];
    const int i = ((int)blockIdx.x - S.firstBlock) * kAdamPerBlock + (int)threadIdx.x * 4;
    if (i >= S.count) return;
    float4 g = *reinterpret_cast<const float4 *>(S.partials + i);
#pragma unroll 8
    for (int q = 1; q < S.splits; ++q) {
        const float4 t = *reinterpret_cast<const float4 *>(S.partials + (size_t)q * S.count + i);
        g.x += t.x, g.y += t.y, g.z += t.z, g.w += t.w;
    }
    float4 m = *reinterpret_cast<const float4 *>(S.m + i), v = *reinterpret_cast<const float4 *>(S.v + i);
    float4 w = *reinterpret_cast<const float4 *>(S.master + i);
    auto step = [&](float gj, float &mj, float &vj, float &wj, int at) {
        mj = A.b1 * mj + (1.f - A.b1) * gj;
        vj = A.b2 * vj + (1.f - A.b2) * gj * gj;
        wj = at < S.zeroFrom ? wj - A.lr * (mj / A.c1) / (sqrtf(vj / A.c2) + A.eps) : 0.f;
    };
    step(g.x, m.x, v.x, w.x, i);
    step(g.y, m.y, v.y, w.y, i + 1);
    step(g.z, m.z, v.z, w.z, i + 2);
    step(g.w, m.w, v.w, w.w, i + 3);
    *reinterpret_cast<float4 *>(S.m + i) = m;
    *reinterpret_cast<float4 *>(S.v + i) = v;
    *reinterpret_cast<float4 *>(S.master + i) = w;
    if (S.weight) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(w.x, w.y), hi = __floats2bfloat162_rn(w.z, w.w);
        *reinterpret_cast<uint2 *>(S.weight + i) =
            make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
    }
}

// One block per instance: bitonic sort of (score, n-space index) pairs, 8192 slots.
__global__ void __launch_bounds__(1024) order_kernel(const float *scores, int ld, const uint8_t *nArr, int nStride,
                                                      int count, uint16_t *order, int orderStride) {
    const int s = blockIdx.x;
    if (s >= count) return;
    __shared__ float key[8192];
    __shared__ uint16_t val[8192];
    const int n = min((int)nArr[(size_t)s * nStride], 32);
    const int T = combinations3(n);
    int size = 1;
    while (size < T) size <<= 1;
    for (int t = threadIdx.x; t < size; t += blockDim.x) {
        float k = -FLT_MAX;
        uint16_t idx = 0xFFFF;
        if (t < T) {
            // n-space lexicographic index t -> (i, j, k)
            int rem = t, i = 0;
            while (i < n - 3 && rem >= (n - 1 - i) * (n - 2 - i) / 2) rem -= (n - 1 - i) * (n - 2 - i) / 2, ++i;
            int j = i + 1;
            while (j < n - 2 && rem >= n - 1 - j) rem -= n - 1 - j, ++j;
            const int kk = j + 1 + rem;
            k = scores[(size_t)s * ld + lex32(i, j, kk)];
            idx = (uint16_t)t;
        }
        key[t] = k;
        val[t] = idx;
    }
    __syncthreads();
    for (int len = 2; len <= size; len <<= 1) {
        for (int stride = len >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < size; t += blockDim.x) {
                const int partner = t ^ stride;
                if (partner > t) {
                    const bool desc = ((t & len) == 0);  // descending overall
                    const float a = key[t], b = key[partner];
                    const bool swap = desc ? (a < b || (a == b && val[t] > val[partner]))
                                           : (a > b || (a == b && val[t] < val[partner]));
                    if (swap) {
                        key[t] = b;
                        key[partner] = a;
                        const uint16_t u = val[t];
                        val[t] = val[partner];
                        val[partner] = u;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int t = threadIdx.x; t < T; t += blockDim.x) order[(size_t)s * orderStride + t] = val[t];
}

// First-level states of the learned order: for instance s and rank r < K1 of its root
// order, the state after the root child order[r] (positions i<j<k of the root's pi array):
// spi' = spi o (a b c)^-1 with a, b, c = pi[i], pi[j], pi[k] (sorting_search.cu:543-555) and
// pi' = pi with [i,j) and [j,k) swapped (transposition.cuh:5-19).  Ranks past the root's
// triple count get n = 0.
__global__ void level1_states_kernel(const uint8_t *spi, const uint8_t *pi, const uint8_t *nArr, int rowStride,
                                     int nStride, int count, const uint16_t *order, int orderStride, int k1,
                                     uint8_t *outSpi, uint8_t *outPi, uint8_t *outN) {
    const int row = blockIdx.x;  // s * k1 + r
    const int s = row / k1, r = row % k1;
    if (s >= count) return;
    const int n = min((int)nArr[(size_t)s * nStride], 32);
    const int T = combinations3(n);
    const int p = threadIdx.x;  // 32 threads: one position / symbol each
    __shared__ int ijk[3];
    if (p == 0) {
        int rem = (r < T) ? (int)order[(size_t)s * orderStride + r] : 0, i = 0;
        while (i < n - 3 && rem >= (n - 1 - i) * (n - 2 - i) / 2) rem -= (n - 1 - i) * (n - 2 - i) / 2, ++i;
        int j = i + 1;
        while (j < n - 2 && rem >= n - 1 - j) rem -= n - 1 - j, ++j;
        ijk[0] = i;
        ijk[1] = j;
        ijk[2] = j + 1 + rem;
    }
    __syncthreads();
    const uint8_t *sp = spi + (size_t)s * rowStride, *pp = pi + (size_t)s * rowStride;
    uint8_t *os = outSpi + (size_t)row * 64, *op = outPi + (size_t)row * 64;
    const bool valid = r < T;
    if (p == 0) outN[row] = valid ? (uint8_t)n : (uint8_t)0;
    if (!valid || p >= n) {
        if (p < 32) os[p] = op[p] = 0;
        return;
    }
    const int i = ijk[0], j = ijk[1], k = ijk[2];
    const int a = pp[i], b = pp[j], c = pp[k];
    uint8_t v = sp[p];
    if (p == a) v = sp[c];
    if (p == b) v = sp[a];
    if (p == c) v = sp[b];
    os[p] = v;
    op[p] = pp[block_swap_src(p, i, j, k)];
}

// The K highest-scoring triples of each state (n-space lexicographic indices, ties to the
// smaller index, the order of order_kernel), by K rounds of a block arg-max; 0xFFFF pads
// states with fewer than K triples.
__global__ void __launch_bounds__(256) topk_kernel(const float *scores, int ld, const uint8_t *nArr, int nStride,
                                                   int count, int k, uint16_t *out, int outStride) {
    constexpr int kPer = 20;  // 256 * 20 >= C(32,3) = 4960
    const int s = blockIdx.x;
    if (s >= count) return;
    const int n = min((int)nArr[(size_t)s * nStride], 32);
    const int T = combinations3(n);
    float key[kPer];
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
        const int t = threadIdx.x + 256 * e;
        key[e] = -FLT_MAX;
        if (t < T) {
            int rem = t, i = 0;
            while (i < n - 3 && rem >= (n - 1 - i) * (n - 2 - i) / 2) rem -= (n - 1 - i) * (n - 2 - i) / 2, ++i;
            int j = i + 1;
            while (j < n - 2 && rem >= n - 1 - j) rem -= n - 1 - j, ++j;
            key[e] = scores[(size_t)s * ld + lex32(i, j, j + 1 + rem)];
        }
    }
    unsigned taken = 0;
    __shared__ float bestKey[8];
    __shared__ int bestIdx[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int round = 0; round < k; ++round) {
        float bk = -FLT_MAX;
        int bi = 0x7FFFFFFF;
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int t = threadIdx.x + 256 * e;
            if (t < T && !((taken >> e) & 1u) && (key[e] > bk || (key[e] == bk && t < bi))) {
                bk = key[e];
                bi = t;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ok = __shfl_xor_sync(0xFFFFFFFFu, bk, o);
            const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
            if (ok > bk || (ok == bk && oi < bi)) {
                bk = ok;
                bi = oi;
            }
        }
        if (lane == 0) {
            bestKey[warp] = bk;
            bestIdx[warp] = bi;
        }
        __syncthreads();
        bk = bestKey[0];
        bi = bestIdx[0];
        for (int w = 1; w < 8; ++w)
            if (bestKey[w] > bk || (bestKey[w] == bk && bestIdx[w] < bi)) {
                bk = bestKey[w];
                bi = bestIdx[w];
            }
        __syncthreads();
        if (threadIdx.x == 0) out[(size_t)s * outStride + round] = bi < T ? (uint16_t)bi : (uint16_t)0xFFFF;
        if (bi < T && (bi & 255) == (int)threadIdx.x) taken |= 1u << (bi >> 8);
    }
}

}  // namespace

void build_features(const uint8_t *spi, const uint8_t *pi, const uint8_t *n, int rowStride, int nStride, int count,
                    __nv_bfloat16 *X, cudaStream_t stream) {
    if (count > 0) features_kernel<<<count, 128, 0, stream>>>(spi, pi, n, rowStride, nStride, count, X);
}

void softmax_xent(const float *logits, int ld, const uint8_t *n, const int32_t *target, int rows,
                  __nv_bfloat16 *dlogits, float *loss, cudaStream_t stream) {
    if (rows > 0)
        softmax_xent_kernel<false><<<rows, kXentThreads, 0, stream>>>(logits, ld, n, target, rows, dlogits, loss, nullptr);
}

void transpose_bf16(const __nv_bfloat16 *in, int rows, int cols, __nv_bfloat16 *out, cudaStream_t stream) {
    const dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
    transpose_kernel<<<grid, block, 0, stream>>>(in, rows, cols, out);
}

void relu_backward(__nv_bfloat16 *grad, const __nv_bfloat16 *act, size_t count, cudaStream_t stream) {
    relu_backward_kernel<<<1184, 256, 0, stream>>>(grad, act, count);
}

void column_sums(const __nv_bfloat16 *grad, int rows, int cols, float *out, cudaStream_t stream) {
    column_sums_kernel<<<(cols + 31) / 32, 1024, 0, stream>>>(grad, rows, cols, out);
}

void adam_step(float *master, __nv_bfloat16 *weight, const float *grad, float *m, float *v, size_t count, float lr,
               float beta1, float beta2, float eps, int step, cudaStream_t stream) {
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    adam_kernel<<<1184, 256, 0, stream>>>(master, weight, grad, m, v, count, lr, beta1, beta2, eps, c1, c2);
}

void order_by_score(const float *scores, int ld, const uint8_t *n, int nStride, int count, uint16_t *order,
                    int orderStride, cudaStream_t stream) {
    if (count > 0) order_kernel<<<count, 1024, 0, stream>>>(scores, ld, n, nStride, count, order, orderStride);
}

void level1_states(const uint8_t *spi, const uint8_t *pi, const uint8_t *n, int rowStride, int nStride, int count,
                   const uint16_t *order, int orderStride, int k1, uint8_t *outSpi, uint8_t *outPi, uint8_t *outN,
                   cudaStream_t stream) {
    if (count > 0 && k1 > 0)
        level1_states_kernel<<<count * k1, 32, 0, stream>>>(spi, pi, n, rowStride, nStride, count, order, orderStride,
                                                            k1, outSpi, outPi, outN);
}

void top_k(const float *scores, int ld, const uint8_t *n, int nStride, int count, int k, uint16_t *out, int outStride,
           cudaStream_t stream) {
    if (count > 0 && k > 0) topk_kernel<<<count, 256, 0, stream>>>(scores, ld, n, nStride, count, k, out, outStride);
}

// ---------------------------------------------------------------- one training step
namespace {

constexpr int kLayers = 4;
constexpr int kOut[kLayers] = {kHidden, kHidden, kHidden, kTriplesPadded};
constexpr int kIn[kLayers] = {kFeatures, kHidden, kHidden, kHidden};

// Scratch of a step, carved from one caller-owned buffer in 256-byte pieces.
struct TrainScratch {
    __nv_bfloat16 *act[kLayers];   // act[l]: input of layer l (act[0] unused: x)
    __nv_bfloat16 *grad[kLayers];  // grad[l]: gradient of layer l's output
    float *logits, *loss, *top1;
    float *weightParts[kLayers], *biasParts[kLayers];
    size_t bytes;
};

TrainScratch carve(uint8_t *base, int rows) {
    TrainScratch S{};
    size_t at = 0;
    auto take = [&](size_t bytes) {
        uint8_t *p = base + at;
        at += (bytes + 255) & ~(size_t)255;
        return static_cast<void *>(p);
    };
    const size_t R = (size_t)rows;
    const int spans = (rows + kSumRows - 1) / kSumRows;
    for (int l = 1; l < kLayers; ++l) S.act[l] = static_cast<__nv_bfloat16 *>(take(R * kHidden * 2));
    S.logits = static_cast<float *>(take(R * kTriplesPadded * 4));
    for (int l = 0; l < kLayers; ++l) {
        S.grad[l] = static_cast<__nv_bfloat16 *>(take(R * kOut[l] * 2));
        S.weightParts[l] =
            static_cast<float *>(take((size_t)weight_grad_splits(rows, kOut[l], kIn[l]) * kOut[l] * kIn[l] * 4));
        S.biasParts[l] = static_cast<float *>(take((size_t)spans * kOut[l] * 4));
    }
    S.loss = static_cast<float *>(take(R * 4));
    S.top1 = static_cast<float *>(take(R * 4));
    S.bytes = at;
    return S;
}

}  // namespace

size_t train_workspace(int rows) { return carve(nullptr, rows).bytes; }

int train_step(const TrainStep &T, int *errorFlag, cudaStream_t stream, std::string &err) {
    const int rows = T.rows;
    if (rows % 8 != 0) {
        err = "gemm operand must be 16-byte aligned with a row length that is a multiple of 8";
        return -1;
    }
    const TrainScratch S = carve(static_cast<uint8_t *>(T.workspace), rows);
    if (T.workspaceBytes < S.bytes) {
        err = "tdp_mlp_train_step: workspace too small";
        return -1;
    }
    const __nv_bfloat16 *act[kLayers] = {T.x, S.act[1], S.act[2], S.act[3]};
    for (int l = 0; l < kLayers; ++l) {
        void *out = l < 3 ? static_cast<void *>(S.act[l + 1]) : static_cast<void *>(S.logits);
        const int rc = gemm_bf16(act[l], T.weight[l], rows, kOut[l], kIn[l], T.bias[l], l < 3, out, l == 3, kOut[l],
                                 errorFlag, stream, err);
        if (rc != 0) return rc;
    }
    softmax_xent_kernel<true><<<rows, kXentThreads, 0, stream>>>(S.logits, kTriplesPadded, T.n, T.target, rows, S.grad[3],
                                                        S.loss, S.top1);
    for (int l = kLayers - 1; l >= 0; --l) {
        int rc = gemm_weight_grad(S.grad[l], act[l], rows, kOut[l], kIn[l], S.weightParts[l], errorFlag, stream, err);
        if (rc == 0 && l > 0)
            rc = gemm_input_grad(S.grad[l], T.weight[l], rows, kOut[l], kIn[l], act[l], S.grad[l - 1], errorFlag,
                                 stream, err);
        if (rc != 0) return rc;
    }
    const int spans = (rows + kSumRows - 1) / kSumRows;
    ColumnSumArgs C{};
    C.rows = rows;
    int blocks = 0;
    for (int l = 0; l < kLayers; ++l) {
        C.grad[l] = S.grad[l];
        C.partials[l] = S.biasParts[l];
        C.cols[l] = kOut[l];
        C.firstBlock[l] = blocks;
        blocks += kOut[l] / 256;
    }
    column_partials_kernel<<<dim3(blocks, spans), 256, 0, stream>>>(C);
    AdamArgs A{};
    A.lr = T.lr;
    A.b1 = T.beta1;
    A.b2 = T.beta2;
    A.eps = T.eps;
    A.c1 = 1.f - powf(T.beta1, (float)T.step);
    A.c2 = 1.f - powf(T.beta2, (float)T.step);
    A.loss = S.loss;
    A.top1 = S.top1;
    A.means = T.means;
    A.rows = rows;
    blocks = 1;
    for (int at = 0; at < 2 * kLayers; ++at) {
        const int k = (at + kLayers) % (2 * kLayers), l = k % kLayers;
        const bool bias = k >= kLayers;
        AdamSegment &G = A.seg[at];
        G.master = bias ? T.bias[l] : T.master[l];
        G.weight = bias ? nullptr : T.weight[l];
        G.partials = bias ? S.biasParts[l] : S.weightParts[l];
        G.m = T.m[k];
        G.v = T.v[k];
        G.splits = bias ? spans : weight_grad_splits(rows, kOut[l], kIn[l]);
        G.count = bias ? kOut[l] : kOut[l] * kIn[l];
        G.zeroFrom = !bias && l == 3 ? kTriples * kHidden : G.count;
        G.firstBlock = blocks;
        blocks += (G.count + kAdamPerBlock - 1) / kAdamPerBlock;
    }
    adam_step_kernel<<<blocks, 256, 0, stream>>>(A);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("tdp_mlp_train_step: ") + cudaGetErrorString(e);
        return -3;
    }
    return 0;
}

}  // namespace mlp
}  // namespace tdp
