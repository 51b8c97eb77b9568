// Learned warm start: a per-cube MLP  F -> 64 -> 64 -> 1  (F = nbins + 5 inputs:
// the histogram normalised by its total, depth / 21, the cube's position inside
// its chunk's node, and the histogram's median indicator), ReLU hidden layers,
// linear output predicting the converged u minus the median indicator (the
// reference's own start), so that the warm start is median + network.  BF16
// weights and activations, FP32 accumulation, on the tensor cores: inference with
// tcgen05.mma over 128-row tiles (k_forward), the training backward pass with
// mma.sync m16n8k16 (row.col), whose fragments its two layers and their
// transposes share in registers; it keeps FP32 accuracy by splitting its FP32
// factors into exact bf16 parts (k_mlp_grad).
//
// Fragment layouts of mma.m16n8k16 (lane t, g = t / 4, c = t % 4):
//   A (16x16, row-major): a0 = A[g][2c..2c+1], a1 = A[g+8][2c..], a2 = A[g][2c+8..], a3 = A[g+8][2c+8..]
//   B (16x8, col-major):  b0 = B[2c..2c+1][g],   b1 = B[2c+8..2c+9][g]
//   C/D (16x8, f32):      c0 = C[g][2c], c1 = C[g][2c+1], c2 = C[g+8][2c], c3 = C[g+8][2c+1]
// so the C tiles of output columns 16j..16j+15 are, packed to bf16, exactly the
// A fragment of input chunk j of the next layer.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_bf16.h>

#include "common.cuh"

namespace tgvg {

constexpr int MLP_K1 = 16;  // padded input width
constexpr int MLP_H = 64;
// fp32 master parameters
constexpr int P_W1 = 0;                  // W1[k][j], k < 16, j < 64
constexpr int P_B1 = P_W1 + MLP_K1 * MLP_H;
constexpr int P_W2 = P_B1 + MLP_H;       // W2[k][j]
constexpr int P_B2 = P_W2 + MLP_H * MLP_H;
constexpr int P_W3 = P_B2 + MLP_H;       // W3[k]
constexpr int P_B3 = P_W3 + MLP_H;
constexpr int P_N = P_B3 + 1;            // 5249
// bf16 B fragments: 64 words per (k-chunk, n-tile)
constexpr int F_W1 = 0;                  // 1 x 8 tiles
constexpr int F_W2 = F_W1 + 8 * 64;      // 4 x 8 tiles
constexpr int F_W3 = F_W2 + 32 * 64;     // 4 x 1 tile (column 0 = W3)
constexpr int F_N = F_W3 + 4 * 64;       // 2816 words

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ void mma_bf16(float& d0, float& d1, float& d2, float& d3, uint32_t a0, uint32_t a1,
                                         uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d0), "+f"(d1), "+f"(d2), "+f"(d3)
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// An FP32 value as the exact sum of three bf16 parts (8 significant bits each,
// cut off, not rounded, so nothing overflows); the first part alone holds an
// infinity, or a NaN as arithmetic makes them (payload in the upper half).
__device__ __forceinline__ void split_bf16(float v, float& hi, float& mid, float& lo) {
    hi = __uint_as_float(__float_as_uint(v) & 0xffff0000u);
    const float r = isfinite(v) ? v - hi : 0.f;
    mid = __uint_as_float(__float_as_uint(r) & 0xffff0000u);
    lo = r - mid;
}
// The weights as inference takes them (k_forward): per layer 64, 64 and 16 columns of
// 32, 80 and 80 inputs, three of them the bias's parts; element (k, column j) at
// (k / 8) (columns x 16 B) + j x 16 B + (k % 8) x 2 B.
constexpr int TC_B1 = 0, TC_B2 = TC_B1 + 64 * 32 * 2, TC_B3 = TC_B2 + 64 * 80 * 2, TC_W = TC_B3 + 16 * 80 * 2;
__device__ __forceinline__ __nv_bfloat16 tc_weight(const float* __restrict__ prm, int e) {
    const bool l1 = e < TC_B2 / 2, l3 = e >= TC_B3 / 2;
    e -= l3 ? TC_B3 / 2 : (l1 ? 0 : TC_B2 / 2);
    const int columns = l3 ? 16 : 64, width = l1 ? MLP_K1 : MLP_H;
    const int k = e / (columns * 8) * 8 + e % 8, j = e / 8 % columns;
    if (k >= width + 3 || (l3 && j > 0)) return __float2bfloat16_rn(0.f);
    if (k < width) return __float2bfloat16_rn(prm[l3 ? P_W3 + k : (l1 ? P_W1 : P_W2) + k * MLP_H + j]);
    float p[3];
    const float b = prm[(l3 ? P_B3 : (l1 ? P_B1 : P_B2)) + j];
    split_bf16(b, p[0], p[1], p[2]);
    if (isnan(b)) p[0] = b;  // cut off, a payload in the low half would leave an infinity
    return __float2bfloat16_rn(p[k - width]);  // exact: a bf16 value
}

// Weight fragments, inference's weights and a bf16-rounded float copy (used by the
// backward pass) from the fp32 master parameters.
__global__ void k_mlp_pack(const float* __restrict__ prm, uint32_t* __restrict__ frag, float* __restrict__ wr,
                           __nv_bfloat16* __restrict__ tc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < TC_W / 2) tc[t] = tc_weight(prm, t);
    if (t < P_N) wr[t] = bf16r(prm[t]);
    if (t >= F_N) return;
    const int tile = t / 64, w = t % 64, lane = w / 2, half = w % 2;
    const int g = lane / 4, c = lane % 4;
    int kc, nt, base;
    if (t < F_W2) { kc = 0; nt = tile; base = P_W1; }
    else if (t < F_W3) { kc = (tile - 8) / 8; nt = (tile - 8) % 8; base = P_W2; }
    else { kc = tile - 40; nt = 0; base = P_W3; }
    const int k = kc * 16 + 2 * c + 8 * half;
    const int n = nt * 8 + g;
    float lo, hi;
    if (base == P_W3) {
        lo = n == 0 ? prm[P_W3 + k] : 0.f;
        hi = n == 0 ? prm[P_W3 + k + 1] : 0.f;
    } else {
        lo = prm[base + k * MLP_H + n];
        hi = prm[base + (k + 1) * MLP_H + n];
    }
    frag[t] = pack_bf16(lo, hi);
}

// A chunk's node as the features need it: the index range of its cubes, the
// fine-grid coordinates of the node's corner and 1 / its edge (a power of two).
struct LeafBox {
    uint32_t first, last;
    uint32_t x, y, z;
    float inv_size;
};
__host__ __device__ __forceinline__ LeafBox leaf_box(const tgvg_leaf& l) {
    const uint64_t key = (uint64_t(l.hi) << 32) | l.lo;
    const int d = l.depth < 0 ? 0 : (l.depth > 21 ? 21 : l.depth);
    return LeafBox{l.first_idx, l.last_idx, gather3(key), gather3(key >> 1), gather3(key >> 2),
                   1.0f / (float)(1u << (21 - d))};
}

// depth / 21 and the median indicator of a first half bin, tabled once per block.
struct FeatureTables {
    float depth[22];
    float med[16];  // [km + 1]; 0: no bin (only a total that wraps 32 bits)
};
template <int NB>
__device__ __forceinline__ void feature_tables(FeatureTables& t) {
    if (threadIdx.x < 22) t.depth[threadIdx.x] = threadIdx.x / 21.0f;
    if (threadIdx.x <= NB)
        t.med[threadIdx.x] = fadd(-1.0f, fdiv(fadd((float)((int)threadIdx.x - 1), 0.5f), NB / 2.0f));
}

// One cube's 16 features as eight bf16 pairs: bins / total, depth / 21, the
// position of the cube's centre inside its chunk's node (the root without one)
// and the median indicator, whose FP32 value (the reference's,
// src/histogram.cpp:12-31; 0 when empty) is returned.  b: the histogram row.
template <int NB>
__device__ __forceinline__ float feature_row(const uint32_t (&b)[NB], const uint4& cb, const LeafBox& box,
                                             const FeatureTables& tab, uint32_t (&out)[8]) {
    float f[MLP_K1];
#pragma unroll
    for (int k = 0; k < MLP_K1; ++k) f[k] = 0.f;
    uint32_t tot = 0;
#pragma unroll
    for (int k = 0; k < NB; ++k) tot += b[k];
    const float inv = tot ? 1.0f / (float)tot : 0.f;
    uint32_t cum = 0;
    int km = -1;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        f[k] = (float)b[k] * inv;
        cum += b[k];
        if (km < 0 && cum * 2 >= tot) km = k;
    }
    const float m = tot ? tab.med[km + 1] : 0.0f;
    f[NB + 4] = m;
    const uint64_t key = (uint64_t(cb.x) << 32) | cb.y;
    const int d = min(21, max(0, (int)cb.w));
    f[NB] = tab.depth[d];
    const float half = 0.5f * (float)(1u << (21 - d));
    // the node's edge is a power of two: the product with its inverse is the quotient
    f[NB + 1] = fminf(fmaxf(((float)gather3(key) - (float)box.x + half) * box.inv_size, 0.f), 1.f);
    f[NB + 2] = fminf(fmaxf(((float)gather3(key >> 1) - (float)box.y + half) * box.inv_size, 0.f), 1.f);
    f[NB + 3] = fminf(fmaxf(((float)gather3(key >> 2) - (float)box.z + half) * box.inv_size, 0.f), 1.f);
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = pack_bf16(f[2 * k], f[2 * k + 1]);
    return m;
}

// A histogram row in registers; vec: rows start on 16 (8 bins) or 8 bytes (10 bins).
template <int NB>
__device__ __forceinline__ void load_bins(const uint32_t* __restrict__ row, bool vec, uint32_t (&b)[NB]) {
    if (vec) {
        if (NB == 8) {
#pragma unroll
            for (int k = 0; k < NB; k += 4) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + k));
                b[k] = v.x; b[k + 1] = v.y; b[k + 2] = v.z; b[k + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < NB; k += 2) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + k));
                b[k] = v.x; b[k + 1] = v.y;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < NB; ++k) b[k] = __ldg(row + k);
    }
}
template <int NB>
__device__ __forceinline__ bool bins_aligned(const uint32_t* hists) {
    return ((uintptr_t)hists & (NB == 8 ? 15 : 7)) == 0;
}

template <int NB>
__global__ void k_mlp_features(int n, const uint4* __restrict__ cubes, const uint32_t* __restrict__ hists,
                               const int* __restrict__ leaf_id, const tgvg_leaf* __restrict__ leaves,
                               uint32_t* __restrict__ X) {
    __shared__ FeatureTables tab;
    feature_tables<NB>(tab);
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t b[NB], w[8];
    load_bins<NB>(hists + (size_t)i * NB, bins_aligned<NB>(hists), b);
    const int l = leaf_id ? leaf_id[i] : -1;
    feature_row<NB>(b, cubes[i], leaf_box(l >= 0 ? leaves[l] : tgvg_leaf{0, 0, 0, 0, 0}), tab, w);
    uint32_t* out = X + (size_t)i * 8;
#pragma unroll
    for (int k = 0; k < 8; ++k) out[k] = w[k];
}

__global__ void k_leaf_id(int n, int nleaf, const tgvg_leaf* __restrict__ leaves, int* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int id = -1;
    for (int l = 0; l < nleaf; ++l)
        if ((uint32_t)i >= leaves[l].first_idx && (uint32_t)i <= leaves[l].last_idx) { id = l; break; }
    out[i] = id;
}

// The first hidden layer over one warp's T 16-row tiles whose inputs are the A
// fragments a[t]: h receives the bf16 activations as the A fragments of the next
// layer (h[t][kc][0..3]: rows g / g+8 of columns 16 kc + 2c.., then of
// 16 kc + 8 + 2c..).  The tiles share the weight fragments' reads.
template <int T>
__device__ __forceinline__ void mlp_layer1(const uint32_t (&a)[T][4], const uint32_t* __restrict__ sfrag,
                                           const float* __restrict__ sbias, uint32_t (&h)[T][4][4]) {
    const int lane = threadIdx.x & 31, c = lane & 3;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float2 b = *reinterpret_cast<const float2*>(sbias + nt * 8 + 2 * c);
        const uint2 w = *reinterpret_cast<const uint2*>(sfrag + F_W1 + nt * 64 + lane * 2);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            float d0 = b.x, d1 = b.y, d2 = b.x, d3 = b.y;
            mma_bf16(d0, d1, d2, d3, a[t][0], a[t][1], a[t][2], a[t][3], w.x, w.y);
            h[t][nt >> 1][(nt & 1) * 2] = pack_bf16(fmaxf(d0, 0.f), fmaxf(d1, 0.f));
            h[t][nt >> 1][(nt & 1) * 2 + 1] = pack_bf16(fmaxf(d2, 0.f), fmaxf(d3, 0.f));
        }
    }
}

// Columns 16 k2 .. 16 k2 + 15 of the second hidden layer: one A fragment per tile.
template <int T>
__device__ __forceinline__ void mlp_layer2(int k2, const uint32_t (&h)[T][4][4], const uint32_t* __restrict__ sfrag,
                                           const float* __restrict__ sbias, uint32_t (&h2)[T][4]) {
    const int lane = threadIdx.x & 31, c = lane & 3;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int nt = 2 * k2 + half;
        const float2 b = *reinterpret_cast<const float2*>(sbias + 64 + nt * 8 + 2 * c);
        float d[T][4];
#pragma unroll
        for (int t = 0; t < T; ++t) { d[t][0] = d[t][2] = b.x; d[t][1] = d[t][3] = b.y; }
#pragma unroll
        for (int kc = 0; kc < 4; ++kc) {
            const uint2 w = *reinterpret_cast<const uint2*>(sfrag + F_W2 + (kc * 8 + nt) * 64 + lane * 2);
#pragma unroll
            for (int t = 0; t < T; ++t)
                mma_bf16(d[t][0], d[t][1], d[t][2], d[t][3], h[t][kc][0], h[t][kc][1], h[t][kc][2], h[t][kc][3], w.x, w.y);
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
            h2[t][half * 2] = pack_bf16(fmaxf(d[t][0], 0.f), fmaxf(d[t][1], 0.f));
            h2[t][half * 2 + 1] = pack_bf16(fmaxf(d[t][2], 0.f), fmaxf(d[t][3], 0.f));
        }
    }
}

// The second hidden layer and the output layer, 16 hidden columns at a time (an
// output product takes each as it is ready, in column order): y[t] for rows g
// and g+8 of tile t, valid on lanes with c == 0.  With h2s the activations are
// kept there.
template <int T>
__device__ __forceinline__ void mlp_rest(const uint32_t (&h)[T][4][4], const uint32_t* __restrict__ sfrag,
                                         const float* __restrict__ sbias, float (&y)[T][2],
                                         uint32_t (*h2s)[4][4] = nullptr) {
    const int lane = threadIdx.x & 31, c = lane & 3;
    const float b3 = (c == 0) ? sbias[128] : 0.f;
    float d[T][4];
#pragma unroll
    for (int t = 0; t < T; ++t) { d[t][0] = d[t][2] = b3; d[t][1] = d[t][3] = 0.f; }
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
        uint32_t h2[T][4];
        mlp_layer2<T>(kc, h, sfrag, sbias, h2);
        const uint2 w = *reinterpret_cast<const uint2*>(sfrag + F_W3 + kc * 64 + lane * 2);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            mma_bf16(d[t][0], d[t][1], d[t][2], d[t][3], h2[t][0], h2[t][1], h2[t][2], h2[t][3], w.x, w.y);
            if (h2s) {
#pragma unroll
                for (int e = 0; e < 4; ++e) h2s[t][kc][e] = h2[t][e];
            }
        }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) { y[t][0] = d[t][0]; y[t][1] = d[t][2]; }
}

__device__ __forceinline__ void load_net(const uint32_t* __restrict__ frag, const float* __restrict__ prm,
                                         uint32_t* sfrag, float* sbias) {
    for (int w = threadIdx.x; w < F_N; w += blockDim.x) sfrag[w] = frag[w];
    for (int k = threadIdx.x; k < 64; k += blockDim.x) {
        sbias[k] = prm[P_B1 + k];
        sbias[64 + k] = prm[P_B2 + k];
    }
    if (threadIdx.x == 0) sbias[128] = prm[P_B3];
    __syncthreads();
}

// Two values whose low 16 bits are zero, as a bf16 pair.
__device__ __forceinline__ uint32_t pack_top(float a, float b) {
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// ---- inference on the fifth-generation tensor cores -----------------------------
// The network over tiles of 128 rows with tcgen05.mma: a group of four warps owns a
// tile, each of its threads a row.  Layer by layer the A operand is written to
// shared memory (K-major, no swizzle: 16 bytes of a row per 8 columns, rows 16
// bytes apart, so a warp's store is contiguous), one thread issues the layer's
// mmas into the group's 64 TMEM columns, and the threads read their row back with
// tcgen05.ld, apply the ReLU and round to bf16 for the next layer.  The biases
// are part of the products: three more rows of the weights hold a bias as the
// exact sum of three bf16 parts, against constant ones in the activations.  They
// come first and the inputs follow in ascending sixteens, so the sums are those of
// mma.sync accumulators that start at the bias: 4.9 M outputs with biases from
// 1e-3 to 100 came out the same, bit for bit.
//
// One block of eight groups per SM shares the weights (16 KB); a group's operands
// are 20 KB, the first layer's in the columns next to the constant ones, and its
// eight tiles in flight cover one another's waits (the 64 registers of 1024
// threads and the 512 TMEM columns both end at eight).  A group's tiles are
// neighbours: the next tile's rows are fetched into L2 ahead, and its chunk is
// looked up again only where one ends.  The waits are bounded; a warp that gives
// up touches neither its operands nor TMEM again, sets *err and yields NaN, and a
// group whose products' warp gave up issues no more and waits, again bounded, for
// the ones in flight before the TMEM goes.
//
// Bytes: 16 + 4 NB read and 4 written per cube, 19 us for 2.2 M cubes of 10 bins;
// what bounds it is the instructions of a row's features and its two epilogues
// (about 610 a warp) and the latency between them.  Those cubes in 128 chunks:
// 104 us with mma.sync, at that instruction's 236 TFLOP/s, -> 93 us with tcgen05,
// 78 us with the ReLU on packed pairs, neighbouring tiles and the prefetch, 77 us
// with the weights copied as the products take them (k_mlp_pack lays them out when
// they change; gathered from the FP32 parameters by each block, a call of 6,000 to
// 600,000 cubes took 1.3 to 1.8 us longer: 17.6 and 36.5 us against 16.3 and 34.7),
// 75 us with the waits decided per warp.
constexpr int TC_GROUPS = 8, TC_THREADS = TC_GROUPS * 128;
constexpr int TC_CORE = 128 * 16;          // 128 rows x 8 columns
constexpr int TC_A = 10 * TC_CORE;         // 80 columns: 64 activations, 3 ones, 13 zeros
constexpr size_t TC_SMEM = TC_W + (size_t)TC_GROUPS * TC_A;

// Shared-memory operand descriptor: address, the distance between the two
// 8-column halves of an mma's 16 columns (leading) and between groups of 8 rows
// (stride), all in 16-byte units; version 1, no swizzle.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t leading, uint32_t stride) {
    return uint64_t((addr >> 4) & 0x3fff) | (uint64_t((leading >> 4) & 0x3fff) << 16) |
           (uint64_t((stride >> 4) & 0x3fff) << 32) | (uint64_t(1) << 46);
}
// Instruction descriptor: FP32 accumulator, bf16 x bf16, both K-major, M = 128.
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(128 >> 4) << 24);
}
// chunks x 16 columns of A (from a_at) times B (rows of n columns from b_at) into TMEM
// columns d, the last 16 columns (the bias) first.
__device__ __forceinline__ void tc_product(uint32_t d, uint32_t a_at, uint32_t b_at, int n, int chunks, uint32_t mbar) {
    for (int e = 0; e < chunks; ++e) {
        const int k = e ? e - 1 : chunks - 1;
        const uint64_t da = tc_desc(a_at + k * 2 * TC_CORE, TC_CORE, 128);
        const uint64_t db = tc_desc(b_at + k * 2 * n * 16, n * 16, 128);
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d), "l"(da), "l"(db), "r"(tc_idesc(n)), "r"(e) : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
constexpr int TC_POLLS = 1 << 15;  // of a wait, at most 20 us each
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity, int polls) {
    for (int spin = 0; spin < polls; ++spin) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 20000;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return true;
        }
    }
    return false;
}
__device__ __forceinline__ void tc_load32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
// Two accumulators as bf16, negative ones and NaN as zero (rounding keeps the sign,
// so the maximum of the pair is taken after it).
__device__ __forceinline__ uint32_t relu_pack(uint32_t lo, uint32_t hi) {
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(pack_bf16(__uint_as_float(lo), __uint_as_float(hi))), "r"(0u));
    return r;
}

// What the generic-proxy stores of the group left in shared memory is there for
// its mmas, and its reads of TMEM are done, once all 128 threads have passed.
__device__ __forceinline__ void tc_group_sync(int group) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// SRC 0: y[i] of the feature rows X.  SRC 1, 2: the warm start u = median indicator
// + network of the cubes, their features built here; the chunk of a cube is found
// by bisection (1: the boxes' index ranges ascend without overlap; a warp looks up
// its first cube and its lanes step on from there) or read from leaf_id (2: the
// first chunk in the caller's order that holds the cube, -1 for none; null: the root).
template <int NB, int SRC>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_forward(int n, const uint4* __restrict__ X, const uint4* __restrict__ cubes, const uint32_t* __restrict__ hists,
          const LeafBox* __restrict__ boxes, int nleaf, const int* __restrict__ leaf_id,
          const __nv_bfloat16* __restrict__ weights, float* __restrict__ out, int* __restrict__ err, int polls) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ FeatureTables tab;
    __shared__ __align__(8) unsigned long long s_bar[TC_GROUPS];
    __shared__ uint32_t s_tmem;
    const int group = threadIdx.x >> 7, row = threadIdx.x & 127, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* A = smem_raw + TC_W + group * TC_A;
    const uint32_t w_at = (uint32_t)__cvta_generic_to_shared(smem_raw), a_at = (uint32_t)__cvta_generic_to_shared(A),
                   bar = (uint32_t)__cvta_generic_to_shared(s_bar + group);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                     ::"r"((uint32_t)__cvta_generic_to_shared(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (row == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    if (SRC) feature_tables<NB>(tab);
    for (int e = threadIdx.x; e < TC_W / 16; e += TC_THREADS)
        reinterpret_cast<uint4*>(smem_raw)[e] = __ldg(reinterpret_cast<const uint4*>(weights) + e);
    // the constant columns 64..79
    *reinterpret_cast<uint4*>(A + 8 * TC_CORE + row * 16) = make_uint4(0x3f803f80u, 0x00003f80u, 0u, 0u);
    *reinterpret_cast<uint4*>(A + 9 * TC_CORE + row * 16) = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t d = s_tmem + group * 64;                          // the group's columns
    const uint32_t mine = d + ((uint32_t)(warp & 3) * 32u << 16);  // this warp's lanes of them
    const bool vec = SRC && bins_aligned<NB>(hists);
    uint32_t phase = 0;  // of the products waited for next
    bool ok = true;      // the same for all of a warp
    auto wait = [&] {
        if (ok) ok = __all_sync(0xffffffffu, tc_wait(bar, phase & 1, polls));
        if (ok) ++phase;
    };
    // Each group's tiles are neighbours, so its chunk seldom changes.
    const int64_t tiles = ((int64_t)n + 127) / 128, runs = (int64_t)gridDim.x * TC_GROUPS,
                  run = blockIdx.x + (int64_t)group * gridDim.x;
    int chunk = -1;  // the last one that starts at or before the warp's first cube
    for (int64_t t = tiles * run / runs, end = tiles * (run + 1) / runs; t < end; ++t) {
        const int64_t i0 = t * 128 + (warp & 3) * 32;  // the warp's first row
        const int64_t i = i0 + lane;
        float med = 0.f;
        uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
        if (i < n) {
            if (SRC == 0) {
                lo = __ldg(X + i * 2);
                hi = __ldg(X + i * 2 + 1);
            } else {
                uint32_t bins[NB], w[8];
                load_bins<NB>(hists + (size_t)i * NB, vec, bins);
                const uint4 cb = __ldg(cubes + i);
                if (i + 128 < n) {  // the next tile's
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(cubes + i + 128));
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(hists + (size_t)(i + 128) * NB));
                }
                LeafBox box{0, 0, 0, 0, 0, 1.0f / (float)(1u << 21)};
                if (SRC == 1) {
                    if (chunk + 1 < nleaf && __ldg(&boxes[chunk + 1].first) <= (uint32_t)i0) {
                        int l = chunk + 2, h = nleaf;  // first box that starts after the warp's first cube
                        while (l < h) {
                            const int mid = (l + h) >> 1;
                            if (__ldg(&boxes[mid].first) <= (uint32_t)i0) l = mid + 1; else h = mid;
                        }
                        chunk = l - 1;
                    }
                    int s = chunk;
                    while (s + 1 < nleaf && __ldg(&boxes[s + 1].first) <= (uint32_t)i) ++s;
                    if (s >= 0 && (uint32_t)i <= __ldg(&boxes[s].last)) box = boxes[s];
                } else if (leaf_id) {
                    const int l = __ldg(leaf_id + i);
                    if (l >= 0) box = boxes[l];
                }
                med = feature_row<NB>(bins, cb, box, tab, w);
                lo = make_uint4(w[0], w[1], w[2], w[3]);
                hi = make_uint4(w[4], w[5], w[6], w[7]);
            }
        }
        // layer 1: columns 48..63 hold the features, 64..79 the ones
        if (ok) {
            *reinterpret_cast<uint4*>(A + 6 * TC_CORE + row * 16) = lo;
            *reinterpret_cast<uint4*>(A + 7 * TC_CORE + row * 16) = hi;
        }
        tc_group_sync(group);
        if (row == 0 && ok) tc_product(d, a_at + 6 * TC_CORE, w_at + TC_B1, 64, 2, bar);
        for (int layer = 0; layer < 2; ++layer) {
            wait();
            if (ok) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t r[32];
                    tc_load32(mine + half * 32, r);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(A + (half * 4 + c) * TC_CORE + row * 16) =
                            make_uint4(relu_pack(r[8 * c], r[8 * c + 1]), relu_pack(r[8 * c + 2], r[8 * c + 3]),
                                       relu_pack(r[8 * c + 4], r[8 * c + 5]), relu_pack(r[8 * c + 6], r[8 * c + 7]));
                }
            }
            tc_group_sync(group);
            if (row == 0 && ok) {
                if (layer == 0) tc_product(d, a_at, w_at + TC_B2, 64, 5, bar);
                else tc_product(d, a_at, w_at + TC_B3, 16, 5, bar);
            }
        }
        wait();
        uint32_t y = 0x7fc00000u;
        if (ok)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n\ttcgen05.wait::ld.sync.aligned;"
                         : "=r"(y) : "r"(mine) : "memory");
        if (i < n) out[i] = SRC ? fadd(med, __uint_as_float(y)) : __uint_as_float(y);
    }
    if (!ok) {
        if (lane == 0) atomicOr(err, 1);
        if (row == 0) tc_wait(bar, phase & 1, TC_POLLS);  // the products still in flight
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tmem) : "memory");
}

// One inference launch; d_id null with leaves means ascending chunks.
template <int NB, int SRC>
static int launch_forward(tgvg_ctx* ctx, int64_t n, const uint32_t* X, const tgvg_cube* d_c, const uint32_t* d_h,
                          const LeafBox* boxes, int nleaf, const int* d_id, const __nv_bfloat16* tc, float* out, int* err,
                          int polls) {
    TGVG_CK(ctx, cudaFuncSetAttribute(k_forward<NB, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
    const int64_t tiles = (n + 127) / 128;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, ctx->sm_count);  // a few tiles spread over the SMs
    k_forward<NB, SRC><<<grid, TC_THREADS, TC_SMEM, ctx->stream>>>(
        (int)n, reinterpret_cast<const uint4*>(X), reinterpret_cast<const uint4*>(d_c), d_h, boxes, nleaf, d_id, tc, out,
        err, polls);
    TGVG_LAUNCHED(ctx);
    return TGVG_OK;
}

__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t (&r)[2], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}

// Gradient of the mean squared error over rows idx[0..m) (idx may be null:
// rows 0..m).  Gradients and the loss sum are added into grad[P_N] and loss[0].
//
// The three products of the backward pass (dZ1 = dZ2 W2^T, dW2 = H1^T dZ2,
// dW1 = X^T dZ1) run on the tensor cores without giving up FP32: one factor is
// bf16 already (weights, activations, inputs), the other, an FP32 array, is
// split into three bf16 parts that add up to it exactly, so every product is
// exact and the three partial products are added in FP32, the small parts
// first.  The tensor core's accumulator is used over 16 rows at a time for the
// leading part (one mma from zero), and the sums over rows are FP32 adds.
//
// A block takes WARPS * 16 rows at a time: each warp runs its 16 rows forward
// and back to dZ1 in registers (an accumulator tile is, packed, the next
// product's A fragment), leaves H1, X and the parts of dZ2, then of dZ1, in
// shared memory, and then owns 8 / WARPS of the eight 8-column tiles of dW2 and
// dW1, reading both factors transposed with ldmatrix.  So the weight gradients
// stay in registers over all of the block's rows (20 a thread with 8 warps) and
// reach global memory once per block.
//
// Bound: the warp-level mma rate (260 mma per 16 rows, 216 of them the split
// products).  Before, the products were FP32 dot products out of shared memory
// with a shared-memory atomic per element and 16 rows.  A gradient call over
// 400,000 rows of host memory: 2363 -> 253 us; over 3,000 rows 122 -> 74 us; an
// epoch of 25 batches of 4,096 rows 2.3 -> 1.0 ms.  Relative error of the
// gradient against 64 bits, mean of four seeds: 400,000 rows 6.1e-7 before and
// after, 10,000 rows 4.4e-7 -> 4.2e-7.
// Row pitches of 72 and 24 halves keep the fragment stores and the eight row
// reads of an ldmatrix on different banks.
constexpr int GP = 72;   // halves per row of H1 and of a dZ part
constexpr int GXP = 24;  // halves per row of X
template <int WARPS>
constexpr size_t grad_smem() {
    return 4 * (size_t)(F_N + 136 + 64 + 32 * 64 + 196) + 2 * (size_t)(WARPS * 16) * (4 * GP + GXP);
}
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 3)
k_mlp_grad(const uint32_t* __restrict__ X, const float* __restrict__ t, const int* __restrict__ idx, int m, float inv_m,
           const uint32_t* __restrict__ frag, const float* __restrict__ prm, const float* __restrict__ wr,
           float* __restrict__ grad, float* __restrict__ loss) {
    constexpr int ROWS = WARPS * 16, NTW = 8 / WARPS;  // rows per step; column tiles per warp
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint32_t* sfrag = reinterpret_cast<uint32_t*>(smem_raw);
    float* sbias = reinterpret_cast<float*>(sfrag + F_N);  // 136
    float* sw3 = sbias + 136;                              // 64: bf16-rounded W3
    uint32_t* sw2t = reinterpret_cast<uint32_t*>(sw3 + 64);  // B fragments of W2^T
    float* sred = reinterpret_cast<float*>(sw2t + 32 * 64);  // dW3, db2, db1, db3 (196)
    uint32_t* sh1 = reinterpret_cast<uint32_t*>(sred + 196);  // [ROWS][GP/2]
    uint32_t* sz = sh1 + ROWS * (GP / 2);                    // [3][ROWS][GP/2]: parts hi, mid, lo
    uint32_t* sx = sz + 3 * ROWS * (GP / 2);                 // [ROWS][GXP/2]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
    for (int w = threadIdx.x; w < 32 * 64; w += WARPS * 32) {
        // tile (kc, nt) of B[j][k] = W2[k][j]: word of lane (g, c), half: rows j = 16 kc + 2c + 8 half, column k = 8 nt + g
        const int tile = w / 64, l = (w % 64) / 2, half = w % 2;
        const int k = (tile % 8) * 8 + l / 4, jj = (tile / 8) * 16 + 2 * (l % 4) + 8 * half;
        sw2t[w] = pack_bf16(wr[P_W2 + k * 64 + jj], wr[P_W2 + k * 64 + jj + 1]);
    }
    for (int k = threadIdx.x; k < 64; k += WARPS * 32) sw3[k] = wr[P_W3 + k];
    for (int k = threadIdx.x; k < 196; k += WARPS * 32) sred[k] = 0.f;
    load_net(frag, prm, sfrag, sbias);  // ends with a block barrier
    float acc2[NTW][4][4], acc1[NTW][4];  // this warp's tiles of dW2 (64 x 8 NTW) and dW1 (16 x 8 NTW)
    float b2s[8][2], b1s[8][2], w3s[8][2], dys = 0.f, lsum = 0.f;
#pragma unroll
    for (int a = 0; a < NTW; ++a)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            acc1[a][e] = 0.f;
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) acc2[a][mt][e] = 0.f;
        }
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) b2s[nt][0] = b2s[nt][1] = b1s[nt][0] = b1s[nt][1] = w3s[nt][0] = w3s[nt][1] = 0.f;
    const int lr = warp * 16 + g;  // this lane's rows of the step: lr and lr + 8
    const uint32_t h1_at = (uint32_t)__cvta_generic_to_shared(sh1), z_at = (uint32_t)__cvta_generic_to_shared(sz),
                   x_at = (uint32_t)__cvta_generic_to_shared(sx);
    // ldmatrix row addresses: A tiles (four 8x8 blocks: rows 0-7 / 8-15 by columns 0-7 / 8-15) and B tiles
    const int a_row = (lane & 7) + ((lane >> 4) & 1) * 8, a_col = ((lane >> 3) & 1) * 8, b_row = lane & 15;
    for (int64_t r0 = (int64_t)blockIdx.x * ROWS; r0 < m; r0 += (int64_t)gridDim.x * ROWS) {
        int rows[2];
        uint32_t a[1][4] = {{0, 0, 0, 0}};
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int64_t b = r0 + lr + 8 * rr;
            rows[rr] = b < m ? (idx ? idx[b] : (int)b) : -1;
            if (rows[rr] >= 0) {
                a[0][rr] = X[(size_t)rows[rr] * 8 + c];
                a[0][rr + 2] = X[(size_t)rows[rr] * 8 + c + 4];
            }
            sx[(lr + 8 * rr) * (GXP / 2) + c] = a[0][rr];
            sx[(lr + 8 * rr) * (GXP / 2) + c + 4] = a[0][rr + 2];
        }
        uint32_t ha1[1][4][4], ha2[1][4][4];
        mlp_layer1<1>(a, sfrag, sbias, ha1);
        uint32_t (&h1)[4][4] = ha1[0], (&h2)[4][4] = ha2[0];
        float y[1][2], dy0 = 0.f, dy1 = 0.f;
        mlp_rest<1>(ha1, sfrag, sbias, y, ha2);
        if (c == 0) {  // dy = 2 (y - t) / m
            if (rows[0] >= 0) { const float e = y[0][0] - t[rows[0]]; lsum += e * e; dy0 = 2.f * e * inv_m; }
            if (rows[1] >= 0) { const float e = y[0][1] - t[rows[1]]; lsum += e * e; dy1 = 2.f * e * inv_m; }
            dys += dy0 + dy1;
        }
        dy0 = __shfl_sync(0xffffffffu, dy0, lane & 28);
        dy1 = __shfl_sync(0xffffffffu, dy1, lane & 28);
        // dZ2 = dy W3 where h2 > 0, its parts as the A fragments of dZ2 W2^T and in shared memory
        uint32_t zp[3][4][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const float2 w3 = *reinterpret_cast<const float2*>(sw3 + nt * 8 + 2 * c);
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const uint32_t hv = h2[nt >> 1][(nt & 1) * 2 + rr];
                const float ha = __uint_as_float(hv << 16), hb = __uint_as_float(hv & 0xffff0000u);
                const float dy = rr ? dy1 : dy0;
                const float za = ha > 0.f ? dy * w3.x : 0.f, zb = hb > 0.f ? dy * w3.y : 0.f;
                w3s[nt][0] += ha * dy;
                w3s[nt][1] += hb * dy;
                b2s[nt][0] += za;
                b2s[nt][1] += zb;
                float ah, am, al, bh, bm, bl;
                split_bf16(za, ah, am, al);
                split_bf16(zb, bh, bm, bl);
                const uint32_t w[3] = {pack_top(ah, bh), pack_top(am, bm), pack_top(al, bl)};
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    zp[q][nt >> 1][(nt & 1) * 2 + rr] = w[q];
                    sz[(q * ROWS + lr + 8 * rr) * (GP / 2) + nt * 4 + c] = w[q];
                }
                sh1[(lr + 8 * rr) * (GP / 2) + nt * 4 + c] = h1[nt >> 1][(nt & 1) * 2 + rr];
            }
        }
        // dZ1 = dZ2 W2^T where h1 > 0 (accumulator layout, columns 8 nt + 2c..)
        float z1[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
            for (int q = 2; q >= 0; --q)
#pragma unroll
                for (int kc = 0; kc < 4; ++kc) {
                    const uint2 bf = *reinterpret_cast<const uint2*>(sw2t + (kc * 8 + nt) * 64 + lane * 2);
                    mma_bf16(d0, d1, d2, d3, zp[q][kc][0], zp[q][kc][1], zp[q][kc][2], zp[q][kc][3], bf.x, bf.y);
                }
            const uint32_t u0 = h1[nt >> 1][(nt & 1) * 2], u1 = h1[nt >> 1][(nt & 1) * 2 + 1];
            z1[nt][0] = __uint_as_float(u0 << 16) > 0.f ? d0 : 0.f;
            z1[nt][1] = __uint_as_float(u0 & 0xffff0000u) > 0.f ? d1 : 0.f;
            z1[nt][2] = __uint_as_float(u1 << 16) > 0.f ? d2 : 0.f;
            z1[nt][3] = __uint_as_float(u1 & 0xffff0000u) > 0.f ? d3 : 0.f;
            b1s[nt][0] += z1[nt][0] + z1[nt][2];
            b1s[nt][1] += z1[nt][1] + z1[nt][3];
        }
        __syncthreads();
        // dW2 += H1^T dZ2 over the block's rows
        {
            float low[NTW][4][4];
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) low[n][mt][e] = 0.f;
#pragma unroll 2
            for (int ks = 0; ks < WARPS; ++ks) {
                uint32_t A[4][4];
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
                    ldsm_x4_trans(A[mt], h1_at + 2 * ((ks * 16 + a_row) * GP + mt * 16 + a_col));
#pragma unroll
                for (int n = 0; n < NTW; ++n)
#pragma unroll
                    for (int q = 2; q >= 0; --q) {
                        uint32_t B[2];
                        ldsm_x2_trans(B, z_at + 2 * ((q * ROWS + ks * 16 + b_row) * GP + (warp * NTW + n) * 8));
#pragma unroll
                        for (int mt = 0; mt < 4; ++mt) {
                            if (q > 0) {
                                mma_bf16(low[n][mt][0], low[n][mt][1], low[n][mt][2], low[n][mt][3], A[mt][0], A[mt][1],
                                         A[mt][2], A[mt][3], B[0], B[1]);
                            } else {
                                float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
                                mma_bf16(d0, d1, d2, d3, A[mt][0], A[mt][1], A[mt][2], A[mt][3], B[0], B[1]);
                                acc2[n][mt][0] += d0; acc2[n][mt][1] += d1; acc2[n][mt][2] += d2; acc2[n][mt][3] += d3;
                            }
                        }
                    }
            }
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc2[n][mt][e] += low[n][mt][e];
        }
        __syncthreads();
        // the parts of dZ1 take dZ2's place
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                float ah, am, al, bh, bm, bl;
                split_bf16(z1[nt][2 * rr], ah, am, al);
                split_bf16(z1[nt][2 * rr + 1], bh, bm, bl);
                uint32_t* z = sz + (lr + 8 * rr) * (GP / 2) + nt * 4 + c;
                z[0] = pack_top(ah, bh);
                z[ROWS * (GP / 2)] = pack_top(am, bm);
                z[2 * ROWS * (GP / 2)] = pack_top(al, bl);
            }
        __syncthreads();
        // dW1 += X^T dZ1
        {
            float low[NTW][4];
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) low[n][e] = 0.f;
#pragma unroll 2
            for (int ks = 0; ks < WARPS; ++ks) {
                uint32_t A[4];
                ldsm_x4_trans(A, x_at + 2 * ((ks * 16 + a_row) * GXP + a_col));
#pragma unroll
                for (int n = 0; n < NTW; ++n)
#pragma unroll
                    for (int q = 2; q >= 0; --q) {
                        uint32_t B[2];
                        ldsm_x2_trans(B, z_at + 2 * ((q * ROWS + ks * 16 + b_row) * GP + (warp * NTW + n) * 8));
                        if (q > 0) {
                            mma_bf16(low[n][0], low[n][1], low[n][2], low[n][3], A[0], A[1], A[2], A[3], B[0], B[1]);
                        } else {
                            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
                            mma_bf16(d0, d1, d2, d3, A[0], A[1], A[2], A[3], B[0], B[1]);
                            acc1[n][0] += d0; acc1[n][1] += d1; acc1[n][2] += d2; acc1[n][3] += d3;
                        }
                    }
            }
#pragma unroll
            for (int n = 0; n < NTW; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc1[n][e] += low[n][e];
        }
        __syncthreads();  // shared memory is rewritten by the next step
    }
    // weight gradients: this warp alone holds its columns of the block's sums
#pragma unroll
    for (int n = 0; n < NTW; ++n) {
        const int col = (warp * NTW + n) * 8 + 2 * c;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            atomicAdd(reinterpret_cast<float2*>(grad + P_W2 + (mt * 16 + g) * 64 + col),
                      make_float2(acc2[n][mt][0], acc2[n][mt][1]));
            atomicAdd(reinterpret_cast<float2*>(grad + P_W2 + (mt * 16 + g + 8) * 64 + col),
                      make_float2(acc2[n][mt][2], acc2[n][mt][3]));
        }
        atomicAdd(reinterpret_cast<float2*>(grad + P_W1 + g * 64 + col), make_float2(acc1[n][0], acc1[n][1]));
        atomicAdd(reinterpret_cast<float2*>(grad + P_W1 + (g + 8) * 64 + col), make_float2(acc1[n][2], acc1[n][3]));
    }
    // column sums: over the eight row groups of the warp, then over the block's warps
    auto col_sum = [&](float v, int at) {
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (g == 0) atomicAdd(sred + at, v);
    };
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            col_sum(w3s[nt][e], nt * 8 + 2 * c + e);
            col_sum(b2s[nt][e], 64 + nt * 8 + 2 * c + e);
            col_sum(b1s[nt][e], 128 + nt * 8 + 2 * c + e);
        }
    for (int o = 16; o > 0; o >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        dys += __shfl_xor_sync(0xffffffffu, dys, o);
    }
    if (lane == 0) {
        atomicAdd(sred + 192, dys);
        atomicAdd(sred + 193, lsum);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 64; k += WARPS * 32) {
        atomicAdd(grad + P_W3 + k, sred[k]);
        atomicAdd(grad + P_B2 + k, sred[64 + k]);
        atomicAdd(grad + P_B1 + k, sred[128 + k]);
    }
    if (threadIdx.x == 0) {
        atomicAdd(grad + P_B3, sred[192]);
        atomicAdd(loss, sred[193]);
    }
}

// One gradient launch over m rows.  128 rows a step (8 warps, two blocks per
// SM) once that many steps fill the SMs; 64 rows (4 warps) below, where a
// mini-batch has too few rows for 152 blocks of 128 (at 4,096 rows: 64 blocks
// instead of 32).
static int launch_grad(tgvg_ctx* ctx, const uint32_t* X, const float* t, const int* idx, int m, const uint32_t* frag,
                       const float* prm, const float* wr, float* grad, float* loss) {
    const bool wide = m >= 128 * ctx->sm_count;
    const int rows = wide ? 128 : 64;
    const unsigned grid = (unsigned)std::max(1, std::min((m + rows - 1) / rows, ctx->sm_count * (wide ? 2 : 3)));
    const float inv_m = 1.0f / (float)m;
    if (wide) {
        TGVG_CK(ctx, cudaFuncSetAttribute(k_mlp_grad<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem<8>()));
        k_mlp_grad<8><<<grid, 256, grad_smem<8>(), ctx->stream>>>(X, t, idx, m, inv_m, frag, prm, wr, grad, loss);
    } else {
        TGVG_CK(ctx, cudaFuncSetAttribute(k_mlp_grad<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem<4>()));
        k_mlp_grad<4><<<grid, 128, grad_smem<4>(), ctx->stream>>>(X, t, idx, m, inv_m, frag, prm, wr, grad, loss);
    }
    TGVG_LAUNCHED(ctx);
    return TGVG_OK;
}

__global__ void k_adam(float* __restrict__ prm, float* __restrict__ m1, float* __restrict__ m2,
                       const float* __restrict__ grad, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P_N) return;
    const float gk = grad[k];
    const float a = b1 * m1[k] + (1.f - b1) * gk;
    const float b = b2 * m2[k] + (1.f - b2) * gk * gk;
    m1[k] = a;
    m2[k] = b;
    prm[k] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
}

}  // namespace tgvg

// ------------------------------------------------------------------ C ABI ---
using namespace tgvg;

struct tgvg_mlp {
    int nbins;
    float* d_prm = nullptr;
    float* d_m1 = nullptr;
    float* d_m2 = nullptr;
    float* d_grad = nullptr;
    float* d_wr = nullptr;
    float* d_loss = nullptr;
    uint32_t* d_frag = nullptr;
    __nv_bfloat16* d_tc = nullptr;
    int step = 0;
    int polls = TC_POLLS;  // of an inference wait
};

static int mlp_repack(tgvg_ctx* ctx, tgvg_mlp* m) {
    k_mlp_pack<<<(TC_W / 2 + 255) / 256, 256, 0, ctx->stream>>>(m->d_prm, m->d_frag, m->d_wr, m->d_tc);  // TC_W / 2 > P_N, F_N
    TGVG_LAUNCHED(ctx);
    return TGVG_OK;
}

extern "C" int tgvg_mlp_create(tgvg_ctx* ctx, int32_t nbins, uint64_t seed, tgvg_mlp** out) {
    if (!ctx || !out || (nbins != 8 && nbins != 10)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    auto* m = new tgvg_mlp();
    m->nbins = nbins;
    float** bufs[] = {&m->d_prm, &m->d_m1, &m->d_m2, &m->d_grad, &m->d_wr};
    bool ok = true;
    for (float** b : bufs) ok = ok && ctx->dev_alloc((void**)b, sizeof(float) * P_N) == cudaSuccess;
    if (!ok || ctx->dev_alloc((void**)&m->d_loss, sizeof(float)) != cudaSuccess ||
        ctx->dev_alloc((void**)&m->d_frag, sizeof(uint32_t) * F_N) != cudaSuccess ||
        ctx->dev_alloc((void**)&m->d_tc, TC_W) != cudaSuccess) {
        cudaGetLastError();
        tgvg_mlp_destroy(m);
        return TGVG_ERR_NOMEM;
    }
    // He-uniform weights over the real fan-in (the padded inputs stay zero), zero biases.
    std::mt19937_64 rng(seed);
    std::vector<float> p(P_N, 0.f);
    const int fan1 = nbins + 4;
    std::uniform_real_distribution<float> u1(-std::sqrt(6.f / fan1), std::sqrt(6.f / fan1));
    std::uniform_real_distribution<float> u2(-std::sqrt(6.f / 64), std::sqrt(6.f / 64));
    std::uniform_real_distribution<float> u3(-std::sqrt(3.f / 64), std::sqrt(3.f / 64));
    for (int k = 0; k < fan1; ++k)
        for (int j = 0; j < 64; ++j) p[P_W1 + k * 64 + j] = u1(rng);
    for (int k = 0; k < 64 * 64; ++k) p[P_W2 + k] = u2(rng);
    for (int k = 0; k < 64; ++k) p[P_W3 + k] = u3(rng);
    TGVG_CK(ctx, cudaMemcpyAsync(m->d_prm, p.data(), sizeof(float) * P_N, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemsetAsync(m->d_m1, 0, sizeof(float) * P_N, ctx->stream));
    TGVG_CK(ctx, cudaMemsetAsync(m->d_m2, 0, sizeof(float) * P_N, ctx->stream));
    int rc = mlp_repack(ctx, m);
    if (rc) return rc;
    TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
    *out = m;
    return TGVG_OK;
}

extern "C" int tgvg_mlp_destroy(tgvg_mlp* m) {
    if (!m) return TGVG_ERR_INVALID;
    cudaFree(m->d_prm); cudaFree(m->d_m1); cudaFree(m->d_m2); cudaFree(m->d_grad); cudaFree(m->d_wr);
    cudaFree(m->d_loss); cudaFree(m->d_frag); cudaFree(m->d_tc);
    delete m;
    return TGVG_OK;
}

extern "C" int32_t tgvg_mlp_num_params(void) { return P_N; }

extern "C" int tgvg_mlp_params(tgvg_ctx* ctx, tgvg_mlp* m, float* get, const float* set) {
    if (!ctx || !m) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (set) {
        TGVG_CK(ctx, cudaMemcpyAsync(m->d_prm, set, sizeof(float) * P_N, cudaMemcpyHostToDevice, ctx->stream));
        int rc = mlp_repack(ctx, m);
        if (rc) return rc;
    }
    if (get) TGVG_CK(ctx, cudaMemcpyAsync(get, m->d_prm, sizeof(float) * P_N, cudaMemcpyDeviceToHost, ctx->stream));
    TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
    return TGVG_OK;
}

extern "C" int tgvg_mlp_features(tgvg_ctx* ctx, const tgvg_cube* cubes, const uint32_t* hists, int64_t n,
                                 int32_t nbins, const tgvg_leaf* leaves, int32_t nleaf, uint16_t* X) {
    if (!ctx || n < 0 || (n > 0 && (!cubes || !hists || !X)) || (nbins != 8 && nbins != 10) || nleaf < 0 ||
        (nleaf > 0 && !leaves) || n > (int64_t(1) << 30))
        return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (n == 0) return TGVG_OK;
    auto* d_c = (tgvg_cube*)ctx->buf(B_T_CUBES, sizeof(tgvg_cube) * n);
    auto* d_h = (uint32_t*)ctx->buf(B_T_HISTS, sizeof(uint32_t) * nbins * n);
    auto* d_x = (uint32_t*)ctx->buf(B_M_X, sizeof(uint32_t) * 8 * n);
    auto* d_l = (tgvg_leaf*)ctx->buf(B_M_LEAVES, sizeof(tgvg_leaf) * std::max(1, nleaf));
    auto* d_id = (int*)ctx->buf(B_M_LEAFID, sizeof(int) * n);
    if (!d_c || !d_h || !d_x || !d_l || !d_id) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, cudaMemcpyAsync(d_c, cubes, sizeof(tgvg_cube) * n, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemcpyAsync(d_h, hists, sizeof(uint32_t) * nbins * n, cudaMemcpyHostToDevice, ctx->stream));
    if (nleaf > 0)
        TGVG_CK(ctx, cudaMemcpyAsync(d_l, leaves, sizeof(tgvg_leaf) * nleaf, cudaMemcpyHostToDevice, ctx->stream));
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (nleaf > 0) {
        k_leaf_id<<<grid, 256, 0, ctx->stream>>>((int)n, nleaf, d_l, d_id);
        TGVG_LAUNCHED(ctx);
    }
    if (nbins == 8)
        k_mlp_features<8><<<grid, 256, 0, ctx->stream>>>((int)n, reinterpret_cast<const uint4*>(d_c), d_h,
                                                         nleaf > 0 ? d_id : nullptr, d_l, d_x);
    else
        k_mlp_features<10><<<grid, 256, 0, ctx->stream>>>((int)n, reinterpret_cast<const uint4*>(d_c), d_h,
                                                          nleaf > 0 ? d_id : nullptr, d_l, d_x);
    TGVG_LAUNCHED(ctx);
    TGVG_CK(ctx, cudaMemcpyAsync(X, d_x, sizeof(uint32_t) * 8 * n, cudaMemcpyDeviceToHost, ctx->stream));
    TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
    return TGVG_OK;
}

// Set by inference waits that run out: [0] in a call that waits for its result,
// [1] in tgvg_mlp_warm_start_dev, which does not (mlp_take_error).  Null: no memory.
static int* inference_error(tgvg_ctx* ctx) {
    const bool fresh = !ctx->bufs[B_M_ERR].p;
    int* e = (int*)ctx->buf(B_M_ERR, 2 * sizeof(int));
    if (e && fresh && cudaMemsetAsync(e, 0, 2 * sizeof(int), ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return e;
}

// Waits for the stream; reports the calling inference when a wait of it ran out.
static int inference_done(tgvg_ctx* ctx, int* err) {
    int e = 0;
    TGVG_CK(ctx, cudaMemcpyAsync(&e, err, sizeof(e), cudaMemcpyDeviceToHost, ctx->stream));
    TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (!e) return TGVG_OK;
    TGVG_CK(ctx, cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
    return ctx->fail(TGVG_ERR_TIMEOUT, "a tensor-core wait of the network timed out");
}

int tgvg::mlp_take_error(tgvg_ctx* ctx) {
    if (!ctx->mlp_pending) return TGVG_OK;
    ctx->mlp_pending = false;
    return inference_done(ctx, (int*)ctx->bufs[B_M_ERR].p + 1);
}

extern "C" int tgvg_mlp_set_wait_limit(tgvg_mlp* m, int32_t polls) {
    if (!m || polls < 0) return TGVG_ERR_INVALID;
    m->polls = polls < TC_POLLS ? polls : TC_POLLS;
    return TGVG_OK;
}

extern "C" int tgvg_mlp_predict(tgvg_ctx* ctx, tgvg_mlp* m, const uint16_t* X, int64_t n, float* y) {
    if (!ctx || !m || n < 0 || (n > 0 && (!X || !y)) || n > (int64_t(1) << 30)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (n == 0) return TGVG_OK;
    auto* d_x = (uint32_t*)ctx->buf(B_M_X, sizeof(uint32_t) * 8 * n);
    auto* d_y = (float*)ctx->buf(B_M_Y, sizeof(float) * n);
    int* err = inference_error(ctx);
    if (!d_x || !d_y || !err) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, cudaMemcpyAsync(d_x, X, sizeof(uint32_t) * 8 * n, cudaMemcpyHostToDevice, ctx->stream));
    int rc = launch_forward<8, 0>(ctx, n, d_x, nullptr, nullptr, nullptr, 0, nullptr, m->d_tc, d_y, err, m->polls);
    if (rc) return rc;
    TGVG_CK(ctx, cudaMemcpyAsync(y, d_y, sizeof(float) * n, cudaMemcpyDeviceToHost, ctx->stream));
    return inference_done(ctx, err);
}

// Warm-start u on the device (u = median + network).  Device cubes / histograms
// / output, host leaves.  Called with ctx->mu held.
static int warm_start_dev(tgvg_ctx* ctx, tgvg_mlp* m, const tgvg_cube* d_c, const uint32_t* d_h, int64_t n,
                          int32_t nbins, const tgvg_leaf* leaves, int32_t nleaf, float* d_u, int* err) {
    auto* d_b = (LeafBox*)ctx->buf(B_M_BOXES, sizeof(LeafBox) * std::max(1, nleaf));
    if (!d_b) return TGVG_ERR_NOMEM;
    // Ranges that ascend without overlap (a treetop's) are found by bisection;
    // any others keep the scan in the caller's order.
    bool sorted = true;
    std::vector<LeafBox> boxes(std::max(1, nleaf));
    for (int l = 0; l < nleaf; ++l) {
        boxes[l] = leaf_box(leaves[l]);
        sorted = sorted && boxes[l].first <= boxes[l].last && (l == 0 || boxes[l].first > boxes[l - 1].last);
    }
    if (nleaf > 0)
        TGVG_CK(ctx, cudaMemcpyAsync(d_b, boxes.data(), sizeof(LeafBox) * nleaf, cudaMemcpyHostToDevice, ctx->stream));
    int* d_id = nullptr;
    if (!sorted) {
        auto* d_l = (tgvg_leaf*)ctx->buf(B_M_LEAVES, sizeof(tgvg_leaf) * nleaf);
        d_id = (int*)ctx->buf(B_M_LEAFID, sizeof(int) * n);
        if (!d_l || !d_id) return TGVG_ERR_NOMEM;
        TGVG_CK(ctx, cudaMemcpyAsync(d_l, leaves, sizeof(tgvg_leaf) * nleaf, cudaMemcpyHostToDevice, ctx->stream));
        k_leaf_id<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>((int)n, nleaf, d_l, d_id);
        TGVG_LAUNCHED(ctx);
    }
    if (nbins == 8)
        return sorted ? launch_forward<8, 1>(ctx, n, nullptr, d_c, d_h, d_b, nleaf, nullptr, m->d_tc, d_u, err, m->polls)
                      : launch_forward<8, 2>(ctx, n, nullptr, d_c, d_h, d_b, nleaf, d_id, m->d_tc, d_u, err, m->polls);
    return sorted ? launch_forward<10, 1>(ctx, n, nullptr, d_c, d_h, d_b, nleaf, nullptr, m->d_tc, d_u, err, m->polls)
                  : launch_forward<10, 2>(ctx, n, nullptr, d_c, d_h, d_b, nleaf, d_id, m->d_tc, d_u, err, m->polls);
}

static bool warm_start_args_ok(tgvg_ctx* ctx, tgvg_mlp* m, const void* c, const void* h, int64_t n, int32_t nbins,
                               const tgvg_leaf* leaves, int32_t nleaf, const void* u) {
    return ctx && m && n >= 0 && (n == 0 || (c && h && u)) && (nbins == 8 || nbins == 10) && nbins == m->nbins &&
           nleaf >= 0 && (nleaf == 0 || leaves) && n <= (int64_t(1) << 30);
}

extern "C" int tgvg_mlp_warm_start(tgvg_ctx* ctx, tgvg_mlp* m, const tgvg_cube* cubes, const uint32_t* hists,
                                   int64_t n, int32_t nbins, const tgvg_leaf* leaves, int32_t nleaf, float* u) {
    if (!warm_start_args_ok(ctx, m, cubes, hists, n, nbins, leaves, nleaf, u)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (n == 0) return TGVG_OK;
    auto* d_c = (tgvg_cube*)ctx->buf(B_T_CUBES, sizeof(tgvg_cube) * n);
    auto* d_h = (uint32_t*)ctx->buf(B_T_HISTS, sizeof(uint32_t) * nbins * n);
    auto* d_u = (float*)ctx->buf(B_M_Y, sizeof(float) * n);
    int* err = inference_error(ctx);
    if (!d_c || !d_h || !d_u || !err) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, cudaMemcpyAsync(d_c, cubes, sizeof(tgvg_cube) * n, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemcpyAsync(d_h, hists, sizeof(uint32_t) * nbins * n, cudaMemcpyHostToDevice, ctx->stream));
    int rc = warm_start_dev(ctx, m, d_c, d_h, n, nbins, leaves, nleaf, d_u, err);
    if (rc) return rc;
    TGVG_CK(ctx, cudaMemcpyAsync(u, d_u, sizeof(float) * n, cudaMemcpyDeviceToHost, ctx->stream));
    return inference_done(ctx, err);
}

extern "C" int tgvg_mlp_warm_start_dev(tgvg_ctx* ctx, tgvg_mlp* m, const tgvg_cube* d_cubes,
                                       const uint32_t* d_hists, int64_t n, int32_t nbins, const tgvg_leaf* leaves,
                                       int32_t nleaf, float* d_u) {
    if (!warm_start_args_ok(ctx, m, d_cubes, d_hists, n, nbins, leaves, nleaf, d_u)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (n == 0) return TGVG_OK;
    int* err = inference_error(ctx);
    if (!err) return TGVG_ERR_NOMEM;
    ctx->mlp_pending = true;
    return warm_start_dev(ctx, m, d_cubes, d_hists, n, nbins, leaves, nleaf, d_u, err + 1);
}

// Gradient of the mean squared error of the whole set (one batch), for checks.
extern "C" int tgvg_mlp_grad(tgvg_ctx* ctx, tgvg_mlp* m, const uint16_t* X, const float* t, int64_t n,
                             float* grad, float* loss) {
    if (!ctx || !m || n <= 0 || !X || !t || !grad || n > (int64_t(1) << 30)) return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    auto* d_x = (uint32_t*)ctx->buf(B_M_X, sizeof(uint32_t) * 8 * n);
    auto* d_t = (float*)ctx->buf(B_M_T, sizeof(float) * n);
    if (!d_x || !d_t) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, cudaMemcpyAsync(d_x, X, sizeof(uint32_t) * 8 * n, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemcpyAsync(d_t, t, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemsetAsync(m->d_grad, 0, sizeof(float) * P_N, ctx->stream));
    TGVG_CK(ctx, cudaMemsetAsync(m->d_loss, 0, sizeof(float), ctx->stream));
    const int rc = launch_grad(ctx, d_x, d_t, nullptr, (int)n, m->d_frag, m->d_prm, m->d_wr, m->d_grad, m->d_loss);
    if (rc) return rc;
    TGVG_CK(ctx, cudaMemcpyAsync(grad, m->d_grad, sizeof(float) * P_N, cudaMemcpyDeviceToHost, ctx->stream));
    float l = 0.f;
    TGVG_CK(ctx, cudaMemcpyAsync(&l, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (loss) *loss = l / (float)n;
    return TGVG_OK;
}

// Adam on the mean squared error over shuffled mini-batches; returns the mean
// loss of the last epoch.
extern "C" int tgvg_mlp_train(tgvg_ctx* ctx, tgvg_mlp* m, const uint16_t* X, const float* t, int64_t n,
                              int32_t epochs, int32_t batch, float lr, uint64_t seed, float* last_loss) {
    if (!ctx || !m || n <= 0 || !X || !t || epochs < 0 || batch <= 0 || n > (int64_t(1) << 30))
        return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    auto* d_x = (uint32_t*)ctx->buf(B_M_X, sizeof(uint32_t) * 8 * n);
    auto* d_t = (float*)ctx->buf(B_M_T, sizeof(float) * n);
    auto* d_idx = (int*)ctx->buf(B_M_IDX, sizeof(int) * n);
    if (!d_x || !d_t || !d_idx) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, cudaMemcpyAsync(d_x, X, sizeof(uint32_t) * 8 * n, cudaMemcpyHostToDevice, ctx->stream));
    TGVG_CK(ctx, cudaMemcpyAsync(d_t, t, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->stream));
    std::vector<int> perm(n);
    for (int64_t i = 0; i < n; ++i) perm[i] = (int)i;
    std::mt19937_64 rng(seed);
    float epoch_loss = 0.f;
    for (int e = 0; e < epochs; ++e) {
        std::shuffle(perm.begin(), perm.end(), rng);
        TGVG_CK(ctx, cudaMemcpyAsync(d_idx, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx->stream));
        TGVG_CK(ctx, cudaMemsetAsync(m->d_loss, 0, sizeof(float), ctx->stream));
        for (int64_t b0 = 0; b0 < n; b0 += batch) {
            const int mb = (int)std::min<int64_t>(batch, n - b0);
            TGVG_CK(ctx, cudaMemsetAsync(m->d_grad, 0, sizeof(float) * P_N, ctx->stream));
            int rc = launch_grad(ctx, d_x, d_t, d_idx + b0, mb, m->d_frag, m->d_prm, m->d_wr, m->d_grad, m->d_loss);
            if (rc) return rc;
            ++m->step;
            const float c1 = 1.f - std::pow(0.9f, (float)m->step), c2 = 1.f - std::pow(0.999f, (float)m->step);
            k_adam<<<(P_N + 255) / 256, 256, 0, ctx->stream>>>(m->d_prm, m->d_m1, m->d_m2, m->d_grad, lr, 0.9f,
                                                               0.999f, 1e-8f, c1, c2);
            TGVG_LAUNCHED(ctx);
            if ((rc = mlp_repack(ctx, m))) return rc;
        }
        float l = 0.f;
        TGVG_CK(ctx, cudaMemcpyAsync(&l, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
        TGVG_CK(ctx, cudaStreamSynchronize(ctx->stream));
        epoch_loss = l / (float)n;
    }
    if (last_loss) *last_loss = epoch_loss;
    return TGVG_OK;
}
