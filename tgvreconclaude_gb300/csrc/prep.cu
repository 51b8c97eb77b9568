// Stage 1 on the GPU: the cubes of one depth map (the reference's
// build_cubes_from_depthmap, src/octree_builder.cpp:30-97, with
// cube_depth_for_radius :11-28 and DepthMap::unproject / sample_radius,
// src/depth_map.cpp:4-30).
//
// One thread per pixel: validity, the sample radius from the valid 4-neighbours,
// the world point, its place in the scene box, the cube depth for the radius
// and the Morton code; then a compaction and a stable radix sort by code, over
// the bits in which the map's codes differ.  The
// float arithmetic is the reference's, in its order, with explicitly rounded
// intrinsics (Eigen's 4x4 matvec and norms as the project's Eigen subset
// evaluates them).  round(log2(y)) of the depth rule is not evaluated on the
// device: the host finds, with its own log2f, the 21 thresholds where it
// reaches 1..21, and the kernel counts the thresholds below y.
//
// Cubes with equal codes come out in pixel order; the reference's std::sort
// leaves their order unspecified (and its parallel row loop makes the
// pre-sort order scheduling-dependent), so only the multiset of cubes is the
// reference's.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"
#include "fileio.h"

namespace tgvg {

struct DmDev {
    float fx, fy, cx, cy;
    float rt[16];  // world <- camera, row-major
    int w, h;
};

__device__ __forceinline__ bool dm_valid(const float* __restrict__ dep, const DmDev& m, int u, int v) {
    if (u < 0 || v < 0 || u >= m.w || v >= m.h) return false;
    const float d = dep[(size_t)v * m.w + u];
    return isfinite(d) && d > 0.0f;
}

// DepthMap::unproject (depth_map.cpp:4-11): cam = ((u - cx) d / fx, (v - cy) d / fy, d, 1), world = Rt cam.
__device__ __forceinline__ void dm_unproject(const float* __restrict__ dep, const DmDev& m, int u, int v, float* p) {
    const float d = dep[(size_t)v * m.w + u];
    const float c[4] = {fdiv(fmul(fsub((float)u, m.cx), d), m.fx), fdiv(fmul(fsub((float)v, m.cy), d), m.fy), d, 1.0f};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float acc = fmul(m.rt[4 * i], c[0]);
#pragma unroll
        for (int k = 1; k < 4; ++k) acc = fadd(acc, fmul(m.rt[4 * i + k], c[k]));
        p[i] = acc;
    }
}

__device__ __forceinline__ float norm3(float x, float y, float z) {
    return fsqrt(fadd(fadd(fmul(x, x), fmul(y, y)), fmul(z, z)));
}

// DepthMap::sample_radius (depth_map.cpp:13-30): half the mean distance to the
// valid 4-neighbours, in the order +u, -u, +v, -v.
__device__ __forceinline__ float dm_radius(const float* __restrict__ dep, const DmDev& m, int u, int v, const float* c) {
    const int du[4] = {1, -1, 0, 0}, dv[4] = {0, 0, 1, -1};
    float sum = 0.0f;
    int count = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int nu = u + du[i], nv = v + dv[i];
        if (!dm_valid(dep, m, nu, nv)) continue;
        float q[3];
        dm_unproject(dep, m, nu, nv, q);
        sum = fadd(sum, norm3(fsub(q[0], c[0]), fsub(q[1], c[1]), fsub(q[2], c[2])));
        ++count;
    }
    if (count == 0) return 0.0f;
    return fdiv(fmul(0.5f, sum), (float)count);
}

// cube_depth_for_radius (octree_builder.cpp:11-28) with max_depth 21.
struct RadiusThr {
    float t[21];
};
__device__ __forceinline__ int depth_for_radius(float r_x, float r_root, const RadiusThr& thr) {
    const float y = fdiv(r_root, fmul(r_x, 1.125f));
    int d = 0;
    if (!(isinf(y) && y > 0.0f)) {  // +inf: the cast of round(log2(inf)) gives INT_MIN on x86, clamped to 0
#pragma unroll
        for (int k = 0; k < 21; ++k) d += y >= thr.t[k] ? 1 : 0;
    }
    for (int tries = 0; tries < 3; ++tries) {
        const float cell = fdiv(r_root, (float)(1u << d));
        const float lo = fmul(0.75f, r_x), hi = fmul(1.5f, r_x);
        if (cell >= lo && cell < hi) break;
        if (cell < lo) { if (d > 0) --d; else break; }
        else { if (d < 21) ++d; else break; }
    }
    return d;
}

// The cube of pixel (u, v): false where it has none.
__device__ __forceinline__ bool stage1_cube(const DmDev& m, const float* __restrict__ dep, int u, int v, float3 o,
                                            float inv_2r, float r_root, const RadiusThr& thr, unsigned long long& key,
                                            float& rc, int& d) {
    if (!dm_valid(dep, m, u, v)) return false;
    float p[3];
    dm_unproject(dep, m, u, v, p);
    const float r_x = dm_radius(dep, m, u, v, p);
    if (!(r_x > 0.0f)) return false;
    const float n[3] = {fmul(fsub(p[0], o.x), inv_2r), fmul(fsub(p[1], o.y), inv_2r), fmul(fsub(p[2], o.z), inv_2r)};
    for (int k = 0; k < 3; ++k)
        if (n[k] < 0.0f || n[k] >= 1.0f) return false;  // the reference's test (a NaN passes it)
    d = depth_for_radius(r_x, r_root, thr);
    const uint32_t g = 1u << d;
    uint32_t ix[3];
    for (int k = 0; k < 3; ++k) {
        uint32_t q = __float2uint_rz(fmul(n[k], (float)g));
        ix[k] = q >= g ? g - 1 : q;
    }
    const int sh = 21 - d;
    key = spread3(ix[0] << sh) | (spread3(ix[1] << sh) << 1) | (spread3(ix[2] << sh) << 2);
    rc = r_x;
    return true;
}

// P1: the cubes of a tile of pixels, packed to the tile's front in pixel order,
// their number, and the bits set in any code (seen[0] high word, [1] low word).
// The packed records wait at the tile's place for the scan of the numbers, so no
// per-pixel flags and positions go through memory.  Bound by the arithmetic of the
// pixels that see a surface (ten IEEE divisions each).  A 1920x1080 map with
// 22 % such pixels, a call: 364 -> 289 us, 100 of them host copies; the sort
// alone 130 -> 75 (five passes of one word instead of eight of three).
constexpr int PIX_THREADS = 256, PIX_TILE = 1024;
__global__ void __launch_bounds__(PIX_THREADS)
k_stage1(DmDev m, const float* __restrict__ dep, float3 o, float inv_2r, float r_root, RadiusThr thr,
         unsigned long long* __restrict__ key, float2* __restrict__ pay, int* __restrict__ sums,
         unsigned* __restrict__ seen) {
    __shared__ int ws[PIX_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * PIX_TILE, npix = (int64_t)m.w * m.h;
    int at = 0;
    unsigned hi = 0, lo = 0;
    for (int k0 = 0; k0 < PIX_TILE; k0 += PIX_THREADS) {
        const int64_t t = base + k0 + threadIdx.x;
        unsigned long long k = 0;
        float rc = 0.f;
        int d = 0;
        const bool have = t < npix && stage1_cube(m, dep, (int)(t % m.w), (int)(t / m.w), o, inv_2r, r_root, thr, k, rc, d);
        const unsigned b = __ballot_sync(0xffffffffu, have);
        if (lane == 0) ws[w] = __popc(b);
        __syncthreads();
        int before = 0, all = 0;
        for (int q = 0; q < PIX_THREADS / 32; ++q) {
            if (q < w) before += ws[q];
            all += ws[q];
        }
        if (have) {
            const int64_t e = base + at + before + __popc(b & ((1u << lane) - 1u));
            key[e] = k;
            pay[e] = make_float2(rc, __int_as_float(d));
            hi |= (unsigned)(k >> 32);
            lo |= (unsigned)k;
        }
        at += all;
        __syncthreads();
    }
    hi = __reduce_or_sync(0xffffffffu, hi);
    lo = __reduce_or_sync(0xffffffffu, lo);
    if (lane == 0 && hi) atomicOr(seen, hi);
    if (lane == 0 && lo) atomicOr(seen + 1, lo);
    if (threadIdx.x == 0) sums[blockIdx.x] = at;
}

// P2: the tiles' records joined.  KEYS: the sort key holds the code's differing
// bits above the record's number (ib bits); else code and number apart.
template <bool KEYS>
__global__ void __launch_bounds__(PIX_THREADS)
k_stage1_join(const unsigned long long* __restrict__ key, const float2* __restrict__ pay, const int* __restrict__ sums,
              int low, int ib, unsigned long long* __restrict__ ckey, int* __restrict__ cidx, float2* __restrict__ cpay) {
    const int64_t base = (int64_t)blockIdx.x * PIX_TILE;
    const int first = sums[blockIdx.x], cnt = sums[blockIdx.x + 1] - first;
    for (int i = threadIdx.x; i < cnt; i += PIX_THREADS) {
        const int e = first + i;
        const unsigned long long k = key[base + i];
        if (KEYS) {
            ckey[e] = ((k >> low) << ib) | (unsigned)e;
        } else {
            ckey[e] = k;
            cidx[e] = e;
        }
        cpay[e] = pay[base + i];
    }
}

// P3: the sorted cubes.
template <bool KEYS>
__global__ void k_stage1_emit(int nc, const unsigned long long* __restrict__ skey, const int* __restrict__ sidx, int low,
                              int ib, const float2* __restrict__ pay, tgvg_cube* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    const unsigned long long s = skey[i];
    const unsigned long long k = KEYS ? (s >> ib) << low : s;
    const float2 p = pay[KEYS ? (int)(s & ((1ull << ib) - 1ull)) : sidx[i]];
    out[i] = tgvg_cube{(uint32_t)(k >> 32), (uint32_t)k, p.x, __float_as_int(p.y)};
}

// Thresholds t[k-1] = smallest float y > 0 with (int)round(log2f(y)) >= k, k = 1..21,
// found by bisection over the positive float bit patterns with the host's log2f.
static void radius_thresholds(float* t) {
    for (int k = 1; k <= 21; ++k) {
        uint32_t lo = 1u, hi = 0x7f7fffffu;  // smallest subnormal .. largest finite
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            float y;
            std::memcpy(&y, &mid, 4);
            if ((int)std::round(std::log2(y)) >= k) hi = mid; else lo = mid + 1;
        }
        std::memcpy(&t[k - 1], &lo, 4);
    }
}

// The cubes of one map.  *count receives their number; they are copied to
// out when it has room for them (cap), else TGVG_ERR_LIMIT; out == nullptr
// asks for the count only.
static int build_cubes(tgvg_ctx* ctx, const tgvg_depthmap* dm, const float* origin, float r_root,
                       tgvg_cube* out, int64_t cap, int64_t* count) {
    const int64_t npix = int64_t(dm->width) * dm->height;
    *count = 0;
    if (npix <= 0) return TGVG_OK;
    if (npix > (int64_t(1) << 30)) return ctx->fail(TGVG_ERR_LIMIT, "depth map larger than 2^30 pixels");
    static const RadiusThr thr = [] {
        RadiusThr r;
        radius_thresholds(r.t);
        return r;
    }();
    DmDev m;
    m.fx = dm->fx; m.fy = dm->fy; m.cx = dm->cx; m.cy = dm->cy;
    std::memcpy(m.rt, dm->rt, sizeof(m.rt));
    m.w = dm->width; m.h = dm->height;
    const float inv_2r = 1.0f / (2.0f * r_root);
    const int tiles = (int)((npix + PIX_TILE - 1) / PIX_TILE);
    auto B = [&](int id, size_t b) { return ctx->buf(id, b); };
    auto* dep = (float*)B(B_P_DEP, 4ull * npix);
    auto* key = (unsigned long long*)B(B_P_KEY, 8ull * npix);
    auto* pay = (float2*)B(B_P_RC, 8ull * npix);
    auto* sums = (int*)B(B_P_POS, 4ull * (tiles + 3));  // [tiles] the total, then the codes' bits
    if (!dep || !key || !pay || !sums) return TGVG_ERR_NOMEM;
    cudaStream_t st = ctx->stream;
    unsigned* seen = (unsigned*)(sums + tiles + 1);
    TGVG_CK(ctx, cudaMemsetAsync(seen, 0, 8, st));
    TGVG_CK(ctx, cudaMemcpyAsync(dep, dm->depths, 4ull * npix, cudaMemcpyHostToDevice, st));
    k_stage1<<<(unsigned)tiles, PIX_THREADS, 0, st>>>(m, dep, make_float3(origin[0], origin[1], origin[2]), inv_2r, r_root,
                                                      thr, key, pay, sums, seen);
    TGVG_LAUNCHED(ctx);
    int rc2 = scan_tile_sums(ctx, sums, tiles);
    if (rc2) return rc2;
    unsigned h[3] = {0, 0, 0};
    TGVG_CK(ctx, cudaMemcpyAsync(h, sums + tiles, sizeof(h), cudaMemcpyDeviceToHost, st));
    TGVG_CK(ctx, cudaStreamSynchronize(st));
    const int64_t nc = (int)h[0];
    *count = nc;
    if (nc == 0 || !out) return TGVG_OK;
    if (cap < nc) return TGVG_ERR_LIMIT;
    // Codes of depth D end in 3 (21 - D) zero bits and a scene leaves the top
    // ones alone, so only bits low .. high - 1 are sorted (33 of 63 on a 1920x1080
    // map at depth 11: five radix passes, not eight).  Where they and the record
    // numbers fit in one word, a record's key is that word and no values move.
    const uint64_t bits = (uint64_t(h[1]) << 32) | h[2];
    const int low = bits ? __builtin_ctzll(bits) : 0, high = bits ? 64 - __builtin_clzll(bits) : 1;
    int ib = 1;
    while ((int64_t(1) << ib) < nc) ++ib;
    const bool keys = high - low + ib <= 64;
    auto* ckey = (unsigned long long*)B(B_P_CKEY, 8ull * nc);
    auto* cidx = (int*)B(B_P_CIDX, keys ? 4ull : 4ull * nc);
    auto* skey = (unsigned long long*)B(B_P_SKEY, 8ull * nc);
    auto* sidx = (int*)B(B_P_SIDX, keys ? 4ull : 4ull * nc);
    auto* cpay = (float2*)B(B_P_DPT, 8ull * nc);
    auto* cub_out = (tgvg_cube*)B(B_P_OUT, sizeof(tgvg_cube) * nc);
    if (!ckey || !cidx || !skey || !sidx || !cpay || !cub_out) return TGVG_ERR_NOMEM;
    if (keys) k_stage1_join<true><<<(unsigned)tiles, PIX_THREADS, 0, st>>>(key, pay, sums, low, ib, ckey, cidx, cpay);
    else k_stage1_join<false><<<(unsigned)tiles, PIX_THREADS, 0, st>>>(key, pay, sums, low, ib, ckey, cidx, cpay);
    TGVG_LAUNCHED(ctx);
    // stable LSD radix sort by the code (library sort: the cube list is input
    // preparation, not the iterated path)
    size_t tb = 0;
    auto sort = [&](void* tmp) {
        return keys ? cub::DeviceRadixSort::SortKeys(tmp, tb, ckey, skey, (int)nc, ib, ib + high - low, st)
                    : cub::DeviceRadixSort::SortPairs(tmp, tb, ckey, skey, cidx, sidx, (int)nc, low, high, st);
    };
    TGVG_CK(ctx, sort(nullptr));
    void* tmp = B(B_P_TMP, std::max<size_t>(tb, 16));
    if (!tmp) return TGVG_ERR_NOMEM;
    TGVG_CK(ctx, sort(tmp));
    const unsigned eg = (unsigned)((nc + 255) / 256);
    if (keys) k_stage1_emit<true><<<eg, 256, 0, st>>>((int)nc, skey, sidx, low, ib, cpay, cub_out);
    else k_stage1_emit<false><<<eg, 256, 0, st>>>((int)nc, skey, sidx, low, ib, cpay, cub_out);
    TGVG_LAUNCHED(ctx);
    TGVG_CK(ctx, cudaMemcpyAsync(out, cub_out, sizeof(tgvg_cube) * nc, cudaMemcpyDeviceToHost, st));
    TGVG_CK(ctx, cudaStreamSynchronize(st));
    return TGVG_OK;
}

}  // namespace tgvg

using namespace tgvg;

extern "C" int tgvg_build_cubes(tgvg_ctx* ctx, const tgvg_depthmap* dm, const float* origin3, float r_root,
                                tgvg_cube* out, int64_t cap, int64_t* count) {
    if (!ctx || !dm || !origin3 || !count || dm->width < 0 || dm->height < 0 ||
        (int64_t(dm->width) * dm->height > 0 && !dm->depths) || !std::isfinite(r_root) || !(r_root > 0.0f))
        return TGVG_ERR_INVALID;
    std::lock_guard<std::mutex> lk(ctx->mu);
    return build_cubes(ctx, dm, origin3, r_root, out, cap, count);
}

extern "C" int tgvg_build_cubes_file(tgvg_ctx* ctx, const tgvg_depthmap* dm, const float* origin3, float r_root,
                                     const char* out_path) {
    int64_t n = 0;
    std::vector<tgvg_cube> cubes(size_t(std::max(0, dm ? dm->width : 0)) * size_t(std::max(0, dm ? dm->height : 0)));
    int rc = tgvg_build_cubes(ctx, dm, origin3, r_root, cubes.data(), int64_t(cubes.size()), &n);
    if (rc) return rc;
    cubes.resize(size_t(n));
    char hdr[16] = {'T', 'G', 'V', '1'};
    const uint32_t ver = 1, cnt = uint32_t(n);
    std::memcpy(hdr + 4, &ver, 4);
    std::memcpy(hdr + 8, &r_root, 4);
    std::memcpy(hdr + 12, &cnt, 4);
    rc = tgvg::fileio::write_file(out_path, hdr, 16, cubes.data(), sizeof(tgvg_cube) * size_t(n));
    return rc ? ctx->fail(rc, std::string("Cannot open output: ") + (out_path ? out_path : "")) : TGVG_OK;
}
