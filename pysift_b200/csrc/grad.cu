// grad.cu -- differentiable forms of the descriptor and of the warp + feather
// blend, with hand-written backward kernels (used by pysift_b200/grad.py).
//
// Descriptor (pysift/core.py:693-835 with keypoint location, scale and
// orientation held fixed): a keypoint is (centre row r0, centre column c0,
// angle in degrees) on one Gaussian level, patch half-width ph.  Each patch
// sample (r0 + dr, c0 + dc), |dr|, |dc| <= ph, inside the rotated 4x4-bin
// window contributes w_y * w_x * w_o * mag * gw to 8 trilinear bins; the
// descriptor is L2-normalise (+1e-14) -> clip 0.2 -> L2-normalise of the
// float histogram.  Backward: through the normalisation and clip to the
// histogram, then per sample through mag = |(dx, dy)|, the orientation
// theta = atan2(dy, dx) (which moves the orientation interpolation weights)
// into the central differences dx = G[r][c+1] - G[r][c-1],
// dy = G[r+1][c] - G[r-1][c] (float atomics into a map of (d/ddx, d/ddy) per
// pixel of the level; the pass that reads the map forms the differences'
// adjoint).  pysift_desc_levels_* run the whole function over the keypoints
// of all levels: the pyramid, one descriptor launch, and backward one adjoint
// launch a level.
//
// Blur adjoint: the transpose of the separable blur with half-sample
// symmetric reflection (pysift/core.py:477-483): a reflected tap folds back
// onto the pixel it was read from.
//
// Warp + feather (float form of image.cu k_warp_feather, no uint8 rounding):
// canvas pixel (u, v) samples image 1 at (sx, sy) = Hinv (u - ox, v - oy)
// (bilinear, zero outside), image 2 sits at integer offset (iox, ioy); where
// both cover, out = (w1 d1 + i2 d2) / (d1 + d2) with d = 1 + distance to the
// image's border.  Backward: image 2 directly, image 1 by the bilinear
// weights (atomics), Hinv through (sx, sy) -> bilinear slope and the feather
// weight d1 (block reduction, then float64 atomics).  Canvas geometry and the
// homography terms are computed in float64 (the images and pixel values stay
// float32): the per-pixel terms of the homography gradient cancel over the
// canvas.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "common.cuh"

namespace pysift {

constexpr int GD_T = 256;
constexpr float GD_PI = 3.14159265358979323846f;

struct DescSample {
    bool act;
    int rr, cc;
    float xr, yr, xb, yb;
};

__device__ __forceinline__ DescSample desc_sample(int idx, int side, int ph, int r0, int c0, int H, int W, float cos_a,
                                                  float sin_a, float scale_sp) {
    DescSample s;
    const int r_off = idx / side - ph, c_off = idx % side - ph;
    s.rr = r0 + r_off;
    s.cc = c0 + c_off;
    s.act = !(s.rr < 1 || s.rr >= H - 1 || s.cc < 1 || s.cc >= W - 1);
    const float fc = (float)c_off, fr = (float)r_off;
    s.xr = cos_a * fc - sin_a * fr;
    s.yr = sin_a * fc + cos_a * fr;
    s.xb = s.xr * scale_sp + 1.5f;
    s.yb = s.yr * scale_sp + 1.5f;
    s.act = s.act && !(s.xb < -0.5f || s.xb >= 3.5f || s.yb < -0.5f || s.yb >= 3.5f);
    return s;
}

struct Corners {
    int bin[8];
    float wsp[4];  // spatial weights of (y0,x0), (y0,x1), (y1,x0), (y1,x1)
    float df;      // orientation fraction: w_o0 = 1 - df, w_o1 = df
};

__device__ __forceinline__ Corners desc_corners(float xb, float yb, float ori_deg) {
    Corners k;
    const float ob = ori_deg * (8.0f / 360.0f);
    const int oi0 = (int)floorf(ob);
    k.df = ob - (float)oi0;
    const int xi0 = (int)floorf(xb), yi0 = (int)floorf(yb);
    const float dxb = xb - (float)xi0, dyb = yb - (float)yi0;
    const int xa = max(0, min(xi0, 3)), xc = max(0, min(xi0 + 1, 3));
    const int ya = max(0, min(yi0, 3)), yc = max(0, min(yi0 + 1, 3));
    const int o0 = ((oi0 % 8) + 8) % 8, o1 = ((oi0 + 1) % 8 + 8) % 8;
    k.wsp[0] = (1.0f - dyb) * (1.0f - dxb);
    k.wsp[1] = (1.0f - dyb) * dxb;
    k.wsp[2] = dyb * (1.0f - dxb);
    k.wsp[3] = dyb * dxb;
    const int sp[4] = {ya * 32 + xa * 8, ya * 32 + xc * 8, yc * 32 + xa * 8, yc * 32 + xc * 8};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        k.bin[2 * q] = sp[q] + o0;
        k.bin[2 * q + 1] = sp[q] + o1;
    }
    return k;
}

__device__ __forceinline__ float block_sum_f(float v, float* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL_MASK, v, o);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    float t = 0.0f;
    if (threadIdx.x < 32) {
        t = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.0f;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(FULL_MASK, t, o);
        if (threadIdx.x == 0) sh[32] = t;
    }
    __syncthreads();
    t = sh[32];
    __syncthreads();
    return t;
}

// The levels keypoints can sit on: entry octave * PYSIFT_MAX_LEVELS + scale
// index (the single-level entry points use entry 0).
struct DescLevel {
    const float* G;  // null: no such level
    float2* map;     // backward: (dL/ddx, dL/ddy) per pixel, pitch P, accumulated with atomics
    int H, W, P, ph;
};
constexpr int GD_LEVELS = PYSIFT_MAX_OCTAVES * PYSIFT_MAX_LEVELS;
struct DescTable {
    DescLevel lv[GD_LEVELS];
};

// keypoint rows: [r0, c0, angle in degrees], or with `levels` [entry, r0, c0, angle]
struct DescKp {
    const DescLevel* lv;
    int r0, c0;
    float ang, sin_a, cos_a;
    float scale_sp, inv_2s2;
    int side;
};

__device__ __forceinline__ DescKp desc_kp(const DescTable& tab, const float* __restrict__ kp, int k, bool levels) {
    DescKp d;
    const float* row = kp + (long long)k * (levels ? 4 : 3);
    int e = 0;
    if (levels) {
        e = (int)row[0];
        ++row;
    }
    d.lv = e >= 0 && e < GD_LEVELS && tab.lv[e].G ? &tab.lv[e] : nullptr;
    d.r0 = (int)row[0];
    d.c0 = (int)row[1];
    d.ang = row[2] * (GD_PI / 180.0f);
    sincosf(d.ang, &d.sin_a, &d.cos_a);
    const int ph = d.lv ? d.lv->ph : 1;
    d.scale_sp = 4.0f / (2.0f * (float)ph);
    const float sigma_d = (float)ph * 0.5657f;
    d.inv_2s2 = 1.0f / (2.0f * sigma_d * sigma_d + 1e-12f);
    d.side = 2 * ph + 1;
    return d;
}

// hist (n, 128) raw, desc (n, 128).  A block per keypoint.  Every lane adds
// its samples into a histogram of its own, 128 words at a stride of 32 (one
// bank a lane): a plain load, add and store per corner without conflicts,
// where a float atomic on shared memory is a compare-and-swap loop (1,068 us
// for the 2,000 keypoints of a 1024x768 image in twelve launches, 115 us so
// in one).  The corners that the clamp at the patch's rim maps to one cell
// are merged first, so a sample's eight words differ and its eight loads can
// be in flight together.
constexpr int GF_T = 128;
constexpr size_t GF_SMEM = (size_t)GF_T * 128 * sizeof(float);

__global__ void __launch_bounds__(GF_T) k_desc_f32_fwd(const __grid_constant__ DescTable tab,
                                                       const float* __restrict__ kp, int n, bool levels,
                                                       float* __restrict__ hist, float* __restrict__ desc) {
    extern __shared__ float lane_hist[];
    __shared__ float sh[33];
    const int tid = threadIdx.x;
    float* const h = lane_hist + (tid >> 5) * (128 * 32) + (tid & 31);
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
#pragma unroll 16
        for (int b = 0; b < 128; ++b) h[b * 32] = 0.0f;
        const DescKp d = desc_kp(tab, kp, k, levels);
        if (d.lv) {
            const float* __restrict__ G = d.lv->G;
            const int H = d.lv->H, W = d.lv->W, ph = d.lv->ph;
            const long long P = d.lv->P;
            for (int idx = tid; idx < d.side * d.side; idx += GF_T) {
                const DescSample s = desc_sample(idx, d.side, ph, d.r0, d.c0, H, W, d.cos_a, d.sin_a, d.scale_sp);
                if (!s.act) continue;
                const float* gp = G + (long long)s.rr * P + s.cc;
                const float dx = gp[1] - gp[-1], dy = gp[P] - gp[-P];
                const float mag = sqrtf(dx * dx + dy * dy);
                float ori = (atan2f(dy, dx) - d.ang) * (180.0f / GD_PI) + 360.0f;
                ori = ori >= 360.0f ? ori - 360.0f : ori;
                const float gw = expf(-(s.xr * s.xr + s.yr * s.yr) * d.inv_2s2);
                const float wm = mag * gw;
                const float ob = ori * (8.0f / 360.0f);
                const int oi0 = (int)floorf(ob);
                const float df = ob - (float)oi0;
                const int xi = (int)floorf(s.xb), yi = (int)floorf(s.yb);
                float wx1 = s.xb - (float)xi, wy1 = s.yb - (float)yi;
                float wx0 = 1.0f - wx1, wy0 = 1.0f - wy1;
                // xi, yi are in -1 .. 3: at either end both corners clamp to one
                // cell, which takes the whole weight; its neighbour gets nothing
                const bool mx = xi < 0 || xi > 2, my = yi < 0 || yi > 2;
                if (mx) wx0 = 1.0f;
                if (my) wy0 = 1.0f;
                const int xa = max(xi, 0), ya = max(yi, 0);
                const int xc = xi < 0 ? 1 : (xi > 2 ? 2 : xi + 1), yc = yi < 0 ? 1 : (yi > 2 ? 2 : yi + 1);
                const int o0 = oi0 & 7, o1 = (oi0 + 1) & 7;
                const float w[4] = {wy0 * wx0, wy0 * wx1, wy1 * wx0, wy1 * wx1};
                float* const c[4] = {h + (ya * 32 + xa * 8) * 32, h + (ya * 32 + xc * 8) * 32,
                                     h + (yc * 32 + xa * 8) * 32, h + (yc * 32 + xc * 8) * 32};
                float v0[4], v1[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v0[q] = c[q][o0 * 32];
                    v1[q] = c[q][o1 * 32];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (((q & 1) && mx) || ((q & 2) && my)) continue;
                    v0[q] += w[q] * (1.0f - df) * wm;
                    v1[q] += w[q] * df * wm;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    c[q][o0 * 32] = v0[q];
                    c[q][o1 * 32] = v1[q];
                }
            }
        }
        __syncthreads();
        // thread b sums bin b over the lanes, starting at its own bank
        float v = 0.0f;
        for (int w = 0; w < GF_T / 32; ++w) {
            const float* src = lane_hist + w * (128 * 32) + tid * 32;
            float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < 32; ++j) part[j & 3] += src[(j + tid) & 31];
            v += (part[0] + part[1]) + (part[2] + part[3]);
        }
        const float n1 = sqrtf(block_sum_f(v * v, sh) + 1e-14f);
        float t = v / n1;
        t = t > 0.2f ? 0.2f : t;
        const float n2 = sqrtf(block_sum_f(t * t, sh) + 1e-14f);
        hist[(long long)k * 128 + tid] = v;
        desc[(long long)k * 128 + tid] = t / n2;
    }
}

// gdesc: dL/ddesc (n, 128).  Into the level's map one vector atomic a sample
// (four scalar ones on the level's gradient, one a neighbour, were 210 us for
// 2,000 keypoints at 1024x768, this 99), or with gG != null (the single-level
// entry point) straight into the level's gradient.
__global__ void __launch_bounds__(GD_T) k_desc_f32_bwd(const __grid_constant__ DescTable tab,
                                                       const float* __restrict__ kp, int n, bool levels,
                                                       const float* __restrict__ hist,
                                                       const float* __restrict__ gdesc, float* __restrict__ gG) {
    __shared__ float hb[128];  // dL/dhist
    __shared__ float sh[33];
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        // backward of L2 -> clip 0.2 -> L2
        const bool own = threadIdx.x < 128;
        const float v = own ? hist[(long long)k * 128 + threadIdx.x] : 0.0f;
        const float gd = own ? gdesc[(long long)k * 128 + threadIdx.x] : 0.0f;
        const float n1 = sqrtf(block_sum_f(v * v, sh) + 1e-14f);
        const float t = v / n1;
        const float c = t > 0.2f ? 0.2f : t;
        const float n2 = sqrtf(block_sum_f(own ? c * c : 0.0f, sh) + 1e-14f);
        const float gc_dot = block_sum_f(gd * c, sh);
        const float gcv = gd / n2 - c * gc_dot / (n2 * n2 * n2);
        const float gt = (t > 0.2f) ? 0.0f : gcv;
        const float gt_dot = block_sum_f(gt * v, sh);
        const float gh = gt / n1 - v * gt_dot / (n1 * n1 * n1);
        if (own) hb[threadIdx.x] = gh;
        __syncthreads();
        const DescKp d = desc_kp(tab, kp, k, levels);
        const int H = d.lv ? d.lv->H : 0, W = d.lv ? d.lv->W : 0, ph = d.lv ? d.lv->ph : 0;
        const long long P = d.lv ? d.lv->P : 0;
        const int ns = d.lv ? d.side * d.side : 0;
        for (int idx = threadIdx.x; idx < ns; idx += GD_T) {
            const DescSample s = desc_sample(idx, d.side, ph, d.r0, d.c0, H, W, d.cos_a, d.sin_a, d.scale_sp);
            if (!s.act) continue;
            const float* gp = d.lv->G + (long long)s.rr * P + s.cc;
            const float dx = gp[1] - gp[-1], dy = gp[P] - gp[-P];
            const float m2 = dx * dx + dy * dy;
            if (!(m2 > 0.0f)) continue;
            const float mag = sqrtf(m2);
            float ori = (atan2f(dy, dx) - d.ang) * (180.0f / GD_PI) + 360.0f;
            ori = ori >= 360.0f ? ori - 360.0f : ori;
            const float gw = expf(-(s.xr * s.xr + s.yr * s.yr) * d.inv_2s2);
            const Corners cr = desc_corners(s.xb, s.yb, ori);
            float gmag = 0.0f, gdf = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float g0 = hb[cr.bin[2 * q]], g1 = hb[cr.bin[2 * q + 1]];
                gmag += cr.wsp[q] * ((1.0f - cr.df) * g0 + cr.df * g1);
                gdf += cr.wsp[q] * (g1 - g0);
            }
            gmag *= gw;
            // d(df)/d(theta) = (180 / pi) / 45 per radian
            const float gth = gdf * gw * mag * (4.0f / GD_PI);
            const float gdx = gmag * dx / mag - gth * dy / m2;
            const float gdy = gmag * dy / mag + gth * dx / m2;
            const long long at = (long long)s.rr * P + s.cc;
            if (gG) {
                atomicAdd(gG + at + 1, gdx);
                atomicAdd(gG + at - 1, -gdx);
                atomicAdd(gG + at + P, gdy);
                atomicAdd(gG + at - P, -gdy);
            } else {
                atomicAdd(d.lv->map + at, make_float2(gdx, gdy));
            }
        }
        __syncthreads();
    }
}

// What is added to a blur adjoint: the adjoint of the central differences of
// a level's map, and at even rows and columns the gradient of the octave that
// the level was subsampled into.
struct AdjTail {
    const float2* map;
    int map_pitch;
    const float* sub;
    int sub_pitch;
    __device__ __forceinline__ float at(int y, int x, int H, int W) const {
        float v = 0.0f;
        if (map) {
            const float2* m = map + (long long)y * map_pitch + x;
            if (x > 0) v += m[-1].x;
            if (x + 1 < W) v -= m[1].x;
            if (y > 0) v += m[-(long long)map_pitch].y;
            if (y + 1 < H) v -= m[map_pitch].y;
        }
        if (sub && !((y | x) & 1)) v += sub[(long long)(y >> 1) * sub_pitch + (x >> 1)];
        return v;
    }
};

struct AdjArgs {
    const float* in;
    long long in_pitch;
    float* out;
    long long out_pitch;
    int H, W;
    float w[PYSIFT_MAX_TAPS];
    const float* wdev;  // device weights in place of w (k_blur_adjoint_axis)
    bool accumulate;    // out += (k_blur_adjoint_axis)
    AdjTail tail;
};

// One axis of the adjoint of y[i] = sum_k w[k] x[refl(i + k - R)] (half-sample
// symmetric reflection, R < n): x_bar[j] = sum_k w[k] sum over the reads of
// pixel j.  axis 0: along rows (x), with the tail; axis 1: along columns (y).
// For any taps and radius, and in place.
__global__ void k_blur_adjoint_axis(const __grid_constant__ AdjArgs a, int R, int axis) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= a.W || y >= a.H) return;
    const int n = axis == 0 ? a.W : a.H, j = axis == 0 ? x : y;
    float acc = 0.0f;
    for (int k = 0; k <= 2 * R; ++k) {
        const float wk = a.wdev ? a.wdev[k] : a.w[k];
        const int cand[3] = {j - k + R, -1 - j - k + R, 2 * n - 1 - j - k + R};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int i = cand[q];
            if (i < 0 || i >= n) continue;
            acc += wk * (axis == 0 ? a.in[(long long)y * a.in_pitch + i] : a.in[(long long)i * a.in_pitch + x]);
        }
    }
    float* o = a.out + (long long)y * a.out_pitch + x;
    if (axis == 0) acc += a.tail.at(y, x, a.H, a.W);
    *o = axis == 0 && a.accumulate ? *o + acc : acc;
}

// Both axes of the adjoint of one 64 x 32 tile, for symmetric taps: then
// B[i][j] = w(j - i) + w(-1 - j - i) + w(2 n - 1 - j - i) is its own transpose
// (w(t) the tap at offset t), so the adjoint is the reflecting blur itself.
// Columns first, into a strip of 64 + 2 R columns, then rows; both passes
// slide a register window over 8 outputs.  One tile pass with the differences
// and the subsampling in its tail replaces two passes over global memory and
// their three candidate reads a tap: 286 us for the 16 levels of a
// 1024x768 image, now 103 with the tails.
constexpr int ADJ_TW = 64, ADJ_TH = 32, ADJ_T = 256;
template <int R>
struct AdjTile {
    static constexpr int ROWS = ADJ_TH + 2 * R, COLS = ADJ_TW + 2 * R, TS = COLS | 1;
    static constexpr size_t bytes = (size_t)(ROWS + ADJ_TH) * TS * sizeof(float);
};
static_assert(AdjTile<16>::bytes <= 48 * 1024, "the tiles stay within the default dynamic shared memory");

template <int R>
__global__ void __launch_bounds__(ADJ_T) k_blur_adjoint(const __grid_constant__ AdjArgs a) {
    using T = AdjTile<R>;
    extern __shared__ float adj_smem[];
    float* const tile = adj_smem;             // input rows [r0 - R, r0 + TH + R), columns [c0 - R, c0 + TW + R)
    float* const mid = adj_smem + T::ROWS * T::TS;
    const int c0 = blockIdx.x * ADJ_TW, r0 = blockIdx.y * ADJ_TH;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int CQ = (T::COLS + 31) / 32;
    int gc[CQ];
#pragma unroll
    for (int q = 0; q < CQ; ++q) gc[q] = reflect_idx(c0 - R + lane + 32 * q, a.W);
    for (int rr = warp; rr < T::ROWS; rr += ADJ_T / 32) {
        const float* src = a.in + (long long)reflect_idx(r0 - R + rr, a.H) * a.in_pitch;
#pragma unroll
        for (int q = 0; q < CQ; ++q)
            if (lane + 32 * q < T::COLS) tile[rr * T::TS + lane + 32 * q] = src[gc[q]];
    }
    __syncthreads();
    for (int i = tid; i < T::COLS * (ADJ_TH / 8); i += ADJ_T) {
        const int cc = i % T::COLS, j0 = (i / T::COLS) * 8;
        float v[8 + 2 * R];
#pragma unroll
        for (int m = 0; m < 8 + 2 * R; ++m) v[m] = tile[(j0 + m) * T::TS + cc];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * R; ++k) acc = fmaf(a.w[k], v[j + k], acc);
            mid[(j0 + j) * T::TS + cc] = acc;
        }
    }
    __syncthreads();
    {
        float v[8 + 2 * R];
#pragma unroll
        for (int m = 0; m < 8 + 2 * R; ++m) v[m] = mid[lane * T::TS + warp * 8 + m];
        // the tile is free: the outputs go through it, so that a warp stores whole rows
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * R; ++k) acc = fmaf(a.w[k], v[j + k], acc);
            tile[lane * T::TS + warp * 8 + j] = acc;
        }
    }
    __syncthreads();
    for (int i = tid; i < ADJ_TH * ADJ_TW; i += ADJ_T) {
        const int y = r0 + i / ADJ_TW, x = c0 + i % ADJ_TW;
        if (y < a.H && x < a.W)
            a.out[(long long)y * a.out_pitch + x] = tile[(i / ADJ_TW) * T::TS + i % ADJ_TW] + a.tail.at(y, x, a.H, a.W);
    }
}

// the tail alone (the top level of an octave)
__global__ void __launch_bounds__(256) k_adjoint_tail(float* __restrict__ out, int out_pitch, int H, int W,
                                                      const AdjTail tail) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x < W) out[(long long)y * out_pitch + x] = tail.at(y, x, H, W);
}

template <int R>
static void adj_launch(const AdjArgs& a, cudaStream_t st) {
    k_blur_adjoint<R><<<dim3(ceil_div(a.W, ADJ_TW), ceil_div(a.H, ADJ_TH)), ADJ_T, AdjTile<R>::bytes, st>>>(a);
}

constexpr int ADJ_MAX_R = 16;  // radii of the tiled kernel

// tmp: as large as the input, for the two-pass form
static int launch_adjoint_axes(const AdjArgs& a, int R, float* tmp, int tmp_pitch, cudaStream_t st) {
    const dim3 grid(ceil_div(a.W, 128), a.H);
    // forward = horizontal then vertical; adjoint = vertical^T then horizontal^T
    AdjArgs b = a;
    b.out = tmp;
    b.out_pitch = tmp_pitch;
    k_blur_adjoint_axis<<<grid, 128, 0, st>>>(b, R, 1);
    PYSIFT_LAUNCH_CHECK("k_blur_adjoint_axis");
    b = a;
    b.in = tmp;
    b.in_pitch = tmp_pitch;
    k_blur_adjoint_axis<<<grid, 128, 0, st>>>(b, R, 0);
    PYSIFT_LAUNCH_CHECK("k_blur_adjoint_axis");
    return PYSIFT_OK;
}

// The tiled kernel for the taps it is right and compiled for (the Gaussian
// tables are symmetric bit for bit), the two-pass form for the others.
static bool adjoint_tiled(const float* w, int R) {
    bool tiled = R <= ADJ_MAX_R;
    for (int k = 0; k < R; ++k) tiled = tiled && w[k] == w[2 * R - k];
    return tiled;
}

static int launch_adjoint(const AdjArgs& a, int R, float* tmp, int tmp_pitch, cudaStream_t st) {
    if (!adjoint_tiled(a.w, R)) return launch_adjoint_axes(a, R, tmp, tmp_pitch, st);
    switch (R) {
        case 0: adj_launch<0>(a, st); break;
        case 1: adj_launch<1>(a, st); break;
        case 2: adj_launch<2>(a, st); break;
        case 3: adj_launch<3>(a, st); break;
        case 4: adj_launch<4>(a, st); break;
        case 5: adj_launch<5>(a, st); break;
        case 6: adj_launch<6>(a, st); break;
        case 7: adj_launch<7>(a, st); break;
        case 8: adj_launch<8>(a, st); break;
        case 9: adj_launch<9>(a, st); break;
        case 10: adj_launch<10>(a, st); break;
        case 11: adj_launch<11>(a, st); break;
        case 12: adj_launch<12>(a, st); break;
        case 13: adj_launch<13>(a, st); break;
        case 14: adj_launch<14>(a, st); break;
        case 15: adj_launch<15>(a, st); break;
        default: adj_launch<16>(a, st); break;
    }
    PYSIFT_LAUNCH_CHECK("k_blur_adjoint");
    return PYSIFT_OK;
}

static int launch_desc_fwd(const DescTable& tab, const float* kp, int n, bool levels, float* hist, float* desc,
                           cudaStream_t st) {
    PYSIFT_CUDA_TRY(cudaFuncSetAttribute(k_desc_f32_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GF_SMEM));
    // three resident blocks an SM; more blocks than that keep the tail short
    k_desc_f32_fwd<<<std::min(n, 148 * 12), GF_T, GF_SMEM, st>>>(tab, kp, n, levels, hist, desc);
    PYSIFT_LAUNCH_CHECK("k_desc_f32_fwd");
    return PYSIFT_OK;
}

static int launch_desc_bwd(const DescTable& tab, const float* kp, int n, bool levels, const float* hist,
                           const float* gdesc, float* gG, cudaStream_t st) {
    k_desc_f32_bwd<<<std::min(n, 148 * 8), GD_T, 0, st>>>(tab, kp, n, levels, hist, gdesc, gG);
    PYSIFT_LAUNCH_CHECK("k_desc_f32_bwd");
    return PYSIFT_OK;
}

// Workspace of pysift_desc_levels_*: the Gaussian levels 0 .. top of every
// octave in use, and backward a map for each level that keypoints sit on (all,
// when `levels` is null).  Once the maps are filled the levels are not needed
// any more: the chain of adjoints runs in their planes (0 and 1 in turn, plane
// min(2, top) for the octave's level-0 gradient).
struct LevelsLayout {
    int n_oct, top;
    int H[PYSIFT_MAX_OCTAVES], W[PYSIFT_MAX_OCTAVES], P[PYSIFT_MAX_OCTAVES];
    bool used[GD_LEVELS];
    size_t off_lev[PYSIFT_MAX_OCTAVES], off_map[GD_LEVELS], off_tmp;
    size_t map_begin, map_end, total;
    size_t plane(int o) const { return (size_t)H[o] * P[o]; }
};

static int levels_layout(const pysift_detect_config* cfg, int H, int W, int n_oct, int top, const uint8_t* levels,
                         bool backward, LevelsLayout& l) {
    PYSIFT_CHECK_ARG(cfg, "config is NULL");
    PYSIFT_CHECK_ARG(H > 2 && W > 2, "image size %dx%d too small", H, W);
    PYSIFT_CHECK_ARG(n_oct >= 1 && n_oct <= PYSIFT_MAX_OCTAVES, "n_octaves %d outside 1..%d", n_oct,
                     PYSIFT_MAX_OCTAVES);
    PYSIFT_CHECK_ARG(cfg->n_scales >= 1 && cfg->n_scales + 3 <= PYSIFT_MAX_LEVELS, "n_scales out of range");
    PYSIFT_CHECK_ARG(top >= cfg->n_scales && top <= cfg->n_scales + 2, "top level %d outside %d..%d", top,
                     cfg->n_scales, cfg->n_scales + 2);
    for (int i = 1; i < 2 + top; ++i)
        PYSIFT_CHECK_ARG(cfg->blur_radius[i] >= 0 && cfg->blur_radius[i] <= PYSIFT_MAX_RADIUS,
                         "blur radius %d outside 0..%d", cfg->blur_radius[i], PYSIFT_MAX_RADIUS);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t r = off;
        off = align_up(off + bytes, 256);
        return r;
    };
    l.n_oct = n_oct;
    l.top = top;
    for (int o = 0; o < n_oct; ++o) {
        l.H[o] = o ? (l.H[o - 1] + 1) / 2 : H;
        l.W[o] = o ? (l.W[o - 1] + 1) / 2 : W;
        PYSIFT_CHECK_ARG(l.H[o] > 2 && l.W[o] > 2, "octave %d of a %dx%d image is too small", o, H, W);
        l.P[o] = (int)align_up((size_t)l.W[o], 32);
    }
    for (int o = 0; o < n_oct; ++o) l.off_lev[o] = take((size_t)(top + 1) * l.plane(o) * sizeof(float));
    l.map_begin = off;
    for (int o = 0; o < n_oct; ++o)
        for (int s = 0; s <= top; ++s) {
            const int e = o * PYSIFT_MAX_LEVELS + s;
            l.used[e] = !levels || levels[e];
            if (backward && l.used[e]) l.off_map[e] = take(l.plane(o) * sizeof(float2));
        }
    l.map_end = off;
    bool tmp = false;  // a plane more for the two-pass adjoint
    for (int s = -1; backward && s < top; ++s) tmp = tmp || !adjoint_tiled(cfg->blur_weights[2 + s], cfg->blur_radius[2 + s]);
    if (tmp) l.off_tmp = take(l.plane(0) * sizeof(float));
    l.total = off;
    return PYSIFT_OK;
}

static float* lev_at(void* ws, const LevelsLayout& l, int o, int s) {
    return reinterpret_cast<float*>(static_cast<char*>(ws) + l.off_lev[o]) + (size_t)s * l.plane(o);
}
static float2* map_at(void* ws, const LevelsLayout& l, int o, int s) {
    const int e = o * PYSIFT_MAX_LEVELS + s;
    return l.used[e] ? reinterpret_cast<float2*>(static_cast<char*>(ws) + l.off_map[e]) : nullptr;
}

// Gaussian levels of the non-doubled image (pysift/core.py:1288-1343)
static int build_levels(const pysift_detect_config* cfg, const float* img, int pitch, void* ws, const LevelsLayout& l,
                        cudaStream_t st) {
    for (int o = 0; o < l.n_oct; ++o) {
        const int H = l.H[o], W = l.W[o], P = l.P[o];
        if (o == 0) {
            const int rc = blur_level(img, pitch, 1, lev_at(ws, l, 0, 0), P, nullptr, H, W, cfg->blur_weights[1],
                                      cfg->blur_radius[1], false, st);
            if (rc) return rc;
        }
        for (int s = 0; s < l.top; ++s) {
            const bool first = o > 0 && s == 0;  // reads level S of the octave before at every second pixel
            const float* in = first ? lev_at(ws, l, o - 1, cfg->n_scales) : lev_at(ws, l, o, s);
            const int rc = blur_level(in, first ? l.P[o - 1] : P, first ? 2 : 1, lev_at(ws, l, o, s + 1), P,
                                      first ? lev_at(ws, l, o, 0) : nullptr, H, W, cfg->blur_weights[2 + s],
                                      cfg->blur_radius[2 + s], true, st);
            if (rc) return rc;
        }
    }
    return PYSIFT_OK;
}

static void levels_table(const pysift_detect_config* cfg, void* ws, const LevelsLayout& l, bool backward,
                         DescTable& tab) {
    memset(&tab, 0, sizeof(tab));
    for (int o = 0; o < l.n_oct; ++o)
        for (int s = 0; s <= l.top; ++s) {
            const int ph = (int)cfg->desc_ph[s];
            if (ph < 1 || ph > 200 || !l.used[o * PYSIFT_MAX_LEVELS + s]) continue;
            DescLevel& v = tab.lv[o * PYSIFT_MAX_LEVELS + s];
            v.G = lev_at(ws, l, o, s);
            v.map = backward ? map_at(ws, l, o, s) : nullptr;
            v.H = l.H[o];
            v.W = l.W[o];
            v.P = l.P[o];
            v.ph = ph;
        }
}

struct WarpF32Args {
    const float* img1;
    int hs, ws, C;
    const float* img2;
    int h2, w2;
    int cw, ch;
    double hinv[9];
    double ox, oy;
    int iox, ioy;
    float* out;      // (ch, cw, C)
    const float* gout;
    float* gimg1;    // (hs, ws, C), atomics
    float* gimg2;    // (h2, w2, C)
    double* ghinv;   // 9, atomics
};

struct WarpGeom {
    bool v1, v2, clamped;
    double X, Y, den, sx, sy;
    float d1, d2;
    int x0, y0, x2, y2;
    float fx, fy;
};

__device__ __forceinline__ WarpGeom warp_geom(const WarpF32Args& a, int u, int v) {
    WarpGeom g;
    g.X = (double)u - a.ox;
    g.Y = (double)v - a.oy;
    const double s0 = a.hinv[0] * g.X + a.hinv[1] * g.Y + a.hinv[2];
    const double s1 = a.hinv[3] * g.X + a.hinv[4] * g.Y + a.hinv[5];
    const double s2 = a.hinv[6] * g.X + a.hinv[7] * g.Y + a.hinv[8];
    g.clamped = !(s2 >= 1e-10);
    g.den = g.clamped ? 1e-10 : s2;
    g.sx = s0 / g.den;
    g.sy = s1 / g.den;
    g.v1 = g.sx >= 0.0 && g.sx <= (double)(a.ws - 1) && g.sy >= 0.0 && g.sy <= (double)(a.hs - 1);
    g.x0 = (int)floor(g.sx);
    g.y0 = (int)floor(g.sy);
    g.fx = (float)(g.sx - (double)g.x0);
    g.fy = (float)(g.sy - (double)g.y0);
    g.d1 = (float)(1.0 + fmin(fmin(g.sx, (double)(a.ws - 1) - g.sx), fmin(g.sy, (double)(a.hs - 1) - g.sy)));
    g.x2 = u - a.iox;
    g.y2 = v - a.ioy;
    g.v2 = g.x2 >= 0 && g.x2 < a.w2 && g.y2 >= 0 && g.y2 < a.h2;
    g.d2 = 1.0f + (float)min(min(g.x2, a.w2 - 1 - g.x2), min(g.y2, a.h2 - 1 - g.y2));
    return g;
}

__device__ __forceinline__ float img1_at(const WarpF32Args& a, int x, int y, int c) {
    return (x >= 0 && x < a.ws && y >= 0 && y < a.hs) ? a.img1[((long long)y * a.ws + x) * a.C + c] : 0.0f;
}

__global__ void k_warp_f32_fwd(const WarpF32Args a) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (u >= a.cw) return;
    const WarpGeom g = warp_geom(a, u, v);
    for (int c = 0; c < a.C; ++c) {
        float w1 = 0.0f;
        if (g.v1) {
            const float p00 = img1_at(a, g.x0, g.y0, c), p01 = img1_at(a, g.x0 + 1, g.y0, c);
            const float p10 = img1_at(a, g.x0, g.y0 + 1, c), p11 = img1_at(a, g.x0 + 1, g.y0 + 1, c);
            w1 = (1.0f - g.fy) * ((1.0f - g.fx) * p00 + g.fx * p01) + g.fy * ((1.0f - g.fx) * p10 + g.fx * p11);
        }
        const float i2 = g.v2 ? a.img2[((long long)g.y2 * a.w2 + g.x2) * a.C + c] : 0.0f;
        float o = 0.0f;
        if (g.v1 && g.v2) o = (w1 * g.d1 + i2 * g.d2) / (g.d1 + g.d2);
        else if (g.v2) o = i2;
        else if (g.v1) o = w1;
        a.out[((long long)v * a.cw + u) * a.C + c] = o;
    }
}

// A block takes WB_T columns of every gridDim.y-th canvas row and adds its nine
// homography sums to global memory once: one block a row and 256 columns put
// thousands of float64 atomics on nine addresses.  Adjacent canvas pixels
// mostly read adjacent image-1 pixels, so a lane hands its right-hand corner
// gradients to the next lane when that lane's left-hand corners are the same
// pixels: half the float atomics.  66.7 -> 46.7 us for the 1024x768x3 views of
// a canvas of 1 Mpixel, whose images, gradients and output gradient are 12 us
// of DRAM traffic.  Eight blocks an SM leave 64 registers; three channels spill
// 132 bytes under that.
constexpr int WB_T = 128;
template <int C>
__global__ void __launch_bounds__(WB_T, 8) k_warp_f32_bwd(const __grid_constant__ WarpF32Args a) {
    __shared__ double sh[9][WB_T / 32];
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double gh[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int v = blockIdx.y; v < a.ch; v += gridDim.y) {
        WarpGeom g = {};
        if (u < a.cw) g = warp_geom(a, u, v);
        double gsx = 0.0, gsy = 0.0, gd1 = 0.0;
        float corner[4][C];
        bool some = false;  // any corner gradient to add
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const float go = u < a.cw ? a.gout[((long long)v * a.cw + u) * C + c] : 0.0f;
            float w1 = 0.0f, dwdx = 0.0f, dwdy = 0.0f, p00 = 0, p01 = 0, p10 = 0, p11 = 0;
            if (g.v1) {
                p00 = img1_at(a, g.x0, g.y0, c);
                p01 = img1_at(a, g.x0 + 1, g.y0, c);
                p10 = img1_at(a, g.x0, g.y0 + 1, c);
                p11 = img1_at(a, g.x0 + 1, g.y0 + 1, c);
                w1 = (1.0f - g.fy) * ((1.0f - g.fx) * p00 + g.fx * p01) + g.fy * ((1.0f - g.fx) * p10 + g.fx * p11);
                dwdx = (1.0f - g.fy) * (p01 - p00) + g.fy * (p11 - p10);
                dwdy = (1.0f - g.fx) * (p10 - p00) + g.fx * (p11 - p01);
            }
            float gw1 = 0.0f;
            if (g.v1 && g.v2) {
                const float i2 = a.img2[((long long)g.y2 * a.w2 + g.x2) * C + c];
                const float s = g.d1 + g.d2;
                const float o = (w1 * g.d1 + i2 * g.d2) / s;
                gw1 = go * g.d1 / s;
                a.gimg2[((long long)g.y2 * a.w2 + g.x2) * C + c] += go * g.d2 / s;
                gd1 += go * (w1 - o) / s;
            } else if (g.v2) {
                a.gimg2[((long long)g.y2 * a.w2 + g.x2) * C + c] += go;
            } else if (g.v1) {
                gw1 = go;
            }
            const float wts[4] = {(1.0f - g.fy) * (1.0f - g.fx), (1.0f - g.fy) * g.fx, g.fy * (1.0f - g.fx),
                                  g.fy * g.fx};
            const bool on = g.v1 && gw1 != 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) corner[q][c] = on ? gw1 * wts[q] : 0.0f;
            if (on) {
                some = true;
                gsx += gw1 * dwdx;
                gsy += gw1 * dwdy;
            }
        }
        // corner q of a pixel: column x0 + (q & 1), row y0 + (q >> 1)
        const int xn = __shfl_down_sync(FULL_MASK, g.x0, 1), yn = __shfl_down_sync(FULL_MASK, g.y0, 1);
        const bool on_next = __shfl_down_sync(FULL_MASK, (int)some, 1) != 0;
        const bool give = some && lane < 31 && on_next && xn == g.x0 + 1 && yn == g.y0;
        const bool take = __shfl_up_sync(FULL_MASK, (int)give, 1) != 0 && lane > 0;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int q = 1; q < 4; q += 2) {
                const float from = __shfl_up_sync(FULL_MASK, corner[q][c], 1);
                if (take) corner[q - 1][c] += from;
            }
        if (some) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int x = g.x0 + (q & 1), y = g.y0 + (q >> 1);
                if ((give && (q & 1)) || x < 0 || x >= a.ws || y < 0 || y >= a.hs) continue;
                float* dst = a.gimg1 + ((long long)y * a.ws + x) * C;
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (corner[q][c] != 0.0f) atomicAdd(dst + c, corner[q][c]);
            }
        }
        if (g.v1 && g.v2) {
            // d1 = 1 + min(sx, ws-1-sx, sy, hs-1-sy): slope of the active term
            const double t0 = g.sx, t1 = (double)(a.ws - 1) - g.sx, t2 = g.sy, t3 = (double)(a.hs - 1) - g.sy;
            const double m = fmin(fmin(t0, t1), fmin(t2, t3));
            if (m == t0) gsx += gd1;
            else if (m == t1) gsx -= gd1;
            else if (m == t2) gsy += gd1;
            else gsy -= gd1;
        }
        if (g.v1 && !g.clamped) {
            const double r = 1.0 / g.den;
            const double a0 = gsx * r, a1 = gsy * r, a2 = -(gsx * g.sx + gsy * g.sy) * r;
            gh[0] += a0 * g.X; gh[1] += a0 * g.Y; gh[2] += a0;
            gh[3] += a1 * g.X; gh[4] += a1 * g.Y; gh[5] += a1;
            gh[6] += a2 * g.X; gh[7] += a2 * g.Y; gh[8] += a2;
        }
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        double x = gh[q];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(FULL_MASK, x, o);
        if (lane == 0) sh[q][warp] = x;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[threadIdx.x][w];
        atomicAdd(&a.ghinv[threadIdx.x], s);
    }
}

struct Mat3 {
    double m[9];
};

// the gradient of the 8 parameters of H from that of its inverse:
// -(Hinv^T G Hinv^T), row-major, without the last entry
__global__ void k_homography_adjoint(const Mat3 hinv, const double* __restrict__ g, double* __restrict__ g8) {
    const int i = threadIdx.x / 3, j = threadIdx.x % 3;
    if (threadIdx.x >= 8) return;
    double s = 0.0;
    for (int k = 0; k < 3; ++k) {
        double t = 0.0;
        for (int l = 0; l < 3; ++l) t = fma(hinv.m[l * 3 + i], g[l * 3 + k], t);
        s = fma(t, hinv.m[j * 3 + k], s);
    }
    g8[threadIdx.x] = -s;
}

}  // namespace pysift

using namespace pysift;

extern "C" {

static void one_level(const float* level, int H, int W, int pitch, int ph, DescTable& tab) {
    memset(&tab, 0, sizeof(tab));
    tab.lv[0] = DescLevel{level, nullptr, H, W, pitch, ph};
}

int pysift_desc_f32_forward(const float* level, int32_t H, int32_t W, int32_t pitch, const float* kp, int32_t n,
                            int32_t ph, float* hist, float* desc, pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(level && kp && hist && desc && H > 2 && W > 2 && pitch >= W && n >= 0 && ph >= 1 && ph <= 200,
                     "bad arguments");
    if (n == 0) return PYSIFT_OK;
    DescTable tab;
    one_level(level, H, W, pitch, ph, tab);
    return launch_desc_fwd(tab, kp, n, false, hist, desc, reinterpret_cast<cudaStream_t>(stream));
}

int pysift_desc_f32_backward(const float* level, int32_t H, int32_t W, int32_t pitch, const float* kp, int32_t n,
                             int32_t ph, const float* hist, const float* gdesc, float* glevel,
                             pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(level && kp && hist && gdesc && glevel && H > 2 && W > 2 && pitch >= W && n >= 0 && ph >= 1 &&
                         ph <= 200,
                     "bad arguments");
    if (n == 0) return PYSIFT_OK;
    DescTable tab;
    one_level(level, H, W, pitch, ph, tab);
    return launch_desc_bwd(tab, kp, n, false, hist, gdesc, glevel, reinterpret_cast<cudaStream_t>(stream));
}

int pysift_blur_adjoint(const float* gout, int32_t gout_pitch, float* gin, int32_t gin_pitch, float* tmp,
                        int32_t tmp_pitch, int32_t H, int32_t W, const float* weights_dev, int32_t radius,
                        int32_t accumulate, pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(gout && gin && tmp && weights_dev && H > 0 && W > 0, "bad arguments");
    PYSIFT_CHECK_ARG(radius >= 0 && radius < H && radius < W && radius <= PYSIFT_MAX_RADIUS,
                     "radius %d must be below both image sides", radius);
    AdjArgs a = {};
    a.in = gout;
    a.in_pitch = gout_pitch;
    a.out = gin;
    a.out_pitch = gin_pitch;
    a.H = H;
    a.W = W;
    a.wdev = weights_dev;
    a.accumulate = accumulate != 0;
    return launch_adjoint_axes(a, radius, tmp, tmp_pitch, reinterpret_cast<cudaStream_t>(stream));
}

int pysift_desc_levels_workspace_size(const pysift_detect_config* cfg, int32_t H, int32_t W, int32_t n_octaves,
                                      int32_t top, const uint8_t* levels, int32_t backward, size_t* bytes) {
    PYSIFT_CHECK_ARG(bytes != nullptr, "bytes is NULL");
    LevelsLayout l = {};
    const int rc = levels_layout(cfg, H, W, n_octaves, top, levels, backward != 0, l);
    if (rc) return rc;
    *bytes = l.total;
    return PYSIFT_OK;
}

int pysift_desc_levels_forward(const pysift_detect_config* cfg, const float* img, int32_t H, int32_t W, int32_t pitch,
                               const float* kp, int32_t n, int32_t n_octaves, int32_t top, const uint8_t* levels,
                               void* workspace, size_t workspace_bytes, float* hist, float* desc,
                               pysift_stream_t stream) {
    LevelsLayout l = {};
    int rc = levels_layout(cfg, H, W, n_octaves, top, levels, false, l);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(img && workspace && pitch >= W && n >= 0 && (n == 0 || (kp && hist && desc)), "bad arguments");
    PYSIFT_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "workspace must be 256-byte aligned");
    if (workspace_bytes < l.total) {
        set_error("workspace %zu bytes < required %zu", workspace_bytes, l.total);
        return PYSIFT_ERR_WORKSPACE;
    }
    if (n == 0) return PYSIFT_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    rc = build_levels(cfg, img, pitch, workspace, l, st);
    if (rc) return rc;
    DescTable tab;
    levels_table(cfg, workspace, l, false, tab);
    return launch_desc_fwd(tab, kp, n, true, hist, desc, st);
}

int pysift_desc_levels_backward(const pysift_detect_config* cfg, const float* img, int32_t H, int32_t W, int32_t pitch,
                                const float* kp, int32_t n, int32_t n_octaves, int32_t top, const uint8_t* levels,
                                void* workspace, size_t workspace_bytes, const float* hist, const float* gdesc,
                                float* gimg, int32_t gimg_pitch, pysift_stream_t stream) {
    LevelsLayout l = {};
    int rc = levels_layout(cfg, H, W, n_octaves, top, levels, true, l);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(img && workspace && gimg && pitch >= W && gimg_pitch >= W && n >= 0 &&
                         (n == 0 || (kp && hist && gdesc)),
                     "bad arguments");
    PYSIFT_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "workspace must be 256-byte aligned");
    for (int o = 0; o < n_octaves; ++o)
        for (int s = o ? 0 : -1; s < top; ++s) {
            const int R = cfg->blur_radius[2 + s];
            PYSIFT_CHECK_ARG(R < l.H[o] && R < l.W[o], "radius %d must be below both image sides", R);
        }
    if (workspace_bytes < l.total) {
        set_error("workspace %zu bytes < required %zu", workspace_bytes, l.total);
        return PYSIFT_ERR_WORKSPACE;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    rc = build_levels(cfg, img, pitch, ws, l, st);
    if (rc) return rc;
    PYSIFT_CUDA_TRY(cudaMemsetAsync(ws + l.map_begin, 0, l.map_end - l.map_begin, st));
    if (n > 0) {
        DescTable tab;
        levels_table(cfg, ws, l, true, tab);
        rc = launch_desc_bwd(tab, kp, n, true, hist, gdesc, nullptr, st);
        if (rc) return rc;
    }
    // the adjoint of the level chain, highest octave first
    for (int o = n_octaves - 1; o >= 0; --o) {
        const int Ho = l.H[o], Wo = l.W[o], P = l.P[o];
        auto tail = [&](int s) {
            AdjTail t = {};
            t.map = map_at(ws, l, o, s);
            t.map_pitch = P;
            if (s == cfg->n_scales && o + 1 < n_octaves) {
                t.sub = lev_at(ws, l, o + 1, std::min(2, top));
                t.sub_pitch = l.P[o + 1];
            }
            return t;
        };
        float* const chain[2] = {lev_at(ws, l, o, 0), lev_at(ws, l, o, 1)};
        float* cur = chain[0];
        k_adjoint_tail<<<dim3(ceil_div(Wo, 256), Ho), 256, 0, st>>>(cur, P, Ho, Wo, tail(top));
        PYSIFT_LAUNCH_CHECK("k_adjoint_tail");
        for (int s = top; s >= (o ? 1 : 0); --s) {
            // level s -> level s - 1 (s = 0: the base blur, into the image's gradient)
            AdjArgs a = {};
            a.in = cur;
            a.in_pitch = P;
            a.out = s == 0 ? gimg : (s == 1 ? lev_at(ws, l, o, std::min(2, top)) : chain[(top - s + 1) & 1]);
            a.out_pitch = s == 0 ? gimg_pitch : P;
            a.H = Ho;
            a.W = Wo;
            const int R = cfg->blur_radius[1 + s];
            for (int k = 0; k <= 2 * R; ++k) a.w[k] = cfg->blur_weights[1 + s][k];
            if (s > 0) a.tail = tail(s - 1);
            rc = launch_adjoint(a, R, reinterpret_cast<float*>(ws + l.off_tmp), P, st);
            if (rc) return rc;
            cur = a.out;
        }
    }
    return PYSIFT_OK;
}

static int warp_args(WarpF32Args& a, const float* img1, int32_t hs, int32_t ws, int32_t C, const float* img2,
                     int32_t h2, int32_t w2, int32_t cw, int32_t ch, const double* hinv, double ox, double oy,
                     int32_t iox, int32_t ioy) {
    PYSIFT_CHECK_ARG(img1 && img2 && hinv && hs > 1 && ws > 1 && h2 > 0 && w2 > 0 && cw > 0 && ch > 0 && C >= 1 &&
                         C <= 4,
                     "bad arguments");
    a.img1 = img1;
    a.hs = hs;
    a.ws = ws;
    a.C = C;
    a.img2 = img2;
    a.h2 = h2;
    a.w2 = w2;
    a.cw = cw;
    a.ch = ch;
    for (int i = 0; i < 9; ++i) a.hinv[i] = hinv[i];
    a.ox = ox;
    a.oy = oy;
    a.iox = iox;
    a.ioy = ioy;
    return PYSIFT_OK;
}

int pysift_warp_f32_forward(const float* img1, int32_t hs, int32_t ws, int32_t C, const float* img2, int32_t h2,
                            int32_t w2, int32_t cw, int32_t ch, const double* hinv_host, double ox, double oy,
                            int32_t iox, int32_t ioy, float* out, pysift_stream_t stream) {
    WarpF32Args a = {};
    int rc = warp_args(a, img1, hs, ws, C, img2, h2, w2, cw, ch, hinv_host, ox, oy, iox, ioy);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(out != nullptr, "out is NULL");
    a.out = out;
    k_warp_f32_fwd<<<dim3(ceil_div(cw, 256), ch), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a);
    PYSIFT_LAUNCH_CHECK("k_warp_f32_fwd");
    return PYSIFT_OK;
}

int pysift_warp_f32_backward(const float* img1, int32_t hs, int32_t ws, int32_t C, const float* img2, int32_t h2,
                             int32_t w2, int32_t cw, int32_t ch, const double* hinv_host, double ox, double oy,
                             int32_t iox, int32_t ioy, const float* gout, float* gimg1, float* gimg2, double* ghinv,
                             pysift_stream_t stream) {
    WarpF32Args a = {};
    int rc = warp_args(a, img1, hs, ws, C, img2, h2, w2, cw, ch, hinv_host, ox, oy, iox, ioy);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(gout && gimg1 && gimg2 && ghinv, "NULL gradient buffer");
    a.gout = gout;
    a.gimg1 = gimg1;
    a.gimg2 = gimg2;
    a.ghinv = ghinv;
    // about two waves of eight blocks an SM
    const int gx = ceil_div(cw, WB_T);
    const dim3 grid(gx, std::max(1, std::min(ch, ceil_div(148 * 16, gx))));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (C) {
        case 1: k_warp_f32_bwd<1><<<grid, WB_T, 0, st>>>(a); break;
        case 2: k_warp_f32_bwd<2><<<grid, WB_T, 0, st>>>(a); break;
        case 3: k_warp_f32_bwd<3><<<grid, WB_T, 0, st>>>(a); break;
        default: k_warp_f32_bwd<4><<<grid, WB_T, 0, st>>>(a); break;
    }
    PYSIFT_LAUNCH_CHECK("k_warp_f32_bwd");
    return PYSIFT_OK;
}

int pysift_homography_adjoint(const double* hinv_host, const double* ghinv, double* gh8, pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(hinv_host && ghinv && gh8, "NULL pointer argument");
    Mat3 m;
    for (int i = 0; i < 9; ++i) m.m[i] = hinv_host[i];
    k_homography_adjoint<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(m, ghinv, gh8);
    PYSIFT_LAUNCH_CHECK("k_homography_adjoint");
    return PYSIFT_OK;
}

}  // extern "C"
