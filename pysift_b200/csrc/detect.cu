// detect.cu -- SIFT detection + description on one device-resident image.
//
// Pipeline (all launches on the caller's stream, no host synchronisation,
// capturable into a CUDA graph):
//   k_histogram          256-bin histogram + entropy threshold (pysift/core.py:1129-1148)
//   k_prefilter_cols, k_prefilter_rows, k_zoom_interp
//                        2x cubic B-spline upsample (pysift/core.py:1270-1275)
//   k_u8_to_f32          base image when not upsampled (pysift/core.py:1248-1261)
//   k_blur<R>            fused H+V separable blur per level (pysift/core.py:475-608,
//                        1288-1343); the first blur of octave o>0 reads the previous
//                        octave's level S with stride 2 and also stores level 0
//   k_extrema_mask       26-neighbour test on DoG computed on the fly from the Gaussian
//                        levels (pysift/core.py:176-217); one bit per voxel + per-row
//                        integer counts
//   k_rowscan, k_scatter deterministic compaction in (s, r, c) order, cap per octave
//   k_refine             Taylor refinement + contrast + edge (pysift/core.py:343-463)
//   k_refine_compact     valid keypoints in candidate order; decides on the starvation
//                        retry at half threshold (pysift/core.py:2066-2071)
//   k_cap                top-cap by response, stable (pysift/core.py:2078-2080)
//   k_orientation        36-bin histogram, peaks (pysift/core.py:228-333)
//   k_expand             orientation expansion + (x, y) sort keys (pysift/core.py:1592-1598)
//   k_br_scan/scatter/rank  rank of each key = output row (pysift/core.py:2128-2134),
//                        and the output-limit order, exactly, through buckets
//   k_descriptor         4x4x8 descriptor (+DSP) + L2/clip/L2 + RootSIFT, written at its
//                        output row (pysift/core.py:693-997, 1870-1873)
#include <algorithm>
#include <cstdarg>
#include <cstring>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "sift_math.cuh"

namespace pysift {

static thread_local std::string g_last_error;
static std::atomic<long long> g_launches{0};

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

// ---------------------------------------------------------------------------
// Device control block (one per run, inside the workspace).
// ---------------------------------------------------------------------------
struct Ctrl {
    double ct;
    float thr[2];
    unsigned int hist[256];
    unsigned int blocks_done;
    int found[PYSIFT_MAX_OCTAVES];
    int ncand[PYSIFT_MAX_OCTAVES];
    int nref[PYSIFT_MAX_OCTAVES];
    int compact_done;  // octaves of the first pass compacted
    int retried;
    int n_total_ref;
    int n_kept;
    int capped;
    int n_oriented;
    int overflow_octs;
    int desc_next;  // next oriented entry a descriptor block takes
    int ori_next;   // next kept keypoint an orientation block takes
};

// buckets of the exact rank kernels (k_br_*)
constexpr int BR_NB = 4096;

struct OctView {
    const float* lev[PYSIFT_MAX_LEVELS];
    int H, W, pitch;
};

// ---------------------------------------------------------------------------
// Workspace layout.
// ---------------------------------------------------------------------------
struct Layout {
    int n_oct, L, S;
    bool doubled;
    int H0, W0, pitch0;  // octave-0 / base image
    int H[PYSIFT_MAX_OCTAVES], W[PYSIFT_MAX_OCTAVES], pitch[PYSIFT_MAX_OCTAVES], wpr[PYSIFT_MAX_OCTAVES];
    size_t off_pyr[PYSIFT_MAX_OCTAVES], off_pyr_r[PYSIFT_MAX_OCTAVES];
    size_t off_mask[PYSIFT_MAX_OCTAVES], off_rowcnt[PYSIFT_MAX_OCTAVES], off_rowoff[PYSIFT_MAX_OCTAVES];
    size_t off_ctrl, off_coef, off_base;
    size_t off_cand, off_rv_valid, off_rv_ri, off_rv_ci, off_rv_si, off_rv_resp;
    size_t off_rf_ri, off_rf_ci, off_rf_si, off_rf_resp;
    size_t off_kp_o, off_kp_si, off_kp_ri, off_kp_ci, off_kp_resp, off_kp_tb;
    size_t off_ang, off_angcnt, off_ent_kp, off_ent_slot, off_keys, off_rank, off_row_resp, off_lrank;
    size_t off_bkt, off_members;  // bucket ranks: [2 orders][cnt | off | cursor][BR_NB], [2][4 kc] members
    size_t off_xblk;              // k_expand block counts
    size_t off_split;             // k_descriptor: totals and counts of the entries cut into parts
    size_t zero_bytes;  // row counts and masks of a pass; the retry's follow the first pass's
    size_t off_rowcnt_base;
    size_t total;
};

static int validate_cfg(const pysift_detect_config* c) {
    PYSIFT_CHECK_ARG(c != nullptr, "config is NULL");
    PYSIFT_CHECK_ARG(c->n_octaves >= 1 && c->n_octaves <= PYSIFT_MAX_OCTAVES, "n_octaves %d outside 1..%d",
                     c->n_octaves, PYSIFT_MAX_OCTAVES);
    PYSIFT_CHECK_ARG(c->n_scales >= 1 && c->n_scales + 3 <= PYSIFT_MAX_LEVELS, "n_scales %d outside 1..%d",
                     c->n_scales, PYSIFT_MAX_LEVELS - 3);
    PYSIFT_CHECK_ARG(c->max_cands_per_octave >= 1 && c->max_cands_per_octave <= (1 << 22),
                     "max_cands_per_octave %d out of range", c->max_cands_per_octave);
    PYSIFT_CHECK_ARG(c->keypoint_cap >= 1 && c->keypoint_cap <= (1 << 20), "keypoint_cap %d out of range",
                     c->keypoint_cap);
    PYSIFT_CHECK_ARG(c->border >= 1 && c->border < 64, "border %d out of range", c->border);
    PYSIFT_CHECK_ARG(c->output_limit >= 0, "output_limit %d is negative", c->output_limit);
    PYSIFT_CHECK_ARG(!c->dsp || (c->n_dsp >= 1 && c->n_dsp <= 8), "n_dsp %d out of range", c->n_dsp);
    for (int i = 0; i < 2 + c->n_scales + 2; ++i)
        PYSIFT_CHECK_ARG(c->blur_radius[i] >= 0 && c->blur_radius[i] <= PYSIFT_MAX_RADIUS,
                         "blur radius %d outside 0..%d", c->blur_radius[i], PYSIFT_MAX_RADIUS);
    for (int s = 1; s <= c->n_scales; ++s) {
        PYSIFT_CHECK_ARG(c->desc_ph[s] >= 1.0f && c->desc_ph[s] <= 200.0f, "desc_ph[%d] out of range", s);
        PYSIFT_CHECK_ARG(c->ori_sigma[s] > 0.0f && c->ori_sigma[s] < 64.0f, "ori_sigma[%d] out of range", s);
    }
    return PYSIFT_OK;
}

static size_t split_bytes(size_t kcap);

static Layout make_layout(const pysift_detect_config* c, int H, int W) {
    Layout l;
    memset(&l, 0, sizeof(l));
    l.n_oct = c->n_octaves;
    l.S = c->n_scales;
    l.L = c->n_scales + 3;
    l.doubled = c->double_image && ((int64_t)H * W < c->double_px_cap);
    l.H0 = l.doubled ? 2 * H : H;
    l.W0 = l.doubled ? 2 * W : W;
    int h = l.H0, w = l.W0;
    for (int o = 0; o < l.n_oct; ++o) {
        l.H[o] = h;
        l.W[o] = w;
        l.pitch[o] = (int)align_up((size_t)w, 32);
        l.wpr[o] = ceil_div(w, 32);
        h = (h + 1) / 2;
        w = (w + 1) / 2;
    }
    l.pitch0 = l.pitch[0];
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t r = off;
        off = align_up(off + bytes, 256);
        return r;
    };
    const size_t cap = (size_t)c->max_cands_per_octave;
    const size_t kc = (size_t)c->keypoint_cap;
    l.off_ctrl = take(sizeof(Ctrl));
    // row counts and masks of all octaves, and a second set for the retry, are
    // contiguous so one memset clears them
    l.off_rowcnt_base = off;
    size_t rc = 0;
    for (int o = 0; o < l.n_oct; ++o) rc += (size_t)l.S * l.H[o];
    size_t start = take(rc * sizeof(int));
    size_t acc = start;
    for (int o = 0; o < l.n_oct; ++o) {
        l.off_rowcnt[o] = acc;
        acc += (size_t)l.S * l.H[o] * sizeof(int);
    }
    for (int o = 0; o < l.n_oct; ++o) l.off_mask[o] = take((size_t)l.S * l.H[o] * l.wpr[o] * sizeof(uint32_t));
    l.zero_bytes = off - l.off_rowcnt_base;
    take(l.zero_bytes);
    for (int o = 0; o < l.n_oct; ++o) l.off_rowoff[o] = take((size_t)l.S * l.H[o] * sizeof(int));
    l.off_cand = take(cap * l.n_oct * sizeof(int4));
    l.off_rv_valid = take(cap * l.n_oct * sizeof(int));
    l.off_rv_ri = take(cap * l.n_oct * sizeof(float));
    l.off_rv_ci = take(cap * l.n_oct * sizeof(float));
    l.off_rv_si = take(cap * l.n_oct * sizeof(int));
    l.off_rv_resp = take(cap * l.n_oct * sizeof(float));
    l.off_rf_ri = take(cap * l.n_oct * sizeof(float));
    l.off_rf_ci = take(cap * l.n_oct * sizeof(float));
    l.off_rf_si = take(cap * l.n_oct * sizeof(int));
    l.off_rf_resp = take(cap * l.n_oct * sizeof(float));
    l.off_kp_o = take(kc * sizeof(int));
    l.off_kp_si = take(kc * sizeof(int));
    l.off_kp_ri = take(kc * sizeof(float));
    l.off_kp_ci = take(kc * sizeof(float));
    l.off_kp_resp = take(kc * sizeof(float));
    l.off_kp_tb = take(kc * sizeof(uint32_t));
    l.off_ang = take(kc * 4 * sizeof(float));
    l.off_angcnt = take(kc * sizeof(int));
    l.off_ent_kp = take(kc * 4 * sizeof(int));
    l.off_ent_slot = take(kc * 4 * sizeof(int));
    l.off_keys = take(kc * 4 * sizeof(uint4));
    l.off_rank = take(kc * 4 * sizeof(int));
    l.off_row_resp = take(kc * 4 * sizeof(float));
    l.off_lrank = take(kc * 4 * sizeof(int));
    l.off_bkt = take(2 * 3 * BR_NB * sizeof(int));
    l.off_members = take(2 * kc * 4 * sizeof(int));
    l.off_xblk = take(((size_t)kc / 2048 + 2) * sizeof(int));
    l.off_split = take(split_bytes(kc));
    if (l.doubled) l.off_coef = take((size_t)H * W * sizeof(double));
    l.off_base = take((size_t)l.H0 * l.pitch0 * sizeof(float));
    for (int o = 0; o < l.n_oct; ++o) l.off_pyr[o] = take((size_t)l.L * l.H[o] * l.pitch[o] * sizeof(float));
    for (int o = 0; o < l.n_oct; ++o) {
        if (c->fp16_pyramid && o >= 2)
            l.off_pyr_r[o] = take((size_t)l.L * l.H[o] * l.pitch[o] * sizeof(float));
        else
            l.off_pyr_r[o] = l.off_pyr[o];
    }
    l.total = off;
    return l;
}

// ---------------------------------------------------------------------------
// A1: histogram + entropy threshold.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_histogram(const uint8_t* __restrict__ img, int H, int W, long long pitch,
                                                   Ctrl* ctrl, double base, int S) {
    __shared__ unsigned int sh[8][256];
    __shared__ double terms[256];
    __shared__ int is_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 8 * 256; i += 256) (&sh[0][0])[i] = 0u;
    __syncthreads();
    // a warp per row; 16-byte loads when every row starts on a 16-byte
    // boundary, else byte loads in batches of 8, all in flight before the
    // shared-memory counts
    const bool vec = ((reinterpret_cast<uintptr_t>(img) | (uintptr_t)pitch) & 15) == 0;
    const int nw = W >> 4;
    for (int r = blockIdx.x * 8 + warp; r < H; r += gridDim.x * 8) {
        const uint8_t* row = img + (long long)r * pitch;
        int c0 = 0;
        if (vec) {
            for (int q0 = 0; q0 < nw; q0 += 64) {
                uint4 u[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int q = q0 + lane + 32 * k;
                    u[k] = q < nw ? reinterpret_cast<const uint4*>(row)[q] : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (q0 + lane + 32 * k >= nw) continue;
                    const uint32_t w4[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int sh8 = 0; sh8 < 32; sh8 += 8) atomicAdd(&sh[warp][(w4[e] >> sh8) & 255u], 1u);
                }
            }
            c0 = nw << 4;
        }
        for (int cb = c0; cb < W; cb += 32 * 8) {
            uint8_t u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = cb + lane + 32 * k;
                u[k] = c < W ? row[c] : 0;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (cb + lane + 32 * k < W) atomicAdd(&sh[warp][u[k]], 1u);
        }
    }
    __syncthreads();
    unsigned int mine = 0;
    for (int w = 0; w < 8; ++w) mine += sh[w][tid];
    if (mine) atomicAdd(&ctrl->hist[tid], mine);
    __threadfence();
    __syncthreads();
    if (tid == 0) is_last = (atomicAdd(&ctrl->blocks_done, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    const double n = (double)H * (double)W;
    unsigned int h = atomicAdd(&ctrl->hist[tid], 0u);
    double t = 0.0;
    if (h) {
        double p = (double)h / n;
        t = p * sm::log2d_(p);
    }
    terms[tid] = t;
    sh[0][tid] = h;
    __syncthreads();
    if (tid == 0) {
        // ascending bins, one double sum; an empty bin holds +0.0, which
        // leaves a sum that started at +0.0 unchanged, so every term is added
        // and the loads run ahead of the chain
        double ent = 0.0;
#pragma unroll 32
        for (int b = 0; b < 256; ++b) ent = ent + terms[b];
        ent = -ent;
        double scale = 0.8 + ent / 40.0;
        if (scale > 1.0) scale = 1.0;
        double ct = base * scale;
        ctrl->ct = ct;
        ctrl->thr[0] = (float)(ct / (double)S);
        ctrl->thr[1] = (float)((ct * 0.5) / (double)S);
    }
}

// ---------------------------------------------------------------------------
// A2/A3: base image.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float u8_to_unit(uint8_t u, int fp16) {
    float f = (float)u / 255.0f;
    return fp16 ? round_half(f) : f;
}

__global__ void k_u8_to_f32(const uint8_t* __restrict__ img, int H, int W, long long pitch, int fp16,
                            float* __restrict__ out, int out_pitch) {
    chain_begin();
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int r = blockIdx.y;
    if (c < W) out[(long long)r * out_pitch + c] = u8_to_unit(img[(long long)r * pitch + c], fp16);
}

// B-spline direct transform (scipy.ndimage.spline_filter, order 3, mirror
// boundary) as a symmetric FIR: on the mirror-extended line the recursive
// prefilter's impulse response is h[k] = (-6 z / (1 - z^2)) z^|k| with
// z = sqrt(3) - 2, truncated at |k| <= SPL_K (|z|^31 < 2e-18).  Taps run
// k = -SPL_K..SPL_K with one fma each.  Columns (axis 0) are filtered first,
// then rows, as scipy does.
constexpr int SPL_K = 30;
constexpr int SPL_TAPS = 2 * SPL_K + 1;

// Taps computed once on the host with the same operation sequence as the
// oracle (IEEE double, no contraction) and passed by value, so that fully
// unrolled loops read them as constant-bank operands.
struct SplTaps {
    double h[SPL_TAPS];
};

static const SplTaps& spline_taps() {
    static const SplTaps taps = [] {
        SplTaps t;
        const double z = sqrt(3.0) - 2.0;
        const double c0 = -6.0 * z / (1.0 - z * z);
        for (int k = -SPL_K; k <= SPL_K; ++k) {
            const int a = k < 0 ? -k : k;
            double zk = 1.0;
            for (int i = 0; i < a; ++i) zk = zk * z;
            t.h[k + SPL_K] = c0 * zk;
        }
        return t;
    }();
    return taps;
}

__device__ __forceinline__ long long mirror_index(long long idx, long long len) {
    if (len <= 1) return 0;
    long long s2 = 2 * len - 2;
    if (idx < 0) {
        idx = s2 * (long long)(-idx / s2) + idx;
        idx = idx <= 1 - len ? idx + s2 : -idx;
    } else if (idx >= len) {
        idx -= s2 * (long long)(idx / s2);
        if (idx >= len) idx = s2 - idx;
    }
    return idx;
}

constexpr int PC_TW = 32, PC_RB = 8, PC_TH = 8 * PC_RB;

// Column FIR straight from the uint8 image: coef[r][x] = sum_k h[k] u[mirror(r+k)][x].
// Each thread produces PC_RB consecutive rows of one column, streaming the
// input window through registers (taps in ascending k for every output).
// Bound by its float64 multiply-adds (61 a coefficient, 39 us for 12 Mpixel);
// the window's bytes go through a table of the 256 widened values and skip
// the mirroring away from the edges: 86 -> 72 us there.
__global__ void __launch_bounds__(256) k_prefilter_cols(const uint8_t* __restrict__ img, int H, int W,
                                                        long long pitch, int fp16, double* __restrict__ coef,
                                                        const SplTaps taps) {
    chain_begin();
    __shared__ double tile[(PC_TH + 2 * SPL_K) * PC_TW];
    // u / 255 as the base image holds it, widened: one conversion a value
    __shared__ double unit[256];
    const int x0 = blockIdx.x * PC_TW, r0 = blockIdx.y * PC_TH;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int x = x0 + tx;
    {
        // every load of the window issued before the first look-up
        constexpr int NL = (PC_TH + 2 * SPL_K + 7) / 8;
        uint8_t u[NL];
        const bool inside = r0 >= SPL_K && r0 + PC_TH + SPL_K <= H;
        const uint8_t* src = img + (long long)(r0 - SPL_K + ty) * pitch + x;
#pragma unroll
        for (int q = 0; q < NL; ++q) {
            const int rr = ty + 8 * q;
            u[q] = 0;
            if (x < W && rr < PC_TH + 2 * SPL_K)
                u[q] = inside ? src[(long long)(8 * q) * pitch] : img[mirror_index(r0 - SPL_K + rr, H) * pitch + x];
        }
        unit[threadIdx.x] = (double)u8_to_unit((uint8_t)threadIdx.x, fp16);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NL; ++q) {
            const int rr = ty + 8 * q;
            if (rr < PC_TH + 2 * SPL_K) tile[rr * PC_TW + tx] = unit[u[q]];
        }
    }
    __syncthreads();
    if (x >= W) return;
    const int y0 = ty * PC_RB;
    double acc[PC_RB];
#pragma unroll
    for (int j = 0; j < PC_RB; ++j) acc[j] = 0.0;
#pragma unroll
    for (int m = 0; m < PC_RB + 2 * SPL_K; ++m) {
        const double t = tile[(y0 + m) * PC_TW + tx];
#pragma unroll
        for (int j = 0; j < PC_RB; ++j) {
            const int k = m - j;
            if (k >= 0 && k < SPL_TAPS) acc[j] = fma(taps.h[k], t, acc[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < PC_RB; ++j) {
        const int r = r0 + y0 + j;
        if (r < H) coef[(long long)r * W + x] = acc[j];
    }
}

// Output-coordinate setup for one axis of scipy's zoom (grid_mode=False,
// mode='constant'): input coordinate k * zoom, zoom = (in-1)/(out-1), the first of the four
// support positions (before mirroring) and cubic B-spline weights; false
// outside [0, in-1] (cval 0).
__device__ __forceinline__ bool zoom_axis(int k, int in_len, double zoom, int& start, double w[4]) {
    double cc = (double)k * zoom;
    if (cc < 0.0 || cc > (double)(in_len - 1)) return false;
    double fl = floor(cc);
    start = (int)fl - 1;
    double y = cc - fl;
    double z = 1.0 - y;
    w[0] = z * z * z / 6.0;
    w[1] = (y * y * (y - 2.0) * 3.0 + 4.0) / 6.0;
    double y1 = 1.0 - y;
    w[2] = (y1 * y1 * (y1 - 2.0) * 3.0 + 4.0) / 6.0;
    w[3] = 1.0 - w[0] - w[1] - w[2];
    return true;
}

// Row FIR in place: coef[r][x] <- sum_k h[k] coef[r][mirror(x-SPL_K+k)], one
// block per row, the row processed in chunks of PR_CW outputs left to right.
// A chunk's window is read before any of its outputs is written; its left
// halo, which the previous chunk has overwritten, comes from a carry of the
// previous chunk's last SPL_K inputs.  Mirrored positions past the right
// end fall at or after the chunk start minus SPL_K once the row spans more
// than one chunk, so the carry and the unwritten part of the row hold every
// input.  The window sits in shared memory with one padding double per 8 so
// that lanes reading 8-output strips hit distinct banks.
constexpr int PR_NT = 256, PR_CW = 2048;
constexpr int PR_EXT = PR_CW + 2 * SPL_K;
__device__ __forceinline__ int pr_phys(int e) { return e + (e >> 3); }

__global__ void __launch_bounds__(PR_NT) k_prefilter_rows(double* __restrict__ coef, int W, const SplTaps taps) {
    chain_begin();
    // a strip that ends past the chunk reads up to 7 positions beyond the
    // window (values that feed no stored output), so the array covers them
    __shared__ double ext[PR_EXT + 7 + (PR_EXT + 7) / 8 + 1];
    __shared__ double carry[SPL_K];
    double* row = coef + (long long)blockIdx.x * W;
    for (int x0 = 0; x0 < W; x0 += PR_CW) {
        const int len = min(PR_CW, W - x0);
        for (int e = threadIdx.x; e < len + 2 * SPL_K; e += PR_NT) {
            const int m = (int)mirror_index((long long)x0 - SPL_K + e, W);
            if (m >= x0) {
                const unsigned d = (unsigned)__cvta_generic_to_shared(&ext[pr_phys(e)]);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(row + m) : "memory");
            } else {
                ext[pr_phys(e)] = carry[m - (x0 - SPL_K)];
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (x0 + PR_CW < W)
            for (int i = threadIdx.x; i < SPL_K; i += PR_NT) carry[i] = ext[pr_phys(PR_CW + i)];
        for (int b = threadIdx.x * 8; b < len; b += PR_NT * 8) {
            double acc[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = 0.0;
#pragma unroll
            for (int m = 0; m < 8 + 2 * SPL_K; ++m) {
                const double t = ext[pr_phys(b + m)];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = m - j;
                    if (k >= 0 && k < SPL_TAPS) acc[j] = fma(taps.h[k], t, acc[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (b + j < len) row[x0 + b + j] = acc[j];
        }
        __syncthreads();
    }
}

// 4x4 cubic interpolation of the prefiltered coefficients on the 2x output
// grid, t = sum_a sum_b (c[a][b] * wy_a) * wx_b in scipy's order, rounded to
// float32.  On the 2x grid the output columns 2k-1 and 2k interpolate the
// same 4 input columns (their input coordinates share the floor k-1), and
// likewise the output rows 2j-1 and 2j, so the grid splits into 2x2 quads of
// common support (the coordinates of 2k-1 and 2k lie (n-k)/(2n-1) above k-1 and
// k/(2n-1) below k on n inputs, far more than their rounding, and the last one
// is n-1 exactly).  A lane owns a column pair and its warp walks down the row
// pairs of a tile: of the 16 coefficients 4 are new at each step (the window
// in shared memory holds mirrored rows and columns past the image's edges, so
// that every support is contiguous), the column weights stay in registers,
// and each c * wy_a serves both columns.  What is left is the 160 float64
// operations of a quad (108 us for the 48 Mpixel of a doubled 4000x3000 image
// at 64 a cycle and SM); with all 16 coefficients and both axes' weights
// fetched from shared memory per quad it was issue-bound: 283 -> 178 us there.
// Three blocks an SM (80 registers) hide the chains' latency best.
constexpr int ZI_T = 256, ZI_W = ZI_T / 32;
constexpr int ZI_MAX_PAIRS = 16;                       // row pairs of a warp, at most
constexpr int ZI_CC = 36;

__global__ void __launch_bounds__(ZI_T, 3) k_zoom_interp(const double* coef, int H, int W, double zy,
                                                      double zx, int fp16, int pairs, float* __restrict__ out, int out_pitch) {
    chain_begin();
    __shared__ __align__(16) double rw[2 * ZI_W * ZI_MAX_PAIRS][4];  // weights of output rows 2 j0 - 1 + i
    __shared__ int rstart[2 * ZI_W * ZI_MAX_PAIRS];                  // first window row of their support, -1: outside
    extern __shared__ double zi_win[];
    double (*const win)[ZI_CC] = reinterpret_cast<double (*)[ZI_CC]>(zi_win);  // ZI_W * pairs + 4 rows
    const int OH = 2 * H, OW = 2 * W;
    const int k0 = blockIdx.x * 32, j0 = blockIdx.y * ZI_W * pairs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int npairs = min(ZI_W * pairs, H + 1 - j0);  // row pairs j0 .. of this tile
    const int ylo = j0 - 2, xlo = k0 - 2;
    {
        const int xm = (int)mirror_index(xlo + lane, W), xn = (int)mirror_index(xlo + 32 + (lane & 3), W);
        for (int yy = warp; yy < npairs + 4; yy += ZI_W) {
            const int y = ylo + yy;
            const double* src = coef + (long long)(y >= 0 && y < H ? y : (int)mirror_index(y, H)) * W;
            const unsigned d = (unsigned)__cvta_generic_to_shared(&win[yy][lane]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src + xm) : "memory");
            if (lane < 4)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + 32 * 8), "l"(src + xn) : "memory");
        }
    }
    for (int i = tid; i < 2 * npairs; i += ZI_T) {
        const int r = 2 * j0 - 1 + i;
        double w[4];
        int start = 0;
        const bool v = r >= 0 && r < OH && zoom_axis(r, H, zy, start, w);
        rstart[i] = v ? start - ylo : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) rw[i][q] = v ? w[q] : 0.0;
    }
    // this lane's column pair 2 k - 1, 2 k
    const int xa = 2 * (k0 + lane) - 1, xb = xa + 1;
    double wxa[4] = {0.0, 0.0, 0.0, 0.0}, wxb[4] = {0.0, 0.0, 0.0, 0.0};
    int sa = 0, sb = 0;
    const bool cva = xa >= 0 && xa < OW && zoom_axis(xa, W, zx, sa, wxa);
    const bool cvb = xb < OW && zoom_axis(xb, W, zx, sb, wxb);
    const int col = cva ? sa - xlo : (cvb ? sb - xlo : 0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const bool pair_stores = (out_pitch & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    double c[4][4];  // rows of the support, rotating
    int have = -2;   // window row of the support's first row
    auto step = [&](int q, auto phase) {
        constexpr int ph = decltype(phase)::value;
        const int pair = warp * pairs + q;
        if (pair >= npairs) return;
        const int i = 2 * pair, ra = 2 * j0 - 1 + i, rb = ra + 1;
        const int ya = rstart[i], yb = rstart[i + 1], y = ya >= 0 ? ya : yb;
        float v[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
        if (y >= 0) {
            if (y == have + 1) {
#pragma unroll
                for (int b = 0; b < 4; ++b) c[(ph + 3) & 3][b] = win[y + 3][col + b];
            } else {
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) c[(ph + a) & 3][b] = win[y + a][col + b];
            }
            have = y;
            double wy[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double2 w2 = reinterpret_cast<const double2*>(rw[i + u])[h];
                    wy[u][2 * h] = w2.x;
                    wy[u][2 * h + 1] = w2.y;
                }
            double t[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const double w0 = wy[0][a], w1 = wy[1][a];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const double p0 = c[(ph + a) & 3][b] * w0, p1 = c[(ph + a) & 3][b] * w1;
                    t[0][0] += p0 * wxa[b];
                    t[0][1] += p0 * wxb[b];
                    t[1][0] += p1 * wxa[b];
                    t[1][1] += p1 * wxb[b];
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const bool rv = (u ? yb : ya) >= 0;
                v[u][0] = rv && cva ? (float)t[u][0] : 0.0f;
                v[u][1] = rv && cvb ? (float)t[u][1] : 0.0f;
                if (fp16) {
                    v[u][0] = round_half(v[u][0]);
                    v[u][1] = round_half(v[u][1]);
                }
            }
        } else {
            have = -2;
        }
        // columns 2 k (this lane's) and 2 k + 1 (the next lane's) as one word
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float right = __shfl_down_sync(FULL_MASK, v[u][0], 1);
            const int r = u ? rb : ra;
            if (r < 0 || r >= OH) continue;
            float* row = out + (long long)r * out_pitch;
            if (lane == 0 && xa >= 0 && xa < OW) row[xa] = v[u][0];
            if (xb < OW) {
                if (lane < 31 && pair_stores) *reinterpret_cast<float2*>(row + xb) = make_float2(v[u][1], right);
                else {
                    row[xb] = v[u][1];
                    if (lane < 31) row[xb + 1] = right;
                }
            }
        }
    };
    for (int q = 0; q < pairs; q += 4) {
        step(q, std::integral_constant<int, 0>{});
        if (q + 1 < pairs) step(q + 1, std::integral_constant<int, 1>{});
        if (q + 2 < pairs) step(q + 2, std::integral_constant<int, 2>{});
        if (q + 3 < pairs) step(q + 3, std::integral_constant<int, 3>{});
    }
}

static int num_sms();

static int launch_zoom2x(const uint8_t* gray, int H, int W, long long pitch, int fp16, double* coef, float* out,
                         int out_pitch, cudaStream_t st) {
    const SplTaps& taps = spline_taps();
    k_prefilter_cols<<<dim3(ceil_div(W, PC_TW), ceil_div(H, PC_TH)), 256, 0, st>>>(gray, H, W, pitch, fp16, coef,
                                                                                  taps);
    PYSIFT_LAUNCH_CHECK("k_prefilter_cols");
    launch_chained(k_prefilter_rows, dim3(H), PR_NT, 0, st, coef, W, taps);
    PYSIFT_LAUNCH_CHECK("k_prefilter_rows");
    // row pairs of a warp: long walks while they fill the SMs, shorter ones for
    // small images
    int pairs = ZI_MAX_PAIRS;
    auto blocks = [&] { return (long long)ceil_div(W + 1, 32) * ceil_div(H + 1, ZI_W * pairs); };
    while (pairs > 1 && blocks() < 3LL * num_sms()) pairs /= 2;
    const double zy = (double)(H - 1) / (double)(2 * H - 1), zx = (double)(W - 1) / (double)(2 * W - 1);
    const size_t window = (size_t)(ZI_W * pairs + 4) * ZI_CC * sizeof(double);
    launch_chained(k_zoom_interp, dim3(ceil_div(W + 1, 32), ceil_div(H + 1, ZI_W * pairs)), ZI_T, window, st,
                   (const double*)coef, H, W, zy, zx, fp16, pairs, out, out_pitch);
    PYSIFT_LAUNCH_CHECK("k_zoom_interp");
    return PYSIFT_OK;
}

// ---------------------------------------------------------------------------
// A4/A5: fused separable blur.
// ---------------------------------------------------------------------------
constexpr int BLUR_PAIR_MAX_R = 16;  // radii with a register-blocked kernel

struct BlurArgs {
    const float* in;
    long long in_pitch;
    int step;  // 1, or 2 when reading level S of the previous octave
    float* out;
    float* out_r;  // binary16-rounded copy (fp16 mode), else null
    float* copy0;  // stores the (subsampled) input tile interior, else null
    float* copy0_r;
    int out_pitch;
    int H, W;
    float w[PYSIFT_MAX_TAPS];
    unsigned long long w2[2 * BLUR_PAIR_MAX_R + 1];  // (w[k], w[k]) packed, radii up to BLUR_PAIR_MAX_R
};

constexpr int BLUR_TW = 64, BLUR_TH = 32, BLUR_NT = 256;

// Loads input rows [r0-R, r0+TH+R) and columns [c0-RA, c0+TW+RA) (RA >= R,
// a multiple of 4) into tile[ROWS][TWP] with reflection.  Tiles whose
// window lies inside the image, read with stride 1 from a 16-byte aligned
// base and pitch, use float4 loads.
__device__ __forceinline__ void blur_load_tile(const BlurArgs& a, float* tile, int R, int RA, int TWP, int ROWS,
                                               int r0, int c0) {
    const bool interior = a.step == 1 && r0 - R >= 0 && r0 + BLUR_TH + R <= a.H && c0 - RA >= 0 &&
                          c0 + BLUR_TW + RA <= a.W && ((a.in_pitch & 3) == 0) &&
                          ((reinterpret_cast<uintptr_t>(a.in) & 15) == 0);
    if (interior) {
        const int q4 = TWP / 4;
        for (int i = threadIdx.x; i < ROWS * q4; i += BLUR_NT) {
            const int rr = i / q4, q = i - rr * q4;
            const float4 v = *reinterpret_cast<const float4*>(a.in + (long long)(r0 - R + rr) * a.in_pitch + c0 - RA +
                                                              4 * q);
            *reinterpret_cast<float4*>(tile + rr * TWP + 4 * q) = v;
        }
        return;
    }
    for (int i = threadIdx.x; i < ROWS * TWP; i += BLUR_NT) {
        int rr = i / TWP, cc = i - rr * TWP;
        int gr = reflect_idx(r0 - R + rr, a.H), gc = reflect_idx(c0 - RA + cc, a.W);
        float v = a.in[(long long)gr * a.step * a.in_pitch + (long long)gc * a.step];
        tile[i] = v;
        if (a.copy0 && rr >= R && rr < R + BLUR_TH && cc >= RA && cc < RA + BLUR_TW) {
            int orow = r0 + rr - R, ocol = c0 + cc - RA;
            if (orow < a.H && ocol < a.W) {
                a.copy0[(long long)orow * a.out_pitch + ocol] = v;
                if (a.copy0_r) a.copy0_r[(long long)orow * a.out_pitch + ocol] = round_half(v);
            }
        }
    }
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// Packed single-precision pairs: fma.rn.f32x2 is an IEEE fused multiply-add
// with round-to-nearest on each half, the same result as fmaf per element.
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b,
                                                    unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float((unsigned)(v & 0xffffffffull)); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }

// Tile geometry of k_blur<R, TH>: input rows [r0-R, r0+TH+R) and columns
// [c0-R, c0+TW+R) at a row stride TS = 2 (mod 4) (8-byte aligned rows; lanes
// that own consecutive rows read 8-byte pairs from distinct banks), then the
// row-filtered rows at the stride HS = 66, also 2 (mod 4).
template <int R, int TH>
struct BlurTile {
    static constexpr int ROWS = TH + 2 * R;
    static constexpr int TWR = BLUR_TW + 2 * R;
    static constexpr int TS = (TWR % 4 == 2) ? TWR : TWR + 2;
    static constexpr int HS = BLUR_TW + 2;
    static constexpr size_t bytes = (size_t)(ROWS * TS + ROWS * HS) * sizeof(float);
};

// Row filter of 8 outputs src[0..7] (+R halo each side) of one tile row into
// dst[0..7]: 4 output pairs, one packed fma per pair and tap, taps in
// ascending order.  Pairs at even offsets are loaded as 8-byte words; the
// pairs at odd offsets are formed from their neighbours.
template <int R, typename WF>
__device__ __forceinline__ void blur_row_strip(const float* src, float* dst, const WF& w2) {
    constexpr int NP = 4 + R;
    unsigned long long E[NP], O[NP - 1];
#pragma unroll
    for (int m = 0; m < NP; ++m) E[m] = reinterpret_cast<const unsigned long long*>(src)[m];
#pragma unroll
    for (int m = 0; m < NP - 1; ++m) O[m] = pack2(hi2(E[m]), lo2(E[m + 1]));
    unsigned long long A[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
    for (int k = 0; k <= 2 * R; ++k) {
        const unsigned long long wk = w2(k);
#pragma unroll
        for (int p = 0; p < 4; ++p) A[p] = ffma2((k & 1) ? O[p + (k >> 1)] : E[p + (k >> 1)], wk, A[p]);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) reinterpret_cast<unsigned long long*>(dst)[p] = A[p];
}

// The source, destination and geometry of one blurred level, as a tile of
// it sees them (the fields of BlurArgs without the weights).
struct TileIO {
    const float* in;
    long long in_pitch;
    int step;
    float* out;
    float* out_r;
    float* copy0;
    float* copy0_r;
    int out_pitch;
    int H, W;
};

// Fused H+V separable blur of one 64 x TH output tile (tile column bx, tile
// row by).  The tile and its reflected halo are filled with cp.async (every
// load in flight at once; reflection computed once per row and once per
// column).  Row pass: a lane per tile row (the rows past the first 32 packed
// densely onto the first warps), 8 outputs per lane.  Column pass: each
// thread filters a pair of adjacent columns over TH / 8 rows.  Both passes
// use packed fma pairs; each output is the same fmaf chain over the taps in
// ascending order.  w2(k) is tap k's weight packed twice.  The caller
// synchronises the block before smem is reused.
template <int R, int TH, typename WF>
__device__ __forceinline__ void blur_tile(const TileIO& a, int bx, int by, float* smem, const WF& w2) {
    using T = BlurTile<R, TH>;
    constexpr int TW = BLUR_TW, ROWS = T::ROWS, TWR = T::TWR, TS = T::TS, HS = T::HS;
    constexpr int RP = TH / 8;  // column-pass rows per thread
    constexpr int CQ = (TWR + 31) / 32;
    static_assert(BLUR_NT / 32 == TW / 8, "one warp per 8-column strip in the row pass");
    static_assert(TH % 8 == 0 && BLUR_NT == (TW / 2) * 8, "one thread per column pair and TH / 8 rows in the column pass");
    float* tile = smem;
    float* hb = smem + ROWS * TS;
    const int c0 = bx * TW, r0 = by * TH;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        long long gcs[CQ];
#pragma unroll
        for (int q = 0; q < CQ; ++q) {
            const int cc = lane + 32 * q;
            gcs[q] = (long long)reflect_idx(c0 - R + (cc < TWR ? cc : 0), a.W) * a.step;
        }
        for (int rr = warp; rr < ROWS; rr += BLUR_NT / 32) {
            const float* rowp = a.in + (long long)reflect_idx(r0 - R + rr, a.H) * a.step * a.in_pitch;
#pragma unroll
            for (int q = 0; q < CQ; ++q) {
                const int cc = lane + 32 * q;
                if (cc < TWR) cp_async4(tile + rr * TS + cc, rowp + gcs[q]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    if (a.copy0) {
        for (int i = threadIdx.x; i < TH * TW; i += BLUR_NT) {
            const int y = i / TW, x = i - y * TW;
            const int orow = r0 + y, ocol = c0 + x;
            if (orow < a.H && ocol < a.W) {
                const float v = tile[(y + R) * TS + x + R];
                a.copy0[(long long)orow * a.out_pitch + ocol] = v;
                if (a.copy0_r) a.copy0_r[(long long)orow * a.out_pitch + ocol] = round_half(v);
            }
        }
    }
    {
        constexpr int NF = ROWS / 32, N2 = ROWS % 32;
#pragma unroll
        for (int round = 0; round < NF; ++round) {
            const int rr = round * 32 + lane;
            blur_row_strip<R>(tile + rr * TS + warp * 8, hb + rr * HS + warp * 8, w2);
        }
        if constexpr (N2 > 0) {
            if (threadIdx.x < N2 * 8) {
                const int rr = NF * 32 + threadIdx.x % N2, x0 = (threadIdx.x / N2) * 8;
                blur_row_strip<R>(tile + rr * TS + x0, hb + rr * HS + x0, w2);
            }
        }
    }
    __syncthreads();
    {
        const int cp = lane, y0 = warp * RP;
        constexpr int NV = RP + 2 * R;
        unsigned long long V[NV];
#pragma unroll
        for (int m = 0; m < NV; ++m) V[m] = reinterpret_cast<const unsigned long long*>(hb + (y0 + m) * HS)[cp];
        unsigned long long A[RP];
#pragma unroll
        for (int j = 0; j < RP; ++j) A[j] = 0ull;
#pragma unroll
        for (int k = 0; k <= 2 * R; ++k) {
            const unsigned long long wk = w2(k);
#pragma unroll
            for (int j = 0; j < RP; ++j) A[j] = ffma2(V[j + k], wk, A[j]);
        }
        const int gc = c0 + 2 * cp;
        const bool vec = gc + 1 < a.W && (a.out_pitch & 1) == 0;
#pragma unroll
        for (int j = 0; j < RP; ++j) {
            const int gr = r0 + y0 + j;
            if (gr >= a.H || gc >= a.W) continue;
            const float v0 = lo2(A[j]), v1 = hi2(A[j]);
            const long long off = (long long)gr * a.out_pitch + gc;
            if (vec) {
                *reinterpret_cast<float2*>(a.out + off) = make_float2(v0, v1);
                if (a.out_r) *reinterpret_cast<float2*>(a.out_r + off) = make_float2(round_half(v0), round_half(v1));
            } else {
                a.out[off] = v0;
                if (a.out_r) a.out_r[off] = round_half(v0);
                if (gc + 1 < a.W) {
                    a.out[off + 1] = v1;
                    if (a.out_r) a.out_r[off + 1] = round_half(v1);
                }
            }
        }
    }
}

// Interior tiles: the window [r0-R, r0+TH+R) x [c0-RA, c0+64+RA) (RA = R
// rounded up to 4) lies inside the level, the source is read with stride 1
// from 16-byte aligned rows and no copy of the input is stored.  Then the
// fill is one 16-byte cp.async per 4 floats, a warp per row, with no
// reflection; the row stride TSF = 4 (mod 8) lets the lane-per-row row pass
// read 16-byte words without bank conflicts; the stores need no bounds
// checks.  Same arithmetic as blur_tile, so the same results.
template <int R>
struct BlurFast {
    static constexpr int RA = (R + 3) / 4 * 4;
    static constexpr int D = RA - R;                          // first needed column of a strip, within its quad
    static constexpr int TWF = BLUR_TW + 2 * RA;              // floats per tile row
    static constexpr int TSF = (TWF % 8 == 4) ? TWF : TWF + 4;  // row stride = 4 (mod 8)
    static constexpr int NQ = (D + 8 + 2 * R + 3) / 4;        // 16-byte words a strip reads
    static_assert(TWF / 4 <= 32, "one warp fills a tile row");
};

template <int R, int TH>
__host__ __device__ constexpr size_t blur_fast_bytes() {
    return (size_t)((TH + 2 * R) * BlurFast<R>::TSF + (TH + 2 * R) * (BLUR_TW + 2)) * sizeof(float);
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ bool blur_tile_is_fast(const TileIO& a, int R, int RA, int TH, int bx, int by) {
    const int c0 = bx * BLUR_TW, r0 = by * TH;
    return a.step == 1 && !a.copy0 && r0 - R >= 0 && r0 + TH + R <= a.H && c0 - RA >= 0 &&
           c0 + BLUR_TW + RA <= a.W && (a.in_pitch & 3) == 0 && (reinterpret_cast<uintptr_t>(a.in) & 15) == 0 &&
           (a.out_pitch & 1) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 7) == 0 &&
           (reinterpret_cast<uintptr_t>(a.out_r) & 7) == 0;
}

// Row filter of one strip from 16-byte words q[0..NQ): output pair p, tap k
// reads floats D + 2p + k and D + 2p + k + 1 of the strip's words.
template <int R, typename WF>
__device__ __forceinline__ void blur_row_strip_q(const float* src, float* dst, const WF& w2) {
    using F = BlurFast<R>;
    constexpr int NF = 4 * F::NQ;
    float v[NF];
#pragma unroll
    for (int i = 0; i < F::NQ; ++i) {
        const float4 t = reinterpret_cast<const float4*>(src)[i];
        v[4 * i] = t.x;
        v[4 * i + 1] = t.y;
        v[4 * i + 2] = t.z;
        v[4 * i + 3] = t.w;
    }
    unsigned long long A[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
    for (int k = 0; k <= 2 * R; ++k) {
        const unsigned long long wk = w2(k);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int e = F::D + 2 * p + k;
            A[p] = ffma2(pack2(v[e], v[e + 1]), wk, A[p]);
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) reinterpret_cast<unsigned long long*>(dst)[p] = A[p];
}

template <int R, int TH, typename WF>
__device__ __forceinline__ void blur_tile_fast(const TileIO& a, int bx, int by, float* smem, const WF& w2) {
    using F = BlurFast<R>;
    constexpr int TW = BLUR_TW, ROWS = TH + 2 * R, TSF = F::TSF, HS = BLUR_TW + 2;
    constexpr int RP = TH / 8;
    float* tile = smem;
    float* hb = smem + ROWS * TSF;
    const int c0 = bx * TW, r0 = by * TH;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const bool act = lane < F::TWF / 4;
        const float* src = a.in + (long long)(r0 - R + warp) * a.in_pitch + (c0 - F::RA) + 4 * lane;
        float* dst = tile + warp * TSF + 4 * lane;
        const long long gstep = 8 * a.in_pitch;
        for (int rr = warp; rr < ROWS; rr += BLUR_NT / 32) {
            if (act) cp_async16(dst, src);
            src += gstep;
            dst += 8 * TSF;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    {
        constexpr int NR = ROWS / 32, N2 = ROWS % 32;
#pragma unroll
        for (int round = 0; round < NR; ++round) {
            const int rr = round * 32 + lane;
            blur_row_strip_q<R>(tile + rr * TSF + warp * 8, hb + rr * HS + warp * 8, w2);
        }
        if constexpr (N2 > 0) {
            if (threadIdx.x < N2 * 8) {
                const int rr = NR * 32 + threadIdx.x % N2, x0 = (threadIdx.x / N2) * 8;
                blur_row_strip_q<R>(tile + rr * TSF + x0, hb + rr * HS + x0, w2);
            }
        }
    }
    __syncthreads();
    {
        const int cp = lane, y0 = warp * RP;
        constexpr int NV = RP + 2 * R;
        unsigned long long V[NV];
#pragma unroll
        for (int m = 0; m < NV; ++m) V[m] = reinterpret_cast<const unsigned long long*>(hb + (y0 + m) * HS)[cp];
        unsigned long long A[RP];
#pragma unroll
        for (int j = 0; j < RP; ++j) A[j] = 0ull;
#pragma unroll
        for (int k = 0; k <= 2 * R; ++k) {
            const unsigned long long wk = w2(k);
#pragma unroll
            for (int j = 0; j < RP; ++j) A[j] = ffma2(V[j + k], wk, A[j]);
        }
        const long long off = (long long)(r0 + y0) * a.out_pitch + c0 + 2 * cp;
        unsigned long long* o = reinterpret_cast<unsigned long long*>(a.out + off);
        const int op2 = a.out_pitch >> 1;
#pragma unroll
        for (int j = 0; j < RP; ++j) o[j * op2] = A[j];
        if (a.out_r) {
            float2* orr = reinterpret_cast<float2*>(a.out_r + off);
#pragma unroll
            for (int j = 0; j < RP; ++j) orr[j * op2] = make_float2(round_half(lo2(A[j])), round_half(hi2(A[j])));
        }
    }
}

template <int R, int TH>
__host__ __device__ constexpr size_t blur_smem_bytes_rt() {
    return BlurTile<R, TH>::bytes > blur_fast_bytes<R, TH>() ? BlurTile<R, TH>::bytes : blur_fast_bytes<R, TH>();
}

template <int R, int TH>
__global__ void __launch_bounds__(BLUR_NT, TH == 40 ? 7 : 1) k_blur(const BlurArgs a) {
    chain_begin();
    extern __shared__ __align__(16) float smem[];
    const TileIO io{a.in, a.in_pitch, a.step, a.out, a.out_r, a.copy0, a.copy0_r, a.out_pitch, a.H, a.W};
    auto w = [&](int k) { return a.w2[k]; };
    if (blur_tile_is_fast(io, R, BlurFast<R>::RA, TH, blockIdx.x, blockIdx.y))
        blur_tile_fast<R, TH>(io, blockIdx.x, blockIdx.y, smem, w);
    else
        blur_tile<R, TH>(io, blockIdx.x, blockIdx.y, smem, w);
}

// Any radius up to PYSIFT_MAX_RADIUS (no register blocking); radius 0 copies.
__global__ void __launch_bounds__(BLUR_NT) k_blur_generic(const BlurArgs a, int R) {
    chain_begin();
    const int RA = (R + 3) / 4 * 4;
    const int TWP = BLUR_TW + 2 * RA, ROWS = BLUR_TH + 2 * R;
    extern __shared__ float smem[];
    float* tile = smem + (RA - R);
    float* hb = smem + ROWS * TWP + 4;
    const int c0 = blockIdx.x * BLUR_TW, r0 = blockIdx.y * BLUR_TH;
    blur_load_tile(a, smem, R, RA, TWP, ROWS, r0, c0);
    __syncthreads();
    for (int i = threadIdx.x; i < ROWS * BLUR_TW; i += BLUR_NT) {
        int rr = i / BLUR_TW, x = i - rr * BLUR_TW;
        float acc = 0.0f;
        if (R == 0) acc = tile[rr * TWP + x];
        else
            for (int k = 0; k <= 2 * R; ++k) acc = fmaf(tile[rr * TWP + x + k], a.w[k], acc);
        hb[i] = acc;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < BLUR_TH * BLUR_TW; i += BLUR_NT) {
        int y = i / BLUR_TW, x = i - y * BLUR_TW;
        float acc = 0.0f;
        if (R == 0) acc = hb[y * BLUR_TW + x];
        else
            for (int k = 0; k <= 2 * R; ++k) acc = fmaf(hb[(y + k) * BLUR_TW + x], a.w[k], acc);
        int gr = r0 + y, gc = c0 + x;
        if (gr < a.H && gc < a.W) {
            a.out[(long long)gr * a.out_pitch + gc] = acc;
            if (a.out_r) a.out_r[(long long)gr * a.out_pitch + gc] = round_half(acc);
        }
    }
}

static size_t blur_smem_bytes(int R) {
    const int RA = (R + 3) / 4 * 4;
    return (size_t)((BLUR_TH + 2 * R) * (BLUR_TW + 2 * RA) + (BLUR_TH + 2 * R) * BLUR_TW + 4) * sizeof(float);
}

typedef void (*BlurKernel)(const BlurArgs);

static int num_sms();

// Register-blocked blur variants: radius 1..16 x tile height 16, 32, 40.
constexpr int BLUR_NV = 3;
constexpr int BLUR_THS[BLUR_NV] = {16, 32, 40};
struct BlurVariant {
    BlurKernel fn;
    size_t smem;
};
static_assert(BlurTile<16, 40>::bytes <= 48 * 1024 && blur_fast_bytes<16, 40>() <= 48 * 1024,
              "k_blur<R, TH> stays within the default dynamic shared memory");

template <int R>
static BlurVariant blur_variant_r(int v) {
    switch (v) {
        case 0: return {k_blur<R, 16>, blur_smem_bytes_rt<R, 16>()};
        case 1: return {k_blur<R, 32>, blur_smem_bytes_rt<R, 32>()};
        default: return {k_blur<R, 40>, blur_smem_bytes_rt<R, 40>()};
    }
}

static BlurVariant blur_variant(int R, int v) {
    switch (R) {
        case 1: return blur_variant_r<1>(v);
        case 2: return blur_variant_r<2>(v);
        case 3: return blur_variant_r<3>(v);
        case 4: return blur_variant_r<4>(v);
        case 5: return blur_variant_r<5>(v);
        case 6: return blur_variant_r<6>(v);
        case 7: return blur_variant_r<7>(v);
        case 8: return blur_variant_r<8>(v);
        case 9: return blur_variant_r<9>(v);
        case 10: return blur_variant_r<10>(v);
        case 11: return blur_variant_r<11>(v);
        case 12: return blur_variant_r<12>(v);
        case 13: return blur_variant_r<13>(v);
        case 14: return blur_variant_r<14>(v);
        case 15: return blur_variant_r<15>(v);
        case 16: return blur_variant_r<16>(v);
        default: return {nullptr, 0};
    }
}

// Resident CTAs per SM of every variant, queried once per device.
static int blur_occupancy(int R, int v) {
    constexpr int MAXDEV = 64;
    static std::once_flag once[MAXDEV];
    static int occ[MAXDEV][BLUR_PAIR_MAX_R + 1][BLUR_NV];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAXDEV) return 1;
    std::call_once(once[dev], [dev] {
        for (int r = 1; r <= BLUR_PAIR_MAX_R; ++r)
            for (int k = 0; k < BLUR_NV; ++k) {
                const BlurVariant bv = blur_variant(r, k);
                int n = 0;
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, bv.fn, BLUR_NT, bv.smem) != cudaSuccess) n = 1;
                occ[dev][r][k] = n > 0 ? n : 1;
            }
    });
    return occ[dev][R][v];
}

// pysift_set_blur_tile_rows: a forced variant (testing), -1 = automatic
static std::atomic<int> g_blur_forced{-1};

// pysift_set_blur_tile_table: a measured variant per (radius, level size
// class), -1 = the cost rule below.  Size class: floor(log2(H W)) - 10,
// clamped to 0 .. BLUR_SIZE_CLASSES - 1.
constexpr int BLUR_SIZE_CLASSES = 16;
static std::atomic<int> g_blur_table[BLUR_PAIR_MAX_R + 1][BLUR_SIZE_CLASSES];
static std::once_flag g_blur_table_once;

static int blur_size_class(int H, int W) {
    const long long px = (long long)H * W;
    int lg = 0;
    while (lg < 62 && (2LL << lg) <= px) ++lg;
    return std::max(0, std::min(BLUR_SIZE_CLASSES - 1, lg - 10));
}

static void blur_table_init() {
    std::call_once(g_blur_table_once, [] {
        for (auto& row : g_blur_table)
            for (auto& e : row) e.store(-1, std::memory_order_relaxed);
    });
}

// The tile height: forced, else tuned, else the one with the fewest (rounds
// of resident CTAs) x (tile rows + halo): big levels avoid a short last
// round, small ones a long CTA.
static int blur_pick(int R, int H, int W) {
    const int forced = g_blur_forced.load(std::memory_order_relaxed);
    if (forced >= 0) return forced;
    blur_table_init();
    const int tuned = g_blur_table[R][blur_size_class(H, W)].load(std::memory_order_relaxed);
    if (tuned >= 0) return tuned;
    int best = 1;
    long long best_cost = -1;
    for (int v = 0; v < BLUR_NV; ++v) {
        const long long blocks = (long long)ceil_div(W, BLUR_TW) * ceil_div(H, BLUR_THS[v]);
        const long long slots = (long long)num_sms() * blur_occupancy(R, v);
        const long long rounds = (blocks + slots - 1) / slots;
        const long long cost = rounds * (BLUR_THS[v] + 2 * R);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = v;
        }
    }
    return best;
}

static int ensure_blur_attrs() {
    static std::once_flag once;
    static cudaError_t err = cudaSuccess;
    std::call_once(once, [] {
        cudaError_t e = cudaFuncSetAttribute(k_blur_generic, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)blur_smem_bytes(PYSIFT_MAX_RADIUS));
        if (e != cudaSuccess) err = e;
    });
    if (err != cudaSuccess) {
        set_error("cudaFuncSetAttribute(k_blur_generic): %s", cudaGetErrorString(err));
        return PYSIFT_ERR_CUDA;
    }
    return PYSIFT_OK;
}

static int launch_blur(BlurArgs& a, int R, const float* w, bool chained, cudaStream_t st) {
    for (int k = 0; k <= 2 * R; ++k) a.w[k] = w[k];
    for (int k = 0; k <= 2 * R && k <= 2 * BLUR_PAIR_MAX_R; ++k) {
        unsigned u = 0;
        memcpy(&u, &w[k], sizeof(u));
        a.w2[k] = ((unsigned long long)u << 32) | u;
    }
    if (R >= 1 && R <= BLUR_PAIR_MAX_R) {
        const int v = blur_pick(R, a.H, a.W);
        const BlurVariant bv = blur_variant(R, v);
        dim3 grid(ceil_div(a.W, BLUR_TW), ceil_div(a.H, BLUR_THS[v]));
        if (chained) launch_chained(bv.fn, grid, BLUR_NT, bv.smem, st, a);
        else bv.fn<<<grid, BLUR_NT, bv.smem, st>>>(a);
        PYSIFT_LAUNCH_CHECK("k_blur");
    } else {
        dim3 grid(ceil_div(a.W, BLUR_TW), ceil_div(a.H, BLUR_TH));
        int rc = ensure_blur_attrs();
        if (rc) return rc;
        k_blur_generic<<<grid, BLUR_NT, blur_smem_bytes(R), st>>>(a, R);
        PYSIFT_LAUNCH_CHECK("k_blur_generic");
    }
    return PYSIFT_OK;
}

int blur_level(const float* in, long long in_pitch, int step, float* out, int out_pitch, float* copy0, int H, int W,
               const float* w, int R, bool chained, cudaStream_t st) {
    static thread_local BlurArgs a;  // large (weights by value); not on the stack
    memset(&a, 0, sizeof(a));
    a.in = in;
    a.in_pitch = in_pitch;
    a.step = step;
    a.out = out;
    a.out_pitch = out_pitch;
    a.copy0 = copy0;
    a.H = H;
    a.W = W;
    return launch_blur(a, R, w, chained, st);
}

// ---------------------------------------------------------------------------
// A7: extrema bitmask + per-row counts, then deterministic compaction.
// ---------------------------------------------------------------------------
struct ExtArgs {
    OctView oct[PYSIFT_MAX_OCTAVES];
    int n_oct, S, border, thr_idx, retry_mode, cap;
    int blk_off[PYSIFT_MAX_OCTAVES + 1];
    int rows;  // rows of a k_extrema_mask strip
    uint32_t* mask[PYSIFT_MAX_OCTAVES];
    int* rowcnt[PYSIFT_MAX_OCTAVES];
    int* rowoff[PYSIFT_MAX_OCTAVES];
    int wpr[PYSIFT_MAX_OCTAVES];
    int4* cand;
};

__device__ __forceinline__ float dog_at(const OctView& v, int s, int r, int c) {
    long long off = (long long)r * v.pitch + c;
    return v.lev[s + 1][off] - v.lev[s][off];
}

__device__ __forceinline__ int find_octave(const int* blk_off, int n_oct, int b) {
    int o = 0;
    while (o + 1 < n_oct && b >= blk_off[o + 1]) ++o;
    return o;
}

// Three-input maximum and minimum (one instruction on sm_100).
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// A warp takes a strip of 64 columns (two adjacent ones a lane) and a.rows rows
// of one octave and walks down it: each Gaussian level is loaded once per
// row, one row ahead, and the DoG values (D_s = G_{s+1} - G_s) of three rows
// stay in registers.  Strips overlap by two columns, so that the 62 pixels
// tested have their neighbours in the warp.  A pixel is tested where |D| >
// threshold inside the border: first against the six neighbours along the
// axes, then, if any lane of the strip is left, against all 26 (D equals the
// maximum or the minimum of its 27): the column maxima over 3 rows and 3
// scales come from registers, the neighbours' by shuffle.  Extrema are rare
// (0.2 % of the pixels), so their bits go into the zeroed mask by atomics.
// Bound by the latency of the level loads (24 bytes a pixel): eight blocks an
// SM at 64 registers beat five with two rows in flight; the spills this costs
// (0, 48, 160, 228 and 496 bytes loaded for 1 .. 5 scales, by the compiler's
// count) leave every scale count faster than with staged tiles: whole
// detections at 1023x767 1.05, 1.10, 1.19, 1.17 and 1.13 times as fast.
// Staging 32 x 32 tiles in shared memory cost the halo's sectors, a store and a
// load per value and a barrier: both launches of a 4000x3000 detection (1.54 GB
// of levels, 235 us at the copy rate, and the retry's empty grid) 411 -> 280
// us, of a 640x480 one 19 -> 13.
constexpr int EX_T = 128, EX_COLS = 62;

template <int NL>
__device__ __forceinline__ void extrema_strips(const ExtArgs& a, int block, float thr) {
    constexpr int S = NL - 3, ND = NL - 1;
    const int o = find_octave(a.blk_off, a.n_oct, block);
    const OctView& v = a.oct[o];
    const int H = v.H, W = v.W, B = a.border, wpr = a.wpr[o];
    const int lane = threadIdx.x & 31;
    const int unit = (block - a.blk_off[o]) * (EX_T / 32) + (threadIdx.x >> 5);
    const int ncx = ceil_div(W, EX_COLS);
    const int ry = unit / ncx, r0 = ry * a.rows;
    if (r0 >= H) return;
    const int r1 = min(r0 + a.rows, H);  // rows r0 .. r1 - 1
    const int c = (unit - ry * ncx) * EX_COLS - 2 + 2 * lane;
    // columns outside the row read any value: their pixels lie in the border.
    // (__ldg: the levels are complete before the first pass, which is launched
    // the ordinary way, so in the chained retry too)
    const long long pitch = v.pitch, plane = v.lev[1] - v.lev[0];
    const float* src = v.lev[0] + (long long)max(r0 - 1, 0) * pitch + max(0, min(c, v.pitch - 2));
    float2 D[3][ND], g[NL];
    auto load = [&]() {
#pragma unroll
        for (int l = 0; l < NL; ++l) g[l] = __ldg(reinterpret_cast<const float2*>(src + l * plane));
    };
    // this lane's pixels: tested by this strip and inside the border
    const bool in0 = lane > 0 && c >= B && c < W - B, in1 = lane < 31 && c + 1 >= B && c + 1 < W - B;
    // row r arrives in slot t; the row before it, in slot t - 1, is tested
    auto step = [&](int r, auto slot) {
        constexpr int t = decltype(slot)::value, tb = (t + 2) % 3, ta = (t + 1) % 3;
#pragma unroll
        for (int s = 0; s < ND; ++s) D[t][s] = make_float2(g[s + 1].x - g[s].x, g[s + 1].y - g[s].y);
        if (r < r1) {
            if (r >= 0 && r + 1 < H) src += pitch;  // rows outside the image repeat the edge: border rows
            load();
        }
        const int rc = r - 1;
        if (rc < r0 || rc < B || rc >= H - B) return;
#pragma unroll
        for (int s = 1; s <= S; ++s) {
            const float2 val = D[tb][s];
            bool p0 = in0 && fabsf(val.x) > thr, p1 = in1 && fabsf(val.y) > thr;
            if (!__any_sync(FULL_MASK, p0 || p1)) continue;
            // most of these fall to their neighbours along the axes
            {
                const float l = __shfl_up_sync(FULL_MASK, val.y, 1), rr = __shfl_down_sync(FULL_MASK, val.x, 1);
                const float2 u = D[ta][s], d = D[t][s], q = D[tb][s - 1], w = D[tb][s + 1];
                p0 = p0 && (val.x >= max3(max3(l, val.y, u.x), max3(d.x, q.x, w.x), val.x) ||
                            val.x <= min3(min3(l, val.y, u.x), min3(d.x, q.x, w.x), val.x));
                p1 = p1 && (val.y >= max3(max3(val.x, rr, u.y), max3(d.y, q.y, w.y), val.y) ||
                            val.y <= min3(min3(val.x, rr, u.y), min3(d.y, q.y, w.y), val.y));
            }
            if (!__any_sync(FULL_MASK, p0 || p1)) continue;
            float mx[2], mn[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                auto at = [&](int row, int lev) { return j == 0 ? D[row][lev].x : D[row][lev].y; };
                mx[j] = max3(max3(at(ta, s - 1), at(tb, s - 1), at(t, s - 1)), max3(at(ta, s), at(tb, s), at(t, s)),
                             max3(at(ta, s + 1), at(tb, s + 1), at(t, s + 1)));
                mn[j] = min3(min3(at(ta, s - 1), at(tb, s - 1), at(t, s - 1)), min3(at(ta, s), at(tb, s), at(t, s)),
                             min3(at(ta, s + 1), at(tb, s + 1), at(t, s + 1)));
            }
            const float xl = __shfl_up_sync(FULL_MASK, mx[1], 1), xr = __shfl_down_sync(FULL_MASK, mx[0], 1);
            const float nl = __shfl_up_sync(FULL_MASK, mn[1], 1), nr = __shfl_down_sync(FULL_MASK, mn[0], 1);
            const bool e0 = p0 && (val.x == max3(xl, mx[0], mx[1]) || val.x == min3(nl, mn[0], mn[1]));
            const bool e1 = p1 && (val.y == max3(mx[0], mx[1], xr) || val.y == min3(mn[0], mn[1], nr));
            const unsigned b0 = __ballot_sync(FULL_MASK, e0), b1 = __ballot_sync(FULL_MASK, e1);
            if (b0 | b1) {
                const int row = (s - 1) * H + rc;
                uint32_t* m = a.mask[o] + (long long)row * wpr;
                if (e0) atomicOr(m + (c >> 5), 1u << (c & 31));
                if (e1) atomicOr(m + ((c + 1) >> 5), 1u << ((c + 1) & 31));
                if (lane == 0) atomicAdd(&a.rowcnt[o][row], __popc(b0) + __popc(b1));
            }
        }
    };
    load();
    for (int r = r0 - 1; r <= r1; r += 3) {
        step(r, std::integral_constant<int, 0>{});
        if (r + 1 <= r1) step(r + 1, std::integral_constant<int, 1>{});
        if (r + 2 <= r1) step(r + 2, std::integral_constant<int, 2>{});
    }
}

template <int NL>
__global__ void __launch_bounds__(EX_T, 8) k_extrema_mask(const __grid_constant__ ExtArgs a, Ctrl* ctrl) {
    chain_begin();
    if (a.retry_mode && !ctrl->retried) return;
    const float thr = ctrl->thr[a.thr_idx];
    for (int b = blockIdx.x; b < a.blk_off[a.n_oct]; b += gridDim.x) extrema_strips<NL>(a, b, thr);
}

typedef void (*ExtremaKernel)(const ExtArgs, Ctrl*);

static ExtremaKernel extrema_kernel(int S) {
    switch (S + 3) {
        case 4: return k_extrema_mask<4>;
        case 5: return k_extrema_mask<5>;
        case 6: return k_extrema_mask<6>;
        case 7: return k_extrema_mask<7>;
        case 8: return k_extrema_mask<8>;
        default: return nullptr;
    }
}
static_assert(PYSIFT_MAX_LEVELS == 8, "extrema_kernel covers n_scales 1..5");

__global__ void __launch_bounds__(1024) k_rowscan(const ExtArgs a, Ctrl* ctrl) {
    chain_begin();
    if (a.retry_mode && !ctrl->retried) return;
    __shared__ int sh[33];
    const int o = blockIdx.x;
    const int n = a.S * a.oct[o].H;
    const int per = (n + (int)blockDim.x - 1) / (int)blockDim.x;
    const int beg = threadIdx.x * per;
    int local = 0;
    for (int i = 0; i < per && beg + i < n; ++i) local += a.rowcnt[o][beg + i];
    int total;
    int off = block_excl_scan(local, &total, sh);
    for (int i = 0; i < per && beg + i < n; ++i) {
        int cnt = a.rowcnt[o][beg + i];
        a.rowoff[o][beg + i] = off;
        off += cnt;
    }
    if (threadIdx.x == 0) {
        ctrl->found[o] = total;
        ctrl->ncand[o] = total < a.cap ? total : a.cap;
        if (total > a.cap) atomicAdd(&ctrl->overflow_octs, 1);
    }
}

__global__ void __launch_bounds__(256) k_scatter(const ExtArgs a, Ctrl* ctrl) {
    chain_begin();
    if (a.retry_mode && !ctrl->retried) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int b = blockIdx.x; b < a.blk_off[a.n_oct]; b += gridDim.x) {
        const int o = find_octave(a.blk_off, a.n_oct, b);
        const int H = a.oct[o].H;
        const int unit = (b - a.blk_off[o]) * 8 + warp;  // (s-1)*H + r
        if (unit >= a.S * H || a.rowcnt[o][unit] == 0) continue;
        const int s = unit / H + 1, r = unit - (s - 1) * H;
        const int wpr = a.wpr[o];
        int base = a.rowoff[o][unit];
        const uint32_t* mrow = a.mask[o] + (long long)unit * wpr;
        int4* out = a.cand + (long long)o * a.cap;
        for (int w0 = 0; w0 < wpr; w0 += 32) {
            uint32_t word = (w0 + lane < wpr) ? mrow[w0 + lane] : 0u;
            int tot;
            int pos = base + warp_excl_scan(__popc(word), &tot);
            while (word) {
                int bit = __ffs(word) - 1;
                word &= word - 1;
                if (pos < a.cap) out[pos] = make_int4(s, r, (w0 + lane) * 32 + bit, 0);
                ++pos;
            }
            base += tot;
        }
    }
}

// ---------------------------------------------------------------------------
// A8: refinement.
// ---------------------------------------------------------------------------
struct RefArgs {
    OctView oct[PYSIFT_MAX_OCTAVES];
    int n_oct, S, border, cap, thr_idx, retry_mode, starvation_min;
    float edge_score;
    const int4* cand;
    int* rv_valid;
    float* rv_ri;
    float* rv_ci;
    int* rv_si;
    float* rv_resp;
    float* rf_ri;
    float* rf_ci;
    int* rf_si;
    float* rf_resp;
};

__global__ void __launch_bounds__(256) k_refine(const RefArgs a, Ctrl* ctrl) {
    chain_begin();
    if (a.retry_mode && !ctrl->retried) return;
    const float cthr = ctrl->thr[a.thr_idx];
    const long long nslots = (long long)a.n_oct * a.cap;
    for (long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x; slot < nslots;
         slot += (long long)gridDim.x * blockDim.x) {
        const int o = (int)(slot / a.cap);
        const int j = (int)(slot - (long long)o * a.cap);
        if (j >= ctrl->ncand[o]) continue;
        const OctView& v = a.oct[o];
        const int4 cd = a.cand[slot];
        int si = cd.x, row = cd.y, col = cd.z;
        const int H = v.H, W = v.W, S = a.S, B = a.border;
        float ox = 0.0f, oy = 0.0f, os_ = 0.0f;
        bool converged = false;
        for (int iter = 0; iter < 5; ++iter) {
            if (si < 1 || si > S || row < B || row >= H - B || col < B || col >= W - B) break;
            float cval = dog_at(v, si, row, col);
            float cxp = dog_at(v, si, row, col + 1), cxm = dog_at(v, si, row, col - 1);
            float cyp = dog_at(v, si, row + 1, col), cym = dog_at(v, si, row - 1, col);
            float sp = dog_at(v, si + 1, row, col), smn = dog_at(v, si - 1, row, col);
            float dx = (cxp - cxm) * 0.5f;
            float dy = (cyp - cym) * 0.5f;
            float ds = (sp - smn) * 0.5f;
            float dxx = cxp - 2.0f * cval + cxm;
            float dyy = cyp - 2.0f * cval + cym;
            float dss = sp - 2.0f * cval + smn;
            float dxy = (dog_at(v, si, row + 1, col + 1) - dog_at(v, si, row + 1, col - 1) -
                         dog_at(v, si, row - 1, col + 1) + dog_at(v, si, row - 1, col - 1)) *
                        0.25f;
            float dxs = (dog_at(v, si + 1, row, col + 1) - dog_at(v, si + 1, row, col - 1) -
                         dog_at(v, si - 1, row, col + 1) + dog_at(v, si - 1, row, col - 1)) *
                        0.25f;
            float dys = (dog_at(v, si + 1, row + 1, col) - dog_at(v, si + 1, row - 1, col) -
                         dog_at(v, si - 1, row + 1, col) + dog_at(v, si - 1, row - 1, col)) *
                        0.25f;
            float det = dxx * (dyy * dss - dys * dys) - dxy * (dxy * dss - dys * dxs) + dxs * (dxy * dys - dyy * dxs);
            if (fabsf(det) < 1e-12f) break;
            float inv_det = 1.0f / det;
            float p = -dx, q = -dy, rv = -ds;
            ox = (p * (dyy * dss - dys * dys) - dxy * (q * dss - dys * rv) + dxs * (q * dys - dyy * rv)) * inv_det;
            oy = (dxx * (q * dss - dys * rv) - p * (dxy * dss - dys * dxs) + dxs * (dxy * rv - q * dxs)) * inv_det;
            os_ = (dxx * (dyy * rv - q * dys) - dxy * (dxy * rv - q * dxs) + p * (dxy * dys - dyy * dxs)) * inv_det;
            if (fabsf(ox) < 0.5f && fabsf(oy) < 0.5f && fabsf(os_) < 0.5f) {
                converged = true;
                break;
            }
            col += (ox >= 0.0f) ? (int)(ox + 0.5f) : (int)(ox - 0.5f);
            row += (oy >= 0.0f) ? (int)(oy + 0.5f) : (int)(oy - 0.5f);
            si += (os_ >= 0.0f) ? (int)(os_ + 0.5f) : (int)(os_ - 0.5f);
        }
        int valid = 0;
        float response = 0.0f;
        if (converged && !(si < 1 || si > S || row < B || row >= H - B || col < B || col >= W - B)) {
            float cval = dog_at(v, si, row, col);
            float cxp = dog_at(v, si, row, col + 1), cxm = dog_at(v, si, row, col - 1);
            float cyp = dog_at(v, si, row + 1, col), cym = dog_at(v, si, row - 1, col);
            float dx_ = (cxp - cxm) * 0.5f;
            float dy_ = (cyp - cym) * 0.5f;
            float ds_ = (dog_at(v, si + 1, row, col) - dog_at(v, si - 1, row, col)) * 0.5f;
            response = fabsf(cval + 0.5f * (dx_ * ox + dy_ * oy + ds_ * os_));
            if (response >= cthr) {
                float dxx = cxp - 2.0f * cval + cxm;
                float dyy = cyp - 2.0f * cval + cym;
                float dxy = (dog_at(v, si, row + 1, col + 1) - dog_at(v, si, row + 1, col - 1) -
                             dog_at(v, si, row - 1, col + 1) + dog_at(v, si, row - 1, col - 1)) *
                            0.25f;
                float trace = dxx + dyy;
                float det2d = dxx * dyy - dxy * dxy;
                if (!(det2d <= 0.0f || (trace * trace / det2d) >= a.edge_score)) valid = 1;
            }
        }
        a.rv_valid[slot] = valid;
        if (valid) {
            a.rv_ri[slot] = (float)row + oy;
            a.rv_ci[slot] = (float)col + ox;
            a.rv_si[slot] = si;
            a.rv_resp[slot] = response;
        }
    }
}

// Ordered compaction of the valid refined candidates of one octave.
struct RefinedRow {
    float ri, ci, resp;
    int si, valid;
};
__global__ void __launch_bounds__(1024) k_refine_compact(const RefArgs a, Ctrl* ctrl) {
    chain_begin();
    if (a.retry_mode && !ctrl->retried) return;
    __shared__ int sh[33];
    const int o = blockIdx.x;
    const int n = ctrl->ncand[o];
    const long long base = (long long)o * a.cap;
    const int total = block_compact<8, RefinedRow>(
        n,
        [&](int j) {
            RefinedRow r;
            r.valid = a.rv_valid[base + j];
            r.ri = a.rv_ri[base + j];
            r.ci = a.rv_ci[base + j];
            r.si = a.rv_si[base + j];
            r.resp = a.rv_resp[base + j];
            return r;
        },
        [](const RefinedRow& r) { return r.valid != 0; },
        [&](int pos, const RefinedRow& r) {
            a.rf_ri[base + pos] = r.ri;
            a.rf_ci[base + pos] = r.ci;
            a.rf_si[base + pos] = r.si;
            a.rf_resp[base + pos] = r.resp;
        },
        sh);
    if (threadIdx.x == 0) {
        ctrl->nref[o] = total;
        if (a.retry_mode) return;
        // the last octave of the first pass decides on the starvation retry
        // (pysift/core.py:2066-2071)
        __threadfence();
        if (atomicAdd(&ctrl->compact_done, 1) == a.n_oct - 1) {
            __threadfence();
            int t = 0;
            for (int k = 0; k < a.n_oct; ++k) t += __ldcg(&ctrl->nref[k]);
            ctrl->retried = t < a.starvation_min ? 1 : 0;
        }
    }
}

// ---------------------------------------------------------------------------
// A9: keypoint cap (top `cap` by response, stable).
// ---------------------------------------------------------------------------
struct CapArgs {
    int n_oct, cap_cand, kp_cap;
    const float* rf_ri;
    const float* rf_ci;
    const int* rf_si;
    const float* rf_resp;
    int* kp_o;
    int* kp_si;
    float* kp_ri;
    float* kp_ci;
    float* kp_resp;
    uint32_t* kp_tb;
};

__device__ __forceinline__ void global_to_local(const int* nref_pref, int n_oct, int g, int* o, int* j) {
    int oo = 0;
    while (oo + 1 < n_oct && g >= nref_pref[oo + 1]) ++oo;
    *o = oo;
    *j = g - nref_pref[oo];
}

// Keys of up to CAP_SMEM_KEYS refined keypoints are staged in shared memory
// for the radix passes; larger sets are read from global memory each pass.
constexpr int CAP_SMEM_KEYS = 40960;
constexpr int CAP_T = 1024;
constexpr size_t CAP_SMEM_BYTES = (size_t)(32 * 256 + CAP_SMEM_KEYS) * sizeof(unsigned int);

__global__ void __launch_bounds__(CAP_T) k_cap(const CapArgs a, Ctrl* ctrl) {
    chain_begin();
    extern __shared__ unsigned int cap_smem[];
    unsigned int* whist = cap_smem;              // [32 warps][256] private digit histograms
    unsigned int* s_keys = cap_smem + 32 * 256;  // staged keys
    __shared__ int sh[33];
    __shared__ int pref[PYSIFT_MAX_OCTAVES + 1];
    __shared__ unsigned int hist[256];
    __shared__ unsigned int s_prefix, s_mask;
    __shared__ int s_need;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        pref[0] = 0;
        for (int o = 0; o < a.n_oct; ++o) pref[o + 1] = pref[o] + ctrl->nref[o];
    }
    __syncthreads();
    const int total = pref[a.n_oct];
    const bool capped = total > a.kp_cap;
    auto load = [&](int g, int* o, int* j) {
        global_to_local(pref, a.n_oct, g, o, j);
        return (long long)(*o) * a.cap_cand + *j;
    };
    if (!capped) {
        for (int g = tid; g < total; g += CAP_T) {
            int o, j;
            long long src = load(g, &o, &j);
            a.kp_o[g] = o;
            a.kp_si[g] = a.rf_si[src];
            a.kp_ri[g] = a.rf_ri[src];
            a.kp_ci[g] = a.rf_ci[src];
            a.kp_resp[g] = a.rf_resp[src];
            a.kp_tb[g] = 0u;
        }
        if (tid == 0) {
            ctrl->n_total_ref = total;
            ctrl->n_kept = total;
            ctrl->capped = 0;
        }
        return;
    }
    const bool in_smem = total <= CAP_SMEM_KEYS;
    if (in_smem) {
        for (int g = tid; g < total; g += CAP_T) {
            int o, j;
            s_keys[g] = __float_as_uint(a.rf_resp[load(g, &o, &j)]);
        }
    }
    auto key_at = [&](int g) {
        if (in_smem) return s_keys[g];
        int o, j;
        return __float_as_uint(a.rf_resp[load(g, &o, &j)]);
    };
    // radix select of the kp_cap-th largest response (non-negative float bits)
    if (tid == 0) {
        s_prefix = 0u;
        s_mask = 0u;
        s_need = a.kp_cap;
    }
    for (int pass = 3; pass >= 0; --pass) {
        for (int i = tid; i < 32 * 256; i += CAP_T) whist[i] = 0u;
        __syncthreads();
        const unsigned int prefix = s_prefix, mask = s_mask;
        for (int g = tid; g < total; g += CAP_T) {
            const unsigned int key = key_at(g);
            if ((key & mask) == prefix) atomicAdd(&whist[warp * 256 + ((key >> (8 * pass)) & 255u)], 1u);
        }
        __syncthreads();
        for (int d = tid; d < 256; d += CAP_T) {
            unsigned int s = 0u;
#pragma unroll 8
            for (int w = 0; w < 32; ++w) s += whist[w * 256 + d];
            hist[d] = s;
        }
        __syncthreads();
        if (warp == 0) {
            // digit d with cum(> d) < need <= cum(>= d): warp suffix sums over 8-digit groups
            int grp = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) grp += (int)hist[lane * 8 + q];
            int suf = grp;  // inclusive suffix sum over lanes lane..31
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_down_sync(FULL_MASK, suf, off);
                if (lane + off < 32) suf += v;
            }
            const int need = s_need;
            const int above = suf - grp;  // keys in higher groups
            const unsigned int who = __ballot_sync(FULL_MASK, above < need && need <= suf);
            if (lane == (who ? __ffs(who) - 1 : 0)) {
                int cum = above, d = lane * 8 + 7;
                for (; d > lane * 8; --d) {
                    if (cum + (int)hist[d] >= need) break;
                    cum += (int)hist[d];
                }
                s_need = need - cum;
                s_prefix = prefix | ((unsigned int)d << (8 * pass));
                s_mask = mask | (255u << (8 * pass));
            }
        }
        __syncthreads();
    }
    const unsigned int T = s_prefix;
    const int need_eq = s_need;
    // kept = every key > T and the first need_eq keys == T (index order), at
    // position #greater-before + min(#equal-before, need_eq); warp ballots of
    // both conditions and one packed scan of the warp counts per chunk
    constexpr int K = 8;
    const unsigned below = (1u << lane) - 1u;
    int gt_base = 0, eq_base = 0;
    for (int c0 = 0; c0 < total; c0 += CAP_T * K) {
        const int wbase = c0 + warp * 32 * K;
        unsigned int key[K], bgt[K], beq[K];
        int so[K], ssi[K];
        float sri[K], sci[K], sresp[K];
        // every load of the chunk first (coalesced within an octave), then the stores
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int g = wbase + k * 32 + lane;
            so[k] = 0;
            ssi[k] = 0;
            sri[k] = sci[k] = sresp[k] = 0.0f;
            if (g < total) {
                int o, j;
                const long long src = load(g, &o, &j);
                so[k] = o;
                ssi[k] = a.rf_si[src];
                sri[k] = a.rf_ri[src];
                sci[k] = a.rf_ci[src];
                sresp[k] = a.rf_resp[src];
            }
            key[k] = __float_as_uint(sresp[k]);
        }
        int cg = 0, ce = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int g = wbase + k * 32 + lane;
            bgt[k] = __ballot_sync(FULL_MASK, g < total && key[k] > T);
            beq[k] = __ballot_sync(FULL_MASK, g < total && key[k] == T);
            cg += __popc(bgt[k]);
            ce += __popc(beq[k]);
        }
        int tot;
        const int pre = block_warp_excl_scan(cg | (ce << 16), &tot, sh);
        int pg = gt_base + (pre & 0xffff), pe = eq_base + (pre >> 16);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const bool is_gt = (bgt[k] >> lane) & 1u, is_eq = (beq[k] >> lane) & 1u;
            const int gb = pg + __popc(bgt[k] & below), eb = pe + __popc(beq[k] & below);
            if (is_gt || (is_eq && eb < need_eq)) {
                const int pos = gb + min(eb, need_eq);
                a.kp_o[pos] = so[k];
                a.kp_si[pos] = ssi[k];
                a.kp_ri[pos] = sri[k];
                a.kp_ci[pos] = sci[k];
                a.kp_resp[pos] = sresp[k];
                a.kp_tb[pos] = ~key[k];
            }
            pg += __popc(bgt[k]);
            pe += __popc(beq[k]);
        }
        gt_base += tot & 0xffff;
        eq_base += tot >> 16;
    }
    if (tid == 0) {
        ctrl->n_total_ref = total;
        ctrl->n_kept = gt_base + min(eq_base, need_eq);
        ctrl->capped = 1;
    }
}

// ---------------------------------------------------------------------------
// A10: orientation.
// ---------------------------------------------------------------------------
struct OriArgs {
    OctView oct[PYSIFT_MAX_OCTAVES];
    float ori_sigma[PYSIFT_MAX_LEVELS];
    const int* kp_o;
    const int* kp_si;
    const float* kp_ri;
    const float* kp_ci;
    float* ang;
    int* angcnt;
};

// Exact, order-independent orientation histograms: each non-negative float32
// contribution is rounded to a multiple of 2^-40 (round to nearest even) and
// added as a 64-bit integer; a bin's value is the integer sum rounded to
// float32 and scaled back.  Contributions are below 2.2 (gradient magnitudes
// of pyramid values in [-0.28, 1.28]), so sums stay far below 2^63.  This makes the histograms independent of which thread adds
// what when, so any number of threads can share a keypoint.
__device__ __forceinline__ unsigned long long fix40(float c) {
    return (unsigned long long)__float2ll_rn(c * 0x1p40f);
}
__device__ __forceinline__ float unfix40(unsigned long long s) { return __ll2float_rn((long long)s) * 0x1p-40f; }

// Warp-private fixed-point orientation histograms with native 32-bit
// shared atomics.  A value q < 2^42 is added as two limbs, q mod 2^21 into
// lo[bin] and q >> 21 into hi[bin]; every FOLD_STEPS warp steps (at most 4
// values per lane and bin per step) the limbs are folded into a 64-bit total
// and cleared, so neither limb can overflow.  Integer sums keep the totals
// exact and independent of the order of the atomics.
constexpr int FOLD_STEPS = 8;

struct WarpHist {
    unsigned int* lo;
    unsigned int* hi;
    unsigned long long* tot;
    int nbins;
    __device__ __forceinline__ int phys(int bin) const { return bin; }
    __device__ __forceinline__ void add(int bin, unsigned long long q) const {
        const int p = phys(bin);
        atomicAdd(lo + p, (unsigned int)(q & 0x1fffffull));
        atomicAdd(hi + p, (unsigned int)(q >> 21));
    }
    // all lanes of the warp call fold() together
    __device__ __forceinline__ void fold() const {
        __syncwarp();
        for (int b = (int)(threadIdx.x & 31); b < nbins; b += 32) {
            const int p = phys(b);
            tot[b] += ((unsigned long long)hi[p] << 21) + (unsigned long long)lo[p];
            lo[p] = 0u;
            hi[p] = 0u;
        }
        __syncwarp();
    }
};

// fmodf(x, 360.0f) for x in (-360, 720): the remainder is exact in both forms
// (Sterbenz), so this matches fmodf bit for bit on the ranges the orientation
// (x in [180, 540]) and descriptor (x in (-180, 540]) formulas produce.
__device__ __forceinline__ float mod360(float x) { return x >= 360.0f ? x - 360.0f : x; }

// A block is one group of 256 threads or four of 64, a keypoint a group at
// a time: its first is the group's index, later ones come from a counter
// (windows differ in size), the next index requested when a keypoint starts
// and read when it ends.  Few keypoints get the whole block each (a window is
// 360 to 840 pixels and a pixel some 250 dependent instructions: 13.5 -> 5.8
// us for a 320x240 image, 14.4 -> 7.6 for 640x480);
// with more than the chip holds at once two warps are the cheapest, since each
// warp clears, folds and hands over a histogram of its own.
constexpr int ORI_T = 256;
constexpr int ORI_W = ORI_T / 32, ORI_G = ORI_T / 64;

__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + id), "r"(threads) : "memory");
}

struct OriShared {
    unsigned int wlo[ORI_W][36], whi[ORI_W][36];
    unsigned long long whist[ORI_W][36];
    float g0[ORI_G][36], g1[ORI_G][36];
    int s_next[ORI_G][2];  // alternates, so a late reader never sees the next keypoint
};

template <int GT>
__device__ __forceinline__ void orientation_groups(const OriArgs& a, Ctrl* ctrl, int n, OriShared& sm_) {
    constexpr int GW = GT / 32;
    auto& wlo = sm_.wlo;
    auto& whi = sm_.whi;
    auto& whist = sm_.whist;
    auto& g0 = sm_.g0;
    auto& g1 = sm_.g1;
    auto& s_next = sm_.s_next;
    const int grp = threadIdx.x / GT;
    const int tid = threadIdx.x % GT, lane = tid & 31, warp = threadIdx.x >> 5;  // warp within the block
    const int gwarp = tid >> 5;
    const int ngroups = (int)gridDim.x * (ORI_T / GT);
    float* const h0 = g0[grp];
    float* const h1 = g1[grp];
    int i = blockIdx.x * (ORI_T / GT) + grp;
    for (int it = 0; i < n; ++it) {
        int next = 0;
        if (tid == 0) next = ngroups + atomicAdd(&ctrl->ori_next, 1);
        for (int b = lane; b < 36; b += 32) {
            whist[warp][b] = 0ull;
            wlo[warp][b] = 0u;
            whi[warp][b] = 0u;
        }
        __syncwarp();
        const int o = a.kp_o[i], si = a.kp_si[i];
        const float ri = a.kp_ri[i], ci = a.kp_ci[i];
        const float sigma = a.ori_sigma[si];
        const OctView& v = a.oct[o];
        const int H = v.H, W = v.W;
        int radius = (int)(4.5f * sigma + 0.5f);
        if (radius < 1) radius = 1;
        const float sigma_w = 1.5f * sigma;
        const float inv_2sw2 = 1.0f / (2.0f * sigma_w * sigma_w + 1e-12f);
        int r_min = (int)ri - radius;
        if (r_min < 1) r_min = 1;
        int r_max = (int)ri + radius;
        if (r_max > H - 2) r_max = H - 2;
        int c_min = (int)ci - radius;
        if (c_min < 1) c_min = 1;
        int c_max = (int)ci + radius;
        if (c_max > W - 2) c_max = W - 2;
        int n_cols = c_max - c_min + 1;
        if (n_cols < 1) n_cols = 1;
        int nr = r_max - r_min + 1;
        if (nr < 0) nr = 0;
        const float* g = v.lev[si];
        const long long P = v.pitch;
        const WarpHist hw{wlo[warp], whi[warp], whist[warp], 36};
        // 8x4 pixel blocks per warp step
        const int tcols = (n_cols + 7) >> 3, trows = (nr + 3) >> 2;
        const int ntiles = tcols * trows;
        int steps = 0;
        // tile t -> (t / tcols, t % tcols), advanced GW tiles at a time
        const int dty = GW / tcols, dtx = GW - dty * tcols;
        int ty = gwarp / tcols, tx = gwarp - ty * tcols;
        for (int t = gwarp; t < ntiles; t += GW) {
            const int pr = ty * 4 + (lane >> 3), pc = tx * 8 + (lane & 7);
            tx += dtx;
            ty += dty;
            if (tx >= tcols) {
                tx -= tcols;
                ++ty;
            }
            const bool act = pr < nr && pc < n_cols;
            if (act) {
                const int r = r_min + pr, c = c_min + pc;
                const float* gp = g + r * P + c;
                float dx = gp[1] - gp[-1];
                float dy = gp[P] - gp[-P];
                float mag = sqrtf(dx * dx + dy * dy);
                float ori = mod360(sm::atan2f_(dy, dx) * 57.29577951f + 360.0f);
                float fr = (float)r - ri, fc = (float)c - ci;
                float wt = sm::expf_(-(fr * fr + fc * fc) * inv_2sw2);
                float bin_f = ori * 0.1f;  // 0 .. 36
                const float bin_fl = floorf(bin_f);
                int b0 = (int)bin_fl;
                b0 = b0 >= 36 ? b0 - 36 : b0;
                const int b1 = b0 == 35 ? 0 : b0 + 1;
                float frac = bin_f - bin_fl;
                float mw = mag * wt;
                hw.add(b0, fix40(mw * (1.0f - frac)));
                hw.add(b1, fix40(mw * frac));
            }
            if (++steps == FOLD_STEPS) {
                hw.fold();
                steps = 0;
            }
        }
        hw.fold();
        group_sync(grp, GT);
        // smoothing and peaks in the group's first warp: lane l owns bins l and
        // l + 32 (l < 4), same arithmetic per bin; the peak height is a maximum
        // (order-free)
        if (gwarp == 0) {
            for (int b = lane; b < 36; b += 32) {
                unsigned long long s = 0ull;
                for (int w = 0; w < GW; ++w) s += whist[warp + w][b];
                h0[b] = unfix40(s);
            }
            __syncwarp();
            for (int b = lane; b < 36; b += 32)
                h1[b] = 0.25f * h0[(b + 35) % 36] + 0.5f * h0[b] + 0.25f * h0[(b + 1) % 36];
            __syncwarp();
            for (int b = lane; b < 36; b += 32)
                h0[b] = 0.25f * h1[(b + 35) % 36] + 0.5f * h1[b] + 0.25f * h1[(b + 1) % 36];
            __syncwarp();
            float peak = 0.0f;
            for (int b = lane; b < 36; b += 32) peak = fmaxf(peak, h0[b]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) peak = fmaxf(peak, __shfl_xor_sync(FULL_MASK, peak, o));
            const float thr = 0.8f * peak;
            bool pk[2] = {false, false};
            float ang2[2] = {0.0f, 0.0f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int b = lane + 32 * h;
                if (b >= 36) continue;
                const float hb = h0[b];
                if (hb >= thr) {
                    const float l = h0[(b + 35) % 36], rv = h0[(b + 1) % 36];
                    if (hb >= l && hb >= rv) {
                        pk[h] = true;
                        const float denom = l - 2.0f * hb + rv;
                        const float fine = (float)b + (fabsf(denom) > 1e-12f ? 0.5f * (l - rv) / denom : 0.0f);
                        ang2[h] = fmodf(fine / 36.0f * 360.0f + 360.0f, 360.0f);
                    }
                }
            }
            const unsigned m0 = __ballot_sync(FULL_MASK, pk[0]), m1 = __ballot_sync(FULL_MASK, pk[1]) & 0xfu;
            const unsigned below = (1u << lane) - 1u;
            const int before0 = __popc(m0 & below), before1 = __popc(m0) + __popc(m1 & below);
            if (pk[0] && before0 < 4) a.ang[i * 4 + before0] = ang2[0];
            if (pk[1] && before1 < 4) a.ang[i * 4 + before1] = ang2[1];
            if (lane == 0) {
                const int cnt = min(4, __popc(m0) + __popc(m1));
                a.angcnt[i] = cnt;
                for (int k = cnt; k < 4; ++k) a.ang[i * 4 + k] = -1.0f;
            }
        }
        if (tid == 0) s_next[grp][it & 1] = next;
        group_sync(grp, GT);
        i = s_next[grp][it & 1];
    }
}

__global__ void __launch_bounds__(ORI_T) k_orientation(const __grid_constant__ OriArgs a, Ctrl* ctrl) {
    chain_begin();
    __shared__ OriShared sh;
    const int n = ctrl->n_kept;
    if (n <= (int)gridDim.x * 2) orientation_groups<256>(a, ctrl, n, sh);
    else orientation_groups<64>(a, ctrl, n, sh);
}

// ---------------------------------------------------------------------------
// Expansion into oriented keypoints + output sort keys.
// ---------------------------------------------------------------------------
struct ExpArgs {
    const int* kp_o;
    const int* kp_si;
    const float* kp_ri;
    const float* kp_ci;
    const uint32_t* kp_tb;
    const int* angcnt;
    int* ent_kp;
    int* ent_slot;
    uint4* keys;
    float coord_scale[PYSIFT_MAX_OCTAVES];  // 2^o * (0.5 if doubled else 1)
    int* xy_cnt;                             // per-bucket counts of the (x, y) order (zeroed)
    int* blk_cnt;                            // entries per k_expand block
    float xy_bscale;                         // BR_NB / image width
};

// Bucket of an (x, y) sort key: its x (a non-negative float) scaled to
// BR_NB bins over the image width.  Non-decreasing in x, hence in the key
// order (x first).
__device__ __forceinline__ int br_bucket_xy(const uint4& k, float bscale) {
    const float t = __uint_as_float(k.x) * bscale;
    return t < (float)(BR_NB - 1) ? (int)t : BR_NB - 1;
}
// Bucket of a response in the output-limit order (larger first): BR_NB - 1
// minus the float's exponent and top 8 mantissa bits, offset so that the
// BR_NB buckets span [2^-12, 2^4) (256 per octave) and clamped at both ends.
// Non-decreasing in that order for non-negative responses.
__device__ __forceinline__ int br_bucket_resp(float r) {
    constexpr int OFF = (127 - 12) << 8;  // the bucket of 2^-12
    const int f = (int)(__float_as_uint(r) >> 15) - OFF;
    return BR_NB - 1 - (f < 0 ? 0 : (f > BR_NB - 1 ? BR_NB - 1 : f));
}

// Expansion of the kept keypoints into their oriented entries (1..4 each),
// in keypoint order, over EXP_T x EXP_K keypoints per block: k_expand_count
// writes each block's entry count; in k_expand each block adds up the counts
// of the blocks before it (there are few) for its first entry, and a block
// scan places its own entries.  The last block stores the total.
constexpr int EXP_K = 8;
constexpr int EXP_T = 256;
constexpr int EXP_PER_BLOCK = EXP_T * EXP_K;

__global__ void __launch_bounds__(EXP_T) k_expand_count(const ExpArgs a, const Ctrl* ctrl) {
    chain_begin();
    __shared__ int sh[33];
    const int n = ctrl->n_kept;
    const int i0 = blockIdx.x * EXP_PER_BLOCK + (int)threadIdx.x * EXP_K;
    int local = 0;
#pragma unroll
    for (int k = 0; k < EXP_K; ++k)
        if (i0 + k < n) local += a.angcnt[i0 + k];
    int tot;
    block_excl_scan(local, &tot, sh);
    if (threadIdx.x == 0) a.blk_cnt[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(EXP_T) k_expand(const ExpArgs a, Ctrl* ctrl) {
    chain_begin();
    __shared__ int sh[33];
    __shared__ int s_base;
    const int n = ctrl->n_kept;
    if (threadIdx.x < 32) {
        int sum = 0;
        for (int b = (int)threadIdx.x; b < (int)blockIdx.x; b += 32) sum += a.blk_cnt[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL_MASK, sum, o);
        if (threadIdx.x == 0) s_base = sum;
    }
    const int i0 = blockIdx.x * EXP_PER_BLOCK + (int)threadIdx.x * EXP_K;
    int cnt[EXP_K];
    uint32_t kx[EXP_K], ky[EXP_K], tb[EXP_K];
    int local = 0;
#pragma unroll
    for (int k = 0; k < EXP_K; ++k) {
        const int i = i0 + k;
        cnt[k] = 0;
        kx[k] = ky[k] = tb[k] = 0u;
        if (i < n) {
            cnt[k] = a.angcnt[i];
            const float sc = a.coord_scale[a.kp_o[i]];
            kx[k] = __float_as_uint(a.kp_ci[i] * sc);
            ky[k] = __float_as_uint(a.kp_ri[i] * sc);
            tb[k] = a.kp_tb[i];
        }
        local += cnt[k];
    }
    int tot;
    const int excl = block_excl_scan(local, &tot, sh);  // its barriers also publish s_base
    int pos = s_base + excl;
#pragma unroll
    for (int k = 0; k < EXP_K; ++k) {
        const int i = i0 + k;
        for (int q = 0; q < cnt[k]; ++q) {
            a.ent_kp[pos + q] = i;
            a.ent_slot[pos + q] = q;
            const uint4 key = make_uint4(kx[k], ky[k], tb[k], (uint32_t)(i * 4 + q));
            a.keys[pos + q] = key;
            atomicAdd(&a.xy_cnt[br_bucket_xy(key, a.xy_bscale)], 1);
        }
        pos += cnt[k];
    }
    if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) ctrl->n_oriented = s_base + tot;
}

__device__ __forceinline__ bool key_less(const uint4& p, const uint4& q) {
    if (p.x != q.x) return p.x < q.x;
    if (p.y != q.y) return p.y < q.y;
    if (p.z != q.z) return p.z < q.z;
    return p.w < q.w;
}

// Exact ranks through buckets.  Keys follow a strict total order; a bucket
// function that never decreases along the order gives
//   rank[i] = #{keys in lower buckets} + #{keys of i's bucket ordered before i},
// the same count as comparing every pair.  Counts come from the kernel that
// writes the keys; k_br_scan turns them into bucket starts, k_br_scatter
// lists each bucket's members (in any order: the in-bucket count does not
// depend on it) and k_br_rank counts.  ORD 0: the (x, y) sort keys, rank =
// output row.  ORD 1: the rows' responses, larger first, ties by lower row
// (the output-limit order); nothing to do unless there are more rows than
// the limit.
struct BRArgs {
    const uint4* keys;      // ORD 0
    const float* row_resp;  // ORD 1
    float xy_bscale;
    int limit;              // ORD 1
    int* cnt;               // [BR_NB] counts
    int* off;               // [BR_NB] bucket starts
    int* cursor;            // [BR_NB] fill positions
    int* members;
    int* rank;
};

template <int ORD>
__device__ __forceinline__ bool br_skip(const BRArgs& a, int n) {
    return ORD == 1 && n <= a.limit;
}
template <int ORD>
__device__ __forceinline__ int br_bucket(const BRArgs& a, int i) {
    if (ORD == 0) return br_bucket_xy(a.keys[i], a.xy_bscale);
    return br_bucket_resp(a.row_resp[i]);
}

template <int ORD>
__global__ void __launch_bounds__(1024) k_br_scan(const BRArgs a, const Ctrl* ctrl) {
    chain_begin();
    __shared__ int sh[33];
    if (br_skip<ORD>(a, ctrl->n_oriented)) return;
    constexpr int PER = BR_NB / 1024;
    int c[PER], local = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        c[k] = a.cnt[threadIdx.x * PER + k];
        local += c[k];
    }
    int tot;
    int pos = block_excl_scan(local, &tot, sh);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        a.off[threadIdx.x * PER + k] = pos;
        a.cursor[threadIdx.x * PER + k] = pos;
        pos += c[k];
    }
}

template <int ORD>
__global__ void k_br_scatter(const BRArgs a, const Ctrl* ctrl) {
    chain_begin();
    const int n = ctrl->n_oriented;
    if (br_skip<ORD>(a, n)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        a.members[atomicAdd(&a.cursor[br_bucket<ORD>(a, i)], 1)] = i;
}

template <int ORD>
__global__ void k_br_rank(const BRArgs a, const Ctrl* ctrl) {
    chain_begin();
    const int n = ctrl->n_oriented;
    if (br_skip<ORD>(a, n)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int b = br_bucket<ORD>(a, i);
        const int s0 = a.off[b], s1 = s0 + a.cnt[b];
        int r = s0;
        if (ORD == 0) {
            const uint4 me = a.keys[i];
            for (int s = s0; s < s1; ++s) r += key_less(a.keys[a.members[s]], me) ? 1 : 0;
        } else {
            const float me = a.row_resp[i];
            for (int s = s0; s < s1; ++s) {
                const int j = a.members[s];
                const float o = a.row_resp[j];
                r += (o > me || (o == me && j < i)) ? 1 : 0;
            }
        }
        a.rank[i] = r;
    }
}

// ---------------------------------------------------------------------------
// A11: descriptor.
// ---------------------------------------------------------------------------
struct DescArgs {
    OctView oct[PYSIFT_MAX_OCTAVES];
    float desc_ph[PYSIFT_MAX_LEVELS];
    float kp_size[PYSIFT_MAX_OCTAVES][PYSIFT_MAX_LEVELS];
    float coord_scale[PYSIFT_MAX_OCTAVES];
    float dsp_scales[8];
    int n_dsp;  // 0 = single scale
    int rootsift;
    const int* kp_o;
    const int* kp_si;
    const float* kp_ri;
    const float* kp_ci;
    const float* kp_resp;
    const float* ang;
    const int* ent_kp;
    const int* ent_slot;
    const int* rank;
    const int* lrank;  // rank by response of each output row (output_limit > 0)
    unsigned long long* split_tot;  // [DESC_SPLIT_MAX][128] totals of the entries cut into parts, zeroed
    int* split_cnt;                 // parts that have arrived, zeroed
    int limit;
    float* out_kpts;
    float* out_resp;
    int* out_oct;
    float* out_desc;
    int n_oct, doubled;  // for the counters
    int32_t* stats;
};

constexpr int DESC_T = 256;
constexpr int DESC_W = DESC_T / 32;
// Lane layout of a descriptor warp step: the 32 lanes form DESC_GR x DESC_GC
// groups of DESC_L consecutive pixels of one row; the groups sit in
// different row bands and column bands of the patch (a band is 1/DESC_GR of
// the patch height, 1/DESC_GC of its width), so lanes of different groups
// fall in different spatial bins and their histogram updates do not
// serialise on one shared-memory word, while each group's loads stay
// contiguous.
#ifndef DESC_GR
#define DESC_GR 4
#endif
#ifndef DESC_GC
#define DESC_GC 2
#endif
constexpr int DESC_L = 32 / (DESC_GR * DESC_GC);
static_assert(DESC_GR * DESC_GC * DESC_L == 32, "descriptor lane groups must tile a warp");

// Descriptor histograms: exact fixed point at a quantum of 2^-24, one 32-bit
// shared word per bin and warp (one atomic per corner).  Pyramid values lie
// in [-0.28, 1.28] (u8/255, widened by the cubic spline of the 2x base), so
// a gradient magnitude is below 2.2 and a pixel's eight corner weights sum
// to at most that; a warp step adds at most 32 * 2.2 * 2^24 + 64 < 1.19e9 to
// one bin, and folding the words into 64-bit totals every DESC_FOLD_STEPS = 3
// steps keeps them below 2^32.  Bin b sits at b ^ (ycell << 3), so the
// y-cell moves a bin to another bank.
constexpr int DESC_FOLD_STEPS = 3;
__device__ __forceinline__ float unfix24(unsigned long long s) { return __ull2float_rn(s) * 0x1p-24f; }

struct DescHist {
    unsigned* h;               // [128] words of this warp
    unsigned long long* tot;   // [128] totals of this warp
    __device__ static __forceinline__ int phys(int bin) { return bin ^ (((bin >> 5) & 3) << 3); }
    // all lanes of the warp call fold() together
    __device__ __forceinline__ void fold() const {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int b = (int)(threadIdx.x & 31) + 32 * i;
            const int p = phys(b);
            tot[b] += (unsigned long long)h[p];
            h[p] = 0u;
        }
        __syncwarp();
    }
};

template <bool SPLIT>
__device__ __forceinline__ void desc_accumulate(const float* __restrict__ g, long long P, int H, int W, float ri,
                                                float ci, float cos_a, float sin_a, float ang_rad, int ph,
                                                const DescHist& hw, int tid, int part, int parts) {
    const float scale_sp = 4.0f / (2.0f * (float)ph);
    const float sigma_d = (float)ph * 0.5657f;
    const float inv_2s2 = 1.0f / (2.0f * sigma_d * sigma_d + 1e-12f);
    const int side = 2 * ph + 1;
    const int r0 = (int)ri, c0 = (int)ci;
    const int lane = tid & 31, warp = tid >> 5;
    const int k = lane % DESC_L, grp = lane / DESC_L;
    const int gi = grp / DESC_GC, gj = grp - gi * DESC_GC;
    const int band_r = (side + DESC_GR - 1) / DESC_GR;  // rows per row band
    const int band_c = (side + DESC_GC - 1) / DESC_GC;  // columns per column band
    const int runs = (band_c + DESC_L - 1) / DESC_L;    // DESC_L-pixel runs per band row
    const int nsteps = band_r * runs;
    // step t -> (u, v) = (t / runs, t % runs), advanced by `every` steps at a
    // time with one carry instead of a division per step
    const int every = SPLIT ? DESC_W * parts : DESC_W, first = SPLIT ? part * DESC_W + warp : warp;
    const int du = every / runs, dv = every - du * runs;
    int u = first / runs, v = first - u * runs;
    const int pr0 = gi * band_r, pc0 = gj * band_c + k;
    // the patch rows, and this lane's patch columns, whose central differences
    // lie inside the level: [r_lo, r_lo + r_n) and [c_lo, c_lo + c_n)
    const int r_lo = max(0, 1 - r0 + ph), c_lo = max(gj * band_c, 1 - c0 + ph);
    const unsigned r_n = (unsigned)max(0, min(side, H - 1 - r0 + ph) - r_lo);
    const unsigned c_n = (unsigned)max(0, min(min(side, (gj + 1) * band_c), W - 1 - c0 + ph) - c_lo);
    unsigned* const hb = hw.h;
    int steps = 0;
    for (int t = first; t < nsteps; t += every) {
        const int pr = pr0 + u, pc = pc0 + v * DESC_L;
        v += dv;
        u += du;
        if (v >= runs) {
            v -= runs;
            ++u;
        }
        const int r_off = pr - ph, c_off = pc - ph;
        float fc = (float)c_off, fr = (float)r_off;
        float xr = cos_a * fc - sin_a * fr;
        float yr = sin_a * fc + cos_a * fr;
        float xb = xr * scale_sp + 1.5f;
        float yb = yr * scale_sp + 1.5f;
        const bool act = (unsigned)(pr - r_lo) < r_n && (unsigned)(pc - c_lo) < c_n &&
                         !(xb < -0.5f || xb >= 3.5f || yb < -0.5f || yb >= 3.5f);
        if (act) {
            const float* gp = g + (r0 + r_off) * P + (c0 + c_off);
            float dx = gp[1] - gp[-1];
            float dy = gp[P] - gp[-P];
            float mag = sqrtf(dx * dx + dy * dy);
            // a flat sample's angle is NaN and its magnitude 0: its
            // contributions convert to 0
            float ori_deg = mod360((sm::atan2f_nonzero_(dy, dx) - ang_rad) * 57.29577951f + 360.0f);
            // |(xr, yr)| <= 1.5 ph: the argument stays above -4
            float gw = sm::expf_neg_(-(xr * xr + yr * yr) * inv_2s2);
            // the quantum's power of two goes into the magnitude: scaling by it
            // commutes with the products' rounding
            const float wmag = mag * gw * 0x1p24f;
            const float ob = ori_deg * 0.02222222f;
            const float of = floorf(ob), xf = floorf(xb), yf = floorf(yb);
            const int oi0 = (int)of, xi0 = (int)xf, yi0 = (int)yf;  // xi0, yi0 in -1 .. 3
            const float df = ob - of, dx_b = xb - xf, dy_b = yb - yf;
            const int xi0c = max(0, xi0), yi0c = max(0, yi0);
            const int xi1c = min(xi0 + 1, 3), yi1c = min(yi0 + 1, 3);
            // orientation bins mod 8 (two's complement & 7 is the
            // non-negative remainder for every int)
            const int oi0w = oi0 & 7, oi1w = (oi0 + 1) & 7;
            float w_y0 = 1.0f - dy_b, w_y1 = dy_b;
            float w_x0 = 1.0f - dx_b, w_x1 = dx_b;
            float w_o0 = 1.0f - df, w_o1 = df;
            // shared-memory word of bin y*32 + x*8 + o: the descriptor
            // histograms store it at y*32 + ((x ^ y) << 3) + o
            const int b00 = yi0c * 32 + ((xi0c ^ yi0c) << 3), b01 = yi0c * 32 + ((xi1c ^ yi0c) << 3);
            const int b10 = yi1c * 32 + ((xi0c ^ yi1c) << 3), b11 = yi1c * 32 + ((xi1c ^ yi1c) << 3);
            const unsigned q[8] = {
                __float2uint_rn(w_y0 * w_x0 * w_o0 * wmag), __float2uint_rn(w_y0 * w_x0 * w_o1 * wmag),
                __float2uint_rn(w_y0 * w_x1 * w_o0 * wmag), __float2uint_rn(w_y0 * w_x1 * w_o1 * wmag),
                __float2uint_rn(w_y1 * w_x0 * w_o0 * wmag), __float2uint_rn(w_y1 * w_x0 * w_o1 * wmag),
                __float2uint_rn(w_y1 * w_x1 * w_o0 * wmag), __float2uint_rn(w_y1 * w_x1 * w_o1 * wmag)};
            const int pb[8] = {b00 + oi0w, b00 + oi1w, b01 + oi0w, b01 + oi1w,
                               b10 + oi0w, b10 + oi1w, b11 + oi0w, b11 + oi1w};
#pragma unroll
            for (int c = 0; c < 8; ++c) atomicAdd(hb + pb[c], q[c]);
        }
        if (++steps == DESC_FOLD_STEPS) {
            hw.fold();
            steps = 0;
        }
    }
    hw.fold();
}

__device__ __forceinline__ float warp_tree_sum(float v) {
    v += __shfl_down_sync(FULL_MASK, v, 16);
    v += __shfl_down_sync(FULL_MASK, v, 8);
    v += __shfl_down_sync(FULL_MASK, v, 4);
    v += __shfl_down_sync(FULL_MASK, v, 2);
    v += __shfl_down_sync(FULL_MASK, v, 1);
    return v;
}

// Sum over the 128 bins (thread = bin) in the reference's order: a warp
// shuffle tree per 32 bins, then the four warp partials in order.
// Called by threads 0..127 only (named barrier 1 over those 4 warps).
__device__ __forceinline__ float bins_sum(float x, float* part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float w = warp_tree_sum(x);
    if (lane == 0) part[warp] = w;
    asm volatile("bar.sync 1, 128;" ::: "memory");
    float s = part[0] + part[1] + part[2] + part[3];
    asm volatile("bar.sync 1, 128;" ::: "memory");
    return s;
}

// The run's counters (one thread).
__device__ void write_stats(const Ctrl* ctrl, int32_t* stats, int n_oct, int doubled, int limit) {
    for (int t = 0; t < PYSIFT_STAT_COUNT; ++t) stats[t] = 0;
    {
        int nref = 0;
        for (int o = 0; o < n_oct; ++o) nref += ctrl->nref[o];
        stats[PYSIFT_STAT_N_KEYPOINTS] = (limit > 0 && ctrl->n_oriented > limit) ? limit : ctrl->n_oriented;
        stats[PYSIFT_STAT_N_REFINED] = nref;
        stats[PYSIFT_STAT_N_KEPT] = ctrl->n_kept;
        stats[PYSIFT_STAT_RETRIED] = ctrl->retried;
        stats[PYSIFT_STAT_CAPPED] = ctrl->capped;
        stats[PYSIFT_STAT_DOUBLED] = doubled;
        stats[PYSIFT_STAT_CAND_OVERFLOW] = ctrl->overflow_octs;
        for (int o = 0; o < n_oct; ++o) {
            stats[PYSIFT_STAT_CANDS + o] = ctrl->found[o];
            stats[PYSIFT_STAT_REFINED_OCT + o] = ctrl->nref[o];
        }
        stats[PYSIFT_STAT_THRESH_BITS] = (int32_t)__float_as_uint(ctrl->thr[ctrl->retried ? 1 : 0]);
    }
}

// One DESC_T-thread block per oriented keypoint at a time; a block takes its
// next entry from a counter (entries differ in patch size, so blocks stay
// busy until the list is done; every entry writes its own output row).
// Warps accumulate into private fixed-point histograms; threads 0..127 then
// own one bin each for the merge, normalisation and RootSIFT.
//
// When the entries are few times the resident blocks, each is cut into parts
// (every parts-th warp step), which add their integer totals to the entry's in
// global memory; the part that arrives last finishes the entry.  The sums are
// exact, so the result does not depend on the cut.  Whole entries left the
// chip waiting for the blocks with one entry more: 425 -> 318 us for the 1,100
// DSP-5 entries of a 1023x767 image, 22.7 -> 16.4 for a 320x240 one.
constexpr int DESC_OCC = 5;          // resident blocks an SM
constexpr int DESC_MAX_PARTS = 8;
// units wanted per resident block before entries stay whole: a part costs its
// clearing and merging (about two steps of its warps), little against the
// five patches of a DSP entry and much against a single one
constexpr int DESC_UNITS_DSP = 6, DESC_UNITS = 1;
constexpr int DESC_SPLIT_MAX = 148 * DESC_OCC * DESC_UNITS_DSP / 2;  // entries that can be cut (two parts at least)

__global__ void __launch_bounds__(DESC_T, DESC_OCC) k_descriptor(const DescArgs a, Ctrl* ctrl) {
    chain_begin();
    __shared__ unsigned int wh32[DESC_W][128];
    __shared__ unsigned long long whist[DESC_W][128];
    __shared__ float part_sum[4];
    __shared__ int s_entry[2];  // alternates, so a late reader never sees the next entry
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int n = ctrl->n_oriented;
    if (blockIdx.x == gridDim.x - 1 && tid == DESC_T - 1) write_stats(ctrl, a.stats, a.n_oct, a.doubled, a.limit);
    const int parts =
        n > DESC_SPLIT_MAX || n == 0
            ? 1
            : max(1, min(DESC_MAX_PARTS, (a.n_dsp > 0 ? DESC_UNITS_DSP : DESC_UNITS) * (int)gridDim.x / n));
    // the first unit is the block index, later ones come from the counter;
    // the next index is requested when a unit starts and read when it ends
    int unit = blockIdx.x;
    for (int it = 0; unit < n * parts; ++it) {
        const int e = unit / parts, part = unit - e * parts;
        int next = 0;
        if (tid == 0) next = (int)gridDim.x + atomicAdd(&ctrl->desc_next, 1);
        for (int b = tid; b < DESC_W * 128; b += DESC_T) {
            (&whist[0][0])[b] = 0ull;
            (&wh32[0][0])[b] = 0u;
        }
        __syncthreads();
        int row = a.rank[e];
        if (a.limit > 0 && n > a.limit) row = a.lrank[row];
        if (!(a.limit > 0 && n > a.limit) || row < a.limit) {  // else the whole block skips this entry
            const int kp = a.ent_kp[e], slot = a.ent_slot[e];
            const int o = a.kp_o[kp], si = a.kp_si[kp];
            const float ri = a.kp_ri[kp], ci = a.kp_ci[kp];
            const float angle = a.ang[kp * 4 + slot];
            const float ang_rad = angle * (float)(3.14159265358979323846 / 180.0);
            const float phf = a.desc_ph[si];
            const OctView& v = a.oct[o];
            float sin_a, cos_a;
            sm::sincosf_(ang_rad, &sin_a, &cos_a);
            const float* g = v.lev[si];
            const DescHist hw{wh32[warp], whist[warp]};
            for (int dd = 0; dd < max(a.n_dsp, 1); ++dd) {
                const int ph = a.n_dsp > 0 ? max(4, (int)(phf * a.dsp_scales[dd] + 0.5f)) : (int)phf;
                if (parts > 1)
                    desc_accumulate<true>(g, v.pitch, v.H, v.W, ri, ci, cos_a, sin_a, ang_rad, ph, hw, tid, part, parts);
                else
                    desc_accumulate<false>(g, v.pitch, v.H, v.W, ri, ci, cos_a, sin_a, ang_rad, ph, hw, tid, 0, 1);
            }
            __syncthreads();
            unsigned long long s = 0ull;
            if (tid < 128) {
#pragma unroll
                for (int w = 0; w < DESC_W; ++w) s += whist[w][tid];
            }
            bool finish = true;
            if (parts > 1) {
                if (tid < 128 && s) atomicAdd(&a.split_tot[(long long)e * 128 + tid], s);
                __threadfence();
                __syncthreads();
                if (tid == 0) s_last = atomicAdd(&a.split_cnt[e], 1) == parts - 1;
                __syncthreads();
                finish = s_last != 0;
                if (finish && tid < 128) {
                    __threadfence();
                    s = __ldcg(&a.split_tot[(long long)e * 128 + tid]);
                }
            }
            if (finish && tid < 128) {
                float val = unfix24(s);
                if (a.n_dsp > 0) val = val * (1.0f / (float)a.n_dsp);
                float inv = 1.0f / sqrtf(bins_sum(val * val, part_sum) + 1e-14f);
                float t = val * inv;
                val = t > 0.2f ? 0.2f : t;
                inv = 1.0f / sqrtf(bins_sum(val * val, part_sum) + 1e-14f);
                val = val * inv;
                if (a.rootsift) {
                    const float den = bins_sum(fabsf(val), part_sum) + 1e-7f;
                    float q = val / den;
                    if (q < 0.0f) q = 0.0f;
                    val = sqrtf(q);
                }
                a.out_desc[(long long)row * 128 + tid] = val;
                if (tid == 0) {
                    const float sc = a.coord_scale[o];
                    a.out_kpts[row * 4 + 0] = ci * sc;
                    a.out_kpts[row * 4 + 1] = ri * sc;
                    a.out_kpts[row * 4 + 2] = a.kp_size[o][si];
                    a.out_kpts[row * 4 + 3] = angle;
                    a.out_resp[row] = a.kp_resp[kp];
                    a.out_oct[row] = o;
                }
            }
        }
        if (tid == 0) s_entry[it & 1] = next;
        __syncthreads();
        unit = s_entry[it & 1];
    }
}

// Response of every output row (rows are the (x, y) ranks of the oriented
// entries), counted into the output-limit order's buckets.
__global__ void k_row_resp(const int* ent_kp, const float* kp_resp, const int* rank, float* __restrict__ row_resp,
                           int* __restrict__ resp_cnt, const Ctrl* ctrl) {
    chain_begin();
    const int n = ctrl->n_oriented;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const float r = kp_resp[ent_kp[e]];
        row_resp[rank[e]] = r;
        atomicAdd(&resp_cnt[br_bucket_resp(r)], 1);
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
static size_t split_entries(size_t kcap) { return std::min<size_t>(4 * kcap, DESC_SPLIT_MAX); }
static size_t split_bytes(size_t kcap) { return split_entries(kcap) * (128 * sizeof(unsigned long long) + sizeof(int)); }

template <typename T>
static T* at(void* ws, size_t off) {
    return reinterpret_cast<T*>(static_cast<char*>(ws) + off);
}

static void fill_oct_views(const Layout& l, void* ws, bool rounded, OctView* out) {
    for (int o = 0; o < l.n_oct; ++o) {
        size_t off = rounded ? l.off_pyr_r[o] : l.off_pyr[o];
        float* base = at<float>(ws, off);
        for (int s = 0; s < PYSIFT_MAX_LEVELS; ++s)
            out[o].lev[s] = (s < l.L) ? base + (size_t)s * l.H[o] * l.pitch[o] : nullptr;
        out[o].H = l.H[o];
        out[o].W = l.W[o];
        out[o].pitch = l.pitch[o];
    }
}

static int g_num_sms = 0;

static int num_sms() {
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        g_num_sms = n > 0 ? n : 148;
    }
    return g_num_sms;
}

// A second stream paired with each caller stream (per host thread and
// device), with events reused from call to call: work that only depends on
// part of the pyramid (the entropy histogram; levels S+1 and S+2 of each
// octave, which no later octave reads) runs there, forked from and joined
// back into the caller's stream, inside a CUDA graph capture too.  The pair
// is created on the first call made with that caller stream outside a
// capture; a call that captures on a stream without a pair returns null
// here and runs everything on the caller's stream (no objects are created
// while a capture is open).
struct SidePair {
    int dev;
    cudaStream_t main, side;
    cudaEvent_t ev[PYSIFT_MAX_OCTAVES + 2];
};

static SidePair* side_pair(cudaStream_t st) {
    constexpr int MAXP = 64;
    thread_local SidePair pairs[MAXP];
    thread_local int n = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        set_error("side_pair: no current device");
        return nullptr;
    }
    for (int i = 0; i < n; ++i)
        if (pairs[i].dev == dev && pairs[i].main == st) return &pairs[i];
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return nullptr;
    if (n == MAXP) return nullptr;
    SidePair p{};
    p.dev = dev;
    p.main = st;
    if (cudaStreamCreateWithFlags(&p.side, cudaStreamNonBlocking) != cudaSuccess) {
        set_error("side_pair: cudaStreamCreateWithFlags failed");
        return nullptr;
    }
    for (auto& e : p.ev) {
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            set_error("side_pair: cudaEventCreateWithFlags failed");
            return nullptr;
        }
    }
    pairs[n] = p;
    return &pairs[n++];
}

static int record_stage(void* const* ev, int i, cudaStream_t st) {
    if (ev && ev[i]) PYSIFT_CUDA_TRY(cudaEventRecord(reinterpret_cast<cudaEvent_t>(ev[i]), st));
    return PYSIFT_OK;
}

#define PYSIFT_STAGE(i)                              \
    do {                                             \
        int rc_ = record_stage(stage_events, i, st); \
        if (rc_) return rc_;                         \
    } while (0)

static int run_detect(const pysift_detect_config* cfg, const uint8_t* gray, int H, int W, long long pitch,
                      void* ws, const Layout& l, float* kpts, float* resp, int32_t* octv, float* desc,
                      int32_t* stats, void* const* stage_events, cudaStream_t st) {
    PYSIFT_STAGE(0);
    const int S = l.S, n_oct = l.n_oct;
    const int cap = cfg->max_cands_per_octave, kcap = cfg->keypoint_cap;
    Ctrl* ctrl = at<Ctrl>(ws, l.off_ctrl);
    PYSIFT_CUDA_TRY(cudaMemsetAsync(ctrl, 0, sizeof(Ctrl), st));
    SidePair* sp = side_pair(st);  // null: everything on st
    const cudaStream_t side = sp ? sp->side : st;
    if (sp) {
        PYSIFT_CUDA_TRY(cudaEventRecord(sp->ev[0], st));
        PYSIFT_CUDA_TRY(cudaStreamWaitEvent(side, sp->ev[0], 0));
    }
    // (side stream, read after the join) what later kernels count in; A1, the threshold of the extrema test
    PYSIFT_CUDA_TRY(cudaMemsetAsync(at<char>(ws, l.off_split), 0, split_bytes(kcap), side));
    int* bkt = at<int>(ws, l.off_bkt);  // [order][cnt | off | cursor][BR_NB]
    PYSIFT_CUDA_TRY(cudaMemsetAsync(bkt, 0, sizeof(int) * 2 * 3 * BR_NB, side));
    PYSIFT_CUDA_TRY(cudaMemsetAsync(at<char>(ws, l.off_rowcnt_base), 0, 2 * l.zero_bytes, side));
    {
        const int blocks = std::max(1, std::min(ceil_div(H, 8), num_sms() * 2));
        k_histogram<<<blocks, 256, 0, side>>>(gray, H, W, pitch, ctrl, cfg->contrast_thresh, S);
        PYSIFT_LAUNCH_CHECK("k_histogram");
    }
    // A2/A3: base image
    float* base = at<float>(ws, l.off_base);
    if (l.doubled) {
        double* coef = at<double>(ws, l.off_coef);
        int rc = launch_zoom2x(gray, H, W, pitch, cfg->fp16_pyramid, coef, base, l.pitch0, st);
        if (rc) return rc;
    } else {
        k_u8_to_f32<<<dim3(ceil_div(W, 256), H), 256, 0, st>>>(gray, H, W, pitch, cfg->fp16_pyramid, base,
                                                               l.pitch0);
        PYSIFT_LAUNCH_CHECK("k_u8_to_f32");
    }
    PYSIFT_STAGE(1);
    // A4/A5: pyramid
    {
        static thread_local BlurArgs a;  // large (weights by value); not on the stack
        for (int o = 0; o < n_oct; ++o) {
            float* pyr = at<float>(ws, l.off_pyr[o]);
            float* pyr_r = (l.off_pyr_r[o] != l.off_pyr[o]) ? at<float>(ws, l.off_pyr_r[o]) : nullptr;
            const size_t lev = (size_t)l.H[o] * l.pitch[o];
            // level 0
            memset(&a, 0, sizeof(a));
            a.H = l.H[o];
            a.W = l.W[o];
            a.out_pitch = l.pitch[o];
            if (o == 0) {
                int k = l.doubled ? 0 : 1;
                a.in = base;
                a.in_pitch = l.pitch0;
                a.step = 1;
                a.out = pyr;
                a.out_r = pyr_r;
                int rc = launch_blur(a, cfg->blur_radius[k], cfg->blur_weights[k], true, st);
                if (rc) return rc;
            }
            for (int s = 0; s < S + 2; ++s) {
                // levels S+1 and S+2 on the side stream, once level S exists
                cudaStream_t ls = st;
                if (s >= S) {
                    ls = side;
                    if (s == S && sp) {
                        PYSIFT_CUDA_TRY(cudaEventRecord(sp->ev[1 + o], st));
                        PYSIFT_CUDA_TRY(cudaStreamWaitEvent(side, sp->ev[1 + o], 0));
                    }
                }
                memset(&a, 0, sizeof(a));
                a.H = l.H[o];
                a.W = l.W[o];
                a.out_pitch = l.pitch[o];
                if (s == 0 && o > 0) {
                    const float* prev = at<float>(ws, l.off_pyr[o - 1]) + (size_t)S * l.H[o - 1] * l.pitch[o - 1];
                    a.in = prev;
                    a.in_pitch = l.pitch[o - 1];
                    a.step = 2;
                    a.copy0 = pyr;
                    a.copy0_r = pyr_r;
                } else {
                    a.in = pyr + (size_t)s * lev;
                    a.in_pitch = l.pitch[o];
                    a.step = 1;
                }
                a.out = pyr + (size_t)(s + 1) * lev;
                a.out_r = pyr_r ? pyr_r + (size_t)(s + 1) * lev : nullptr;
                int rc = launch_blur(a, cfg->blur_radius[2 + s], cfg->blur_weights[2 + s], s != S || !sp, ls);
                if (rc) return rc;
            }
        }
    }
    if (sp) {
        PYSIFT_CUDA_TRY(cudaEventRecord(sp->ev[PYSIFT_MAX_OCTAVES + 1], side));
        PYSIFT_CUDA_TRY(cudaStreamWaitEvent(st, sp->ev[PYSIFT_MAX_OCTAVES + 1], 0));
    }
    PYSIFT_STAGE(2);
    // A7/A8 (+ retry)
    static thread_local ExtArgs ea;
    static thread_local RefArgs ra;
    memset(&ea, 0, sizeof(ea));
    memset(&ra, 0, sizeof(ra));
    fill_oct_views(l, ws, true, ea.oct);
    fill_oct_views(l, ws, true, ra.oct);
    ea.n_oct = ra.n_oct = n_oct;
    ea.S = ra.S = S;
    ea.border = ra.border = cfg->border;
    ea.cap = ra.cap = cap;
    ea.cand = at<int4>(ws, l.off_cand);
    ra.cand = ea.cand;
    int mask_blocks = 0, row_blocks = 0;
    int row_off[PYSIFT_MAX_OCTAVES + 1];
    // Strips of 32 rows (6 % of the rows loaded twice) when they fill the
    // SMs' warps twice over, else shorter ones: a strip is a serial walk, and
    // a small image would wait for a few long ones.
    auto strips = [&](int rows) {
        long long n = 0;
        for (int o = 0; o < n_oct; ++o) n += (long long)ceil_div(l.H[o], rows) * ceil_div(l.W[o], EX_COLS);
        return n;
    };
    const int retry_blocks = num_sms() * 8;
    ea.rows = 32;
    while (ea.rows > 4 && strips(ea.rows) < 40LL * num_sms()) ea.rows /= 2;
    for (int o = 0; o < n_oct; ++o) {
        ea.blk_off[o] = mask_blocks;
        mask_blocks += ceil_div(ceil_div(l.H[o], ea.rows) * ceil_div(l.W[o], EX_COLS), EX_T / 32);
        row_off[o] = row_blocks;
        row_blocks += ceil_div(S * l.H[o], 8);
        ea.rowoff[o] = at<int>(ws, l.off_rowoff[o]);
        ea.wpr[o] = l.wpr[o];
    }
    ea.blk_off[n_oct] = mask_blocks;
    row_off[n_oct] = row_blocks;
    ra.edge_score = cfg->edge_score;
    ra.starvation_min = cfg->starvation_min;
    ra.rv_valid = at<int>(ws, l.off_rv_valid);
    ra.rv_ri = at<float>(ws, l.off_rv_ri);
    ra.rv_ci = at<float>(ws, l.off_rv_ci);
    ra.rv_si = at<int>(ws, l.off_rv_si);
    ra.rv_resp = at<float>(ws, l.off_rv_resp);
    ra.rf_ri = at<float>(ws, l.off_rf_ri);
    ra.rf_ci = at<float>(ws, l.off_rf_ci);
    ra.rf_si = at<int>(ws, l.off_rf_si);
    ra.rf_resp = at<float>(ws, l.off_rf_resp);
    const int refine_blocks = (int)std::min<long long>(ceil_div_ll((long long)n_oct * cap, 256), num_sms() * 8);
    for (int pass = 0; pass < 2; ++pass) {
        ea.thr_idx = ra.thr_idx = pass;
        ea.retry_mode = ra.retry_mode = pass;
        for (int o = 0; o < n_oct; ++o) {
            ea.mask[o] = at<uint32_t>(ws, l.off_mask[o] + pass * l.zero_bytes);
            ea.rowcnt[o] = at<int>(ws, l.off_rowcnt[o] + pass * l.zero_bytes);
        }
        // the retry's grid is small (its kernels loop), so that finding nothing
        // to do is cheap
        if (pass == 0) extrema_kernel(S)<<<mask_blocks, EX_T, 0, st>>>(ea, ctrl);
        else launch_chained(extrema_kernel(S), dim3(std::min(mask_blocks, retry_blocks)), EX_T, 0, st, ea, ctrl);
        PYSIFT_LAUNCH_CHECK("k_extrema_mask");
        if (pass == 0) PYSIFT_STAGE(3);
        launch_chained(k_rowscan, dim3(n_oct), 1024, 0, st, ea, ctrl);
        PYSIFT_LAUNCH_CHECK("k_rowscan");
        // k_scatter indexes blocks by (s, r) rows: reuse blk_off for its own table
        ExtArgs& sa = ea;
        int saved[PYSIFT_MAX_OCTAVES + 1];
        memcpy(saved, sa.blk_off, sizeof(saved));
        memcpy(sa.blk_off, row_off, sizeof(row_off));
        launch_chained(k_scatter, dim3(pass == 0 ? row_blocks : std::min(row_blocks, retry_blocks)), 256, 0, st, sa, ctrl);
        PYSIFT_LAUNCH_CHECK("k_scatter");
        memcpy(sa.blk_off, saved, sizeof(saved));
        launch_chained(k_refine, dim3(refine_blocks), 256, 0, st, ra, ctrl);
        PYSIFT_LAUNCH_CHECK("k_refine");
        launch_chained(k_refine_compact, dim3(n_oct), 1024, 0, st, ra, ctrl);
        PYSIFT_LAUNCH_CHECK("k_refine_compact");
    }
    // A9
    CapArgs ca;
    ca.n_oct = n_oct;
    ca.cap_cand = cap;
    ca.kp_cap = kcap;
    ca.rf_ri = ra.rf_ri;
    ca.rf_ci = ra.rf_ci;
    ca.rf_si = ra.rf_si;
    ca.rf_resp = ra.rf_resp;
    ca.kp_o = at<int>(ws, l.off_kp_o);
    ca.kp_si = at<int>(ws, l.off_kp_si);
    ca.kp_ri = at<float>(ws, l.off_kp_ri);
    ca.kp_ci = at<float>(ws, l.off_kp_ci);
    ca.kp_resp = at<float>(ws, l.off_kp_resp);
    ca.kp_tb = at<uint32_t>(ws, l.off_kp_tb);
    {
        PYSIFT_CUDA_TRY(
            cudaFuncSetAttribute(k_cap, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CAP_SMEM_BYTES));
        launch_chained(k_cap, dim3(1), CAP_T, CAP_SMEM_BYTES, st, ca, ctrl);
    }
    PYSIFT_LAUNCH_CHECK("k_cap");
    PYSIFT_STAGE(4);
    // A10
    static thread_local OriArgs oa;
    memset(&oa, 0, sizeof(oa));
    fill_oct_views(l, ws, true, oa.oct);
    for (int s = 0; s < PYSIFT_MAX_LEVELS; ++s) oa.ori_sigma[s] = cfg->ori_sigma[s];
    oa.kp_o = ca.kp_o;
    oa.kp_si = ca.kp_si;
    oa.kp_ri = ca.kp_ri;
    oa.kp_ci = ca.kp_ci;
    oa.ang = at<float>(ws, l.off_ang);
    oa.angcnt = at<int>(ws, l.off_angcnt);
    launch_chained(k_orientation, dim3(std::min(kcap, num_sms() * 5)), ORI_T, 0, st, oa, ctrl);
    PYSIFT_LAUNCH_CHECK("k_orientation");
    // expansion + keys + rank
    ExpArgs xa;
    memset(&xa, 0, sizeof(xa));
    xa.kp_o = ca.kp_o;
    xa.kp_si = ca.kp_si;
    xa.kp_ri = ca.kp_ri;
    xa.kp_ci = ca.kp_ci;
    xa.kp_tb = ca.kp_tb;
    xa.angcnt = oa.angcnt;
    xa.ent_kp = at<int>(ws, l.off_ent_kp);
    xa.ent_slot = at<int>(ws, l.off_ent_slot);
    xa.keys = at<uint4>(ws, l.off_keys);
    for (int o = 0; o < n_oct; ++o) xa.coord_scale[o] = (float)((double)(1 << o) * (l.doubled ? 0.5 : 1.0));
    xa.xy_cnt = bkt;
    xa.xy_bscale = (float)BR_NB / (float)W;
    xa.blk_cnt = at<int>(ws, l.off_xblk);
    const int exp_blocks = ceil_div(kcap, EXP_PER_BLOCK);
    launch_chained(k_expand_count, dim3(exp_blocks), EXP_T, 0, st, xa, ctrl);
    PYSIFT_LAUNCH_CHECK("k_expand_count");
    launch_chained(k_expand, dim3(exp_blocks), EXP_T, 0, st, xa, ctrl);
    PYSIFT_LAUNCH_CHECK("k_expand");
    int* rank = at<int>(ws, l.off_rank);
    const int br_blocks = std::max(1, std::min(ceil_div(4 * kcap, 128), num_sms() * 4));
    BRArgs bx{};
    bx.keys = xa.keys;
    bx.xy_bscale = xa.xy_bscale;
    bx.cnt = bkt;
    bx.off = bkt + BR_NB;
    bx.cursor = bkt + 2 * BR_NB;
    bx.members = at<int>(ws, l.off_members);
    bx.rank = rank;
    const int br_threads = 128;
    launch_chained(k_br_scan<0>, dim3(1), 1024, 0, st, bx, ctrl);
    PYSIFT_LAUNCH_CHECK("k_br_scan");
    launch_chained(k_br_scatter<0>, dim3(br_blocks), br_threads, 0, st, bx, ctrl);
    PYSIFT_LAUNCH_CHECK("k_br_scatter");
    launch_chained(k_br_rank<0>, dim3(br_blocks), br_threads, 0, st, bx, ctrl);
    PYSIFT_LAUNCH_CHECK("k_br_rank");
    PYSIFT_STAGE(5);
    // A11
    static thread_local DescArgs da;
    memset(&da, 0, sizeof(da));
    fill_oct_views(l, ws, true, da.oct);
    for (int s = 0; s < PYSIFT_MAX_LEVELS; ++s) da.desc_ph[s] = cfg->desc_ph[s];
    for (int o = 0; o < n_oct; ++o) {
        for (int s = 0; s < PYSIFT_MAX_LEVELS; ++s) da.kp_size[o][s] = cfg->kp_size[l.doubled ? 1 : 0][o][s];
        da.coord_scale[o] = xa.coord_scale[o];
    }
    da.n_dsp = cfg->dsp ? cfg->n_dsp : 0;
    for (int d = 0; d < 8; ++d) da.dsp_scales[d] = cfg->dsp_scales[d];
    da.rootsift = cfg->rootsift;
    da.kp_o = ca.kp_o;
    da.kp_si = ca.kp_si;
    da.kp_ri = ca.kp_ri;
    da.kp_ci = ca.kp_ci;
    da.kp_resp = ca.kp_resp;
    da.ang = oa.ang;
    da.ent_kp = xa.ent_kp;
    da.ent_slot = xa.ent_slot;
    da.rank = rank;
    da.split_tot = at<unsigned long long>(ws, l.off_split);
    da.split_cnt = reinterpret_cast<int*>(da.split_tot + 128 * split_entries(kcap));
    da.limit = cfg->output_limit;
    da.lrank = at<int>(ws, l.off_lrank);
    if (cfg->output_limit > 0) {
        float* row_resp = at<float>(ws, l.off_row_resp);
        BRArgs br{};
        br.row_resp = row_resp;
        br.limit = cfg->output_limit;
        br.cnt = bkt + 3 * BR_NB;
        br.off = bkt + 4 * BR_NB;
        br.cursor = bkt + 5 * BR_NB;
        br.members = at<int>(ws, l.off_members) + 4 * (size_t)kcap;
        br.rank = at<int>(ws, l.off_lrank);
        launch_chained(k_row_resp, dim3(br_blocks), br_threads, 0, st, (const int*)xa.ent_kp, (const float*)ca.kp_resp,
                       (const int*)rank, row_resp, br.cnt, ctrl);
        PYSIFT_LAUNCH_CHECK("k_row_resp");
        launch_chained(k_br_scan<1>, dim3(1), 1024, 0, st, br, ctrl);
        PYSIFT_LAUNCH_CHECK("k_br_scan");
        launch_chained(k_br_scatter<1>, dim3(br_blocks), br_threads, 0, st, br, ctrl);
        PYSIFT_LAUNCH_CHECK("k_br_scatter");
        launch_chained(k_br_rank<1>, dim3(br_blocks), br_threads, 0, st, br, ctrl);
        PYSIFT_LAUNCH_CHECK("k_br_rank");
    }
    da.out_kpts = kpts;
    da.out_resp = resp;
    da.out_oct = octv;
    da.out_desc = desc;
    da.n_oct = n_oct;
    da.doubled = l.doubled ? 1 : 0;
    da.stats = stats;
    launch_chained(k_descriptor, dim3(std::min(4 * kcap, num_sms() * DESC_OCC)), DESC_T, 0, st, da, ctrl);
    PYSIFT_LAUNCH_CHECK("k_descriptor");
    PYSIFT_STAGE(6);
    return PYSIFT_OK;
}

}  // namespace pysift

using namespace pysift;

extern "C" {

const char* pysift_last_error(void) { return g_last_error.c_str(); }

const char* pysift_b200_version(void) { return "pysift_b200 0.1.0 (sm_100a)"; }

size_t pysift_detect_config_size(void) { return sizeof(pysift_detect_config); }

int64_t pysift_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

void pysift_count_launches(int64_t n) { g_launches.fetch_add((long long)n, std::memory_order_relaxed); }

int pysift_detect_workspace_size(const pysift_detect_config* cfg, int32_t H, int32_t W, size_t* bytes) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(H > 0 && W > 0, "image size %dx%d must be positive", H, W);
    PYSIFT_CHECK_ARG(bytes != nullptr, "bytes is NULL");
    Layout l = make_layout(cfg, H, W);
    *bytes = l.total;
    return PYSIFT_OK;
}

int32_t pysift_detect_max_keypoints(const pysift_detect_config* cfg) {
    if (!cfg) return 0;
    return 4 * cfg->keypoint_cap;
}

int pysift_detect_workspace_view(const pysift_detect_config* cfg, int32_t H, int32_t W, int32_t what, int32_t octave,
                                 int32_t level, size_t* offset, int32_t* rows, int32_t* cols, int32_t* pitch_floats) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(H > 0 && W > 0, "image size %dx%d must be positive", H, W);
    PYSIFT_CHECK_ARG(offset && rows && cols && pitch_floats, "NULL output pointer");
    Layout l = make_layout(cfg, H, W);
    if (what == 0) {
        PYSIFT_CHECK_ARG(octave >= 0 && octave < l.n_oct && level >= 0 && level < l.L, "octave/level out of range");
        *offset = l.off_pyr_r[octave] + (size_t)level * l.H[octave] * l.pitch[octave] * sizeof(float);
        *rows = l.H[octave];
        *cols = l.W[octave];
        *pitch_floats = l.pitch[octave];
    } else if (what == 1) {
        *offset = l.off_base;
        *rows = l.H0;
        *cols = l.W0;
        *pitch_floats = l.pitch0;
    } else {
        set_error("unknown view %d", what);
        return PYSIFT_ERR_INVALID_ARG;
    }
    return PYSIFT_OK;
}

int pysift_detect_and_compute(const pysift_detect_config* cfg, const uint8_t* gray, int32_t H, int32_t W,
                              int64_t pitch_bytes, void* workspace, size_t workspace_bytes, float* kpts,
                              float* response, int32_t* octave, float* desc, int32_t max_out, int32_t* stats,
                              void* const* stage_events, pysift_stream_t stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    PYSIFT_CHECK_ARG(H > 0 && W > 0, "image size %dx%d must be positive", H, W);
    PYSIFT_CHECK_ARG(pitch_bytes >= W, "pitch %lld smaller than width %d", (long long)pitch_bytes, W);
    PYSIFT_CHECK_ARG(gray && workspace && kpts && response && octave && desc && stats, "NULL pointer argument");
    Layout l = make_layout(cfg, H, W);
    if (workspace_bytes < l.total) {
        set_error("workspace %zu bytes < required %zu", workspace_bytes, l.total);
        return PYSIFT_ERR_WORKSPACE;
    }
    if (max_out < 4 * cfg->keypoint_cap) {
        set_error("max_out %d < 4 * keypoint_cap (%d)", max_out, 4 * cfg->keypoint_cap);
        return PYSIFT_ERR_CAPACITY;
    }
    if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) {
        set_error("workspace must be 256-byte aligned");
        return PYSIFT_ERR_INVALID_ARG;
    }
    return run_detect(cfg, gray, H, W, pitch_bytes, workspace, l, kpts, response, octave, desc, stats,
                      stage_events, reinterpret_cast<cudaStream_t>(stream));
}

int pysift_gauss_blur(const float* in, int32_t in_pitch, float* out, int32_t out_pitch, int32_t H, int32_t W,
                      const float* weights, int32_t radius, pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(in && out && weights, "NULL pointer argument");
    PYSIFT_CHECK_ARG(H > 0 && W > 0 && in_pitch >= W && out_pitch >= W, "bad sizes");
    PYSIFT_CHECK_ARG(radius >= 0 && radius <= PYSIFT_MAX_RADIUS, "radius %d outside 0..%d", radius,
                     PYSIFT_MAX_RADIUS);
    return blur_level(in, in_pitch, 1, out, out_pitch, nullptr, H, W, weights, radius, false,
                      reinterpret_cast<cudaStream_t>(stream));
}

int pysift_set_blur_tile_rows(int32_t rows) {
    int v = -1;
    for (int k = 0; k < BLUR_NV; ++k)
        if (rows == BLUR_THS[k]) v = k;
    PYSIFT_CHECK_ARG(rows == 0 || v >= 0, "tile rows %d: 0 (automatic), 16, 32 or 40", rows);
    g_blur_forced.store(rows == 0 ? -1 : v, std::memory_order_relaxed);
    return PYSIFT_OK;
}

int pysift_blur_size_class(int32_t H, int32_t W) { return (H > 0 && W > 0) ? blur_size_class(H, W) : -1; }

int pysift_set_blur_tile_table(const int32_t* rows, int32_t n) {
    constexpr int N = (BLUR_PAIR_MAX_R + 1) * BLUR_SIZE_CLASSES;
    PYSIFT_CHECK_ARG(n == 0 || (rows && n == N), "the table has %d entries (0 clears it)", N);
    int v[N];
    for (int i = 0; i < n; ++i) {
        v[i] = -1;
        for (int k = 0; k < BLUR_NV; ++k)
            if (rows[i] == BLUR_THS[k]) v[i] = k;
        PYSIFT_CHECK_ARG(rows[i] == 0 || v[i] >= 0, "entry %d: tile rows %d: 0 (rule), 16, 32 or 40", i, rows[i]);
    }
    blur_table_init();
    for (int i = 0; i < N; ++i)
        g_blur_table[i / BLUR_SIZE_CLASSES][i % BLUR_SIZE_CLASSES].store(n ? v[i] : -1, std::memory_order_relaxed);
    return PYSIFT_OK;
}

int pysift_zoom2x_u8(const uint8_t* gray, int32_t H, int32_t W, int64_t pitch_bytes, int32_t fp16_round,
                     double* coef, float* out, int32_t out_pitch, pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(gray && coef && out, "NULL pointer argument");
    PYSIFT_CHECK_ARG(H > 0 && W > 0 && pitch_bytes >= W && out_pitch >= 2 * W, "bad sizes");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    return launch_zoom2x(gray, H, W, pitch_bytes, fp16_round, coef, out, out_pitch, st);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free variant of pysift_zoom2x_u8.
//
// Some callers cannot allocate device memory at the call site: for example a
// plugin loaded into a host application that owns the whole device heap and
// forbids cudaMalloc inside plugins, or code that runs under a fixed device
// memory budget with no allocator handle to pass in.  For them this entry
// point keeps the spline-coefficient scratch in a file-scope device array of
// PYSIFT_ZOOM2X_NOALLOC_MAX_PIXELS doubles (8 MiB), which every GPU that
// loads the library holds until the process exits.
//
// Host code cannot pass g_zoom2x_scratch to a kernel directly (in host code
// the name is a host-side stand-in, not a device address), so the device
// address is looked up with cudaGetSymbolAddress once per device, on the
// first call made with that device current, and cached.
// ---------------------------------------------------------------------------
namespace pysift {

static __device__ __align__(256) double g_zoom2x_scratch[PYSIFT_ZOOM2X_NOALLOC_MAX_PIXELS];

static int zoom2x_scratch_ptr(double** out) {
    constexpr int MAX_DEVICES = 64;
    static std::mutex mu;
    static double* ptrs[MAX_DEVICES] = {nullptr};
    int dev = 0;
    PYSIFT_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) {
        set_error("device ordinal %d not supported by the allocation-free entry point", dev);
        return PYSIFT_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!ptrs[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_zoom2x_scratch);
        if (e != cudaSuccess || p == nullptr) {
            set_error("cudaGetSymbolAddress(g_zoom2x_scratch) on device %d failed: %s", dev,
                      cudaGetErrorString(e));
            return PYSIFT_ERR_CUDA;
        }
        ptrs[dev] = static_cast<double*>(p);
    }
    *out = ptrs[dev];
    return PYSIFT_OK;
}

}  // namespace pysift

extern "C" int pysift_zoom2x_u8_noalloc(const uint8_t* gray, int32_t H, int32_t W, int64_t pitch_bytes,
                                        int32_t fp16_round, float* out, int32_t out_pitch,
                                        pysift_stream_t stream) {
    PYSIFT_CHECK_ARG(gray && out, "NULL pointer argument");
    PYSIFT_CHECK_ARG(H > 0 && W > 0 && pitch_bytes >= W && out_pitch >= 2 * W, "bad sizes");
    if ((int64_t)H * W > (int64_t)PYSIFT_ZOOM2X_NOALLOC_MAX_PIXELS) {
        set_error("pysift_zoom2x_u8_noalloc: %dx%d = %lld pixels exceeds the fixed scratch of %d pixels; "
                  "use pysift_zoom2x_u8 with caller-provided scratch",
                  H, W, (long long)H * W, (int)PYSIFT_ZOOM2X_NOALLOC_MAX_PIXELS);
        return PYSIFT_ERR_CAPACITY;
    }
    double* coef = nullptr;
    int rc = zoom2x_scratch_ptr(&coef);
    if (rc) return rc;
    // Every scratch element the kernels read is written earlier in this same
    // call (k_prefilter_cols fills all H*W coefficients), so nothing needs
    // clearing between calls.
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    return launch_zoom2x(gray, H, W, pitch_bytes, fp16_round, coef, out, out_pitch, st);
}
