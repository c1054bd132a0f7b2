// engine.cu — the B200 geodesic engine: host side, the C ABI (include/sirius_cuda.h)
// and the kernels around the tracer.
//
// Kernels here
//   flux_table_kernel     per-frame Page-Thorne flux tables of the mixed path.
//   sur_* kernels         surrogate-gated rendering (features, gate, compaction,
//                         shading, audit judgement).
//   beam_kernel           geodesic deviation around each pixel ray (beam.cuh).
//   metric_kernel         IMetric::evaluate for a batch of points.
//   dp45_step_kernel      one Geodesic::integrateStepRK45 attempt per state.
//   fma_peak_kernel       FP32/FP64 FMA-chain microbenchmark (roofline peak).
// The trace kernels themselves (tracer.cuh) are instantiated in
// trace_ks_mixed.cu, trace_ks_fp64.cu and trace_families.cu; the surrogate MLP
// and its training kernels in surrogate.cuh and train.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "tracer.cuh"
#include "surrogate.cuh"
#include "train.cuh"

using namespace sirius;

static_assert(sizeof(sirius_metric) == 80, "sirius_metric layout");
static_assert(sizeof(sirius_camera) == 64, "sirius_camera layout");
static_assert(sizeof(sirius_frame) == 176, "sirius_frame layout");
static_assert(sizeof(sirius_ray_result) == 256, "sirius_ray_result layout");
static_assert(sizeof(sirius_camera_ray) == 64, "sirius_camera_ray layout");
static_assert(sizeof(sirius_surrogate_config) == 40, "sirius_surrogate_config layout");
static_assert(sizeof(sirius_surrogate_stats) == 56, "sirius_surrogate_stats layout");
static_assert(sizeof(sirius_train_config) == 64, "sirius_train_config layout");
static_assert(sizeof(sirius_beam_result) == 32, "sirius_beam_result layout");

using namespace sirius::eng;

namespace {

// One block of kFluxN threads per frame.
__global__ void __launch_bounds__(kFluxN) flux_table_kernel(const FrameDev* frames, float* table) {
    __shared__ float node[kFluxN];
    const FrameDev& F = frames[blockIdx.x];
    const int j = threadIdx.x;
    const bool disk = F.m.family == SIRIUS_METRIC_KERR_SCHILD && F.has_horizon;
    const double span = F.disk_out - F.disk_in;
    float v = 0.f;
    if (disk) {
        const double u = double(j) / (kFluxN - 1);
        v = float(nt_flux(F.disk_in + span * u * u, F.a_star, F.isco, F.disk_in, F.disk_out));
    }
    node[j] = v;
    __syncthreads();
    float flag = 0.f;
    if (disk && j < kFluxN - 1) {
        const double x = j + 0.5, u = x / (kFluxN - 1);
        const double exact = nt_flux(F.disk_in + span * u * u, F.a_star, F.isco, F.disk_in, F.disk_out);
        if (fabs(flux_cubic(node, x) - exact) > 1e-6 * fabs(exact)) flag = 1.f;
    }
    float* t = table + size_t(blockIdx.x) * kFluxTable;
    t[j] = v;
    t[kFluxN + j] = flag;
}

constexpr int kDefaultMinBlocks = 2;       // up to 255 registers
constexpr int kDefaultMinBlocksMixed = 4;  // 128 registers: mixed DP45
constexpr int kDefaultMinBlocksFp64 = 3;   // 168 registers: FP64 DP45
constexpr int kDefaultRaysPerThread = 1;   // rays per thread of mixed DP45 over Kerr-Schild frames
// a one-frame trace into host memory of at least kPieceMinBlocks tiles runs as
// up to kMaxPieces launches of tile rows, each piece's rays copied to the host
// while the next pieces trace
constexpr int kMaxPieces = 8;
constexpr long long kPieceMinBlocks = 2048;

// A kernel specialised for one metric family carries only that family's
// right-hand side (a smaller loop body and register set); kAnyFamily
// dispatches per ray. The Kerr-Schild kernels come in every register budget,
// and for one-frame launches (uni) with the frame in the parameter bank.
TraceFn pick_kernel(bool mixed, int minb, int fam, bool symp, bool uni = false) {
    if (fam == SIRIUS_METRIC_KERR_SCHILD)
        return mixed ? pick_ks_mixed(minb, uni, symp) : pick_ks_fp64(minb, uni, symp);
    return pick_family(mixed, fam, symp);
}

// ---------------------------------------------------------------------------
// Surrogate-gated rendering: features and gate per pixel, the MLP on every
// pixel, shading from its outputs, then the integrator on the compacted list
// of gated (near-critical) and audit rays, which overwrite their pixels.
// ---------------------------------------------------------------------------
constexpr int kCurveN = 256;      // critical-curve points per frame, ordered by angle about its centre
constexpr double kInnerGateDefault = 2.75;  // inner-disk gate: r_1 < 2.75 r_in (2048^2 bench frame: L-inf 8.3e-3 of the peak; 1.07e-2 at 2.5)
constexpr int kCoarseStrideDefault = 8;    // inner-disk gate: 8 x 8 pixels per coarse cell
constexpr float kSurRScale = 15.f;   // MLP output 1: r_1 = 15 (1 + o_1)
constexpr float kSurHigher = 1e-3f;  // MLP output 3: higher-order intensity / 1e-3
constexpr float kEmptyLogit = -4.f;  // empty pixels: every neighbouring coarse cell's hit logit below this

struct SurFrameDev {
    double sin_o, theta_deg;      // camera Boyer-Lindquist polar angle
    float ac;                     // centre (alpha_c, 0) of the critical curve
    int kerr;                     // 1: Kerr frame (no charge, no Lambda) the MLP covers; 0: integrate every ray
    float ca[kCurveN], cb[kCurveN];
    // inner-disk gate: the frame's coarse cells (cw x ch, row-major from coarse_offset)
    long long coarse_offset;
    int cw, ch;
    float r1_max;                 // inner_gate * r_in (0: off)
};

// The inner-disk gate's coarse pass: the features of each coarse cell's centre
// pixel (stride s), cells of all frames concatenated.
__global__ void sur_coarse_gather_kernel(const FrameDev* frames, const SurFrameDev* sf, int n_frames, int stride,
                                         long long n_coarse, const float* feat, float* cfeat) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_coarse) return;
    int f = 0;
    while (f + 1 < n_frames && sf[f + 1].coarse_offset <= c) ++f;
    const SurFrameDev& S = sf[f];
    const FrameDev& F = frames[f];
    const long long cc = c - S.coarse_offset;
    const int cx = int(cc % S.cw), cy = int(cc / S.cw);
    const long long rows = F.n_rays / F.width;
    const int x = min(cx * stride + stride / 2, F.width - 1);
    const long long y = min((long long)cy * stride + stride / 2, rows - 1);
    const long long idx = F.ray_offset + y * F.width + x;
#pragma unroll
    for (int k = 0; k < 5; ++k) cfeat[c * 5 + k] = feat[idx * 5 + k];
}

__device__ __forceinline__ unsigned audit_hash(unsigned long long idx, unsigned seed) {
    unsigned long long z = idx * 0x9E3779B97F4A7C15ull + seed;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return unsigned((z ^ (z >> 31)) >> 32);
}

__device__ __forceinline__ float seg_dist2(float px, float py, float ax, float ay, float bx, float by) {
    const float ux = bx - ax, uy = by - ay, vx = px - ax, vy = py - ay;
    const float t = fminf(fmaxf((vx * ux + vy * uy) / fmaxf(ux * ux + uy * uy, 1e-20f), 0.f), 1.f);
    const float dx = vx - t * ux, dy = vy - t * uy;
    return dx * dx + dy * dy;
}

// features (a, inclination, alpha, beta, r_obs), normalised
__global__ void sur_features_kernel(const FrameDev* frames, const SurFrameDev* sf, int n_frames, long long total,
                                    float* feat) {
    // the metric and the Boyer-Lindquist radius at the camera, once per block for
    // the frame of its first pixel (a thread of another frame computes its own)
    __shared__ double g_cam[16], r_cam;
    __shared__ int f_cam;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x == 0) {
        const long long first = (long long)blockIdx.x * blockDim.x;
        const int f0 = n_frames > 1 ? find_frame(frames, n_frames, first) : 0;
        f_cam = (frames[f0].m.family == SIRIUS_METRIC_MORRIS_THORNE || frames[f0].observer != SIRIUS_OBSERVER_STATIC)
                    ? -1 : f0;
        if (f_cam >= 0) {
            double x[4];
            camera_position_ks(frames[f0], x);
            metric_g(frames[f0].m, x, g_cam);
            InvForm IF;
            inv_form(frames[f0].m, x, IF);
            r_cam = IF.r;
        }
    }
    __syncthreads();
    if (idx >= total) return;
    const int f = n_frames > 1 ? find_frame(frames, n_frames, idx) : 0;
    const FrameDev& F = frames[f];
    const SurFrameDev& S = sf[f];
    const long long pix = idx - F.ray_offset;
    double dir[4], x[4], p[4], r;
    camera_dir(F, int(pix % F.width), F.row0 + int(pix / F.width), dir);
    if (f == f_cam) {
        init_state_ks(F, dir, g_cam, x, p);
        r = r_cam;
    } else {
        init_state(F, dir, x, p);
        InvForm IF;
        inv_form(F.m, x, IF);
        r = IF.r;
    }
    // celestial coordinates from the ray's own constants of motion:
    // alpha = -L_z / (E sin theta_o), beta = p_theta / E
    const double E = -p[0], L = x[1] * p[2] - x[2] * p[1];
    const double ct = fmin(fmax(x[3] / r, -1.0), 1.0), st = sqrt(fmax(1.0 - ct * ct, 1e-30));
    const double pth = (ct / st) * (x[1] * p[1] + x[2] * p[2]) - r * st * p[3];
    float* o = feat + idx * 5;
    o[0] = float(2.0 * F.a_star - 1.0);
    o[1] = float((S.theta_deg - 47.0) / 42.0);
    o[2] = float(-L / (E * S.sin_o) / 20.0);
    o[3] = float(pth / E / 20.0);
    o[4] = float((F.cam_r - 110.0) / 90.0);
}

// gate per pixel from its celestial coordinates (features 2 and 3): 1 = within
// `band` of the critical curve (or a frame the MLP does not cover), 2 = audit,
// 0 = the MLP's pixel; and the rays to integrate counted per block and class
// (sur_scan_kernel and sur_scatter_kernel list every gated ray before every
// audit ray, each class in pixel order)
// The pixel of this thread in the gate and scatter kernels: in pixel order, or,
// for one frame whose width and row count are multiples of 16 (tile_w = its
// width), in 16 x 16 tiles of 256-thread blocks with 8 x 4 pixels per warp, so
// that the compacted list of gated rays, which follows this order, hands the
// integrator warps of neighbouring pixels (as the tiled one-frame launch does).
__device__ __forceinline__ long long sur_pixel(int tile_w) {
    if (tile_w <= 0) return (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int bpr = tile_w / 16, b = int(blockIdx.x), w = int(threadIdx.x >> 5), l = int(threadIdx.x & 31);
    const int x = (b % bpr) * 16 + (w & 1) * 8 + (l & 7);
    const int y = (b / bpr) * 16 + (w >> 1) * 4 + (l >> 3);
    return (long long)y * tile_w + x;
}

__global__ void sur_gate_kernel(const FrameDev* frames, const SurFrameDev* sf, int n_frames, long long total,
                                float band, unsigned audit_threshold, unsigned seed, const float* feat,
                                int stride, const float* cout, unsigned char* gate, unsigned* block_counts,
                                int tile_w, int empty_skip) {
    const long long idx = sur_pixel(tile_w);
    unsigned char g = 0;
    if (idx < total) {
        const int f = n_frames > 1 ? find_frame(frames, n_frames, idx) : 0;
        const SurFrameDev& S = sf[f];
        if (!S.kerr) {
            g = 1;
        } else {
            const float alpha = feat[idx * 5 + 2] * 20.f, beta = feat[idx * 5 + 3] * 20.f;
            const float dx = alpha - S.ac, dy = beta;
            const float phi = atan2f(dy, dx);
            const int j0 = int(floorf((phi + float(kPi)) * (kCurveN / (2.f * float(kPi)))));
            float d2 = 1e30f;
            for (int k = j0 - 6; k <= j0 + 6; ++k) {
                const int a = ((k % kCurveN) + kCurveN) % kCurveN, b = (a + 1) % kCurveN;
                d2 = fminf(d2, seg_dist2(alpha, beta, S.ca[a], S.cb[a], S.ca[b], S.cb[b]));
            }
            if (d2 < band * band) g = 1;
            // inner-disk gate: the coarse cell of the pixel or a neighbouring one
            // predicts a disk hit inside r1_max
            if (!g && S.r1_max > 0.f) {
                const FrameDev& F = frames[f];
                const long long pix = idx - F.ray_offset;
                const int cx = int(pix % F.width) / stride, cy = int(pix / F.width / stride);
                for (int dy = -1; dy <= 1 && !g; ++dy)
                    for (int dx2 = -1; dx2 <= 1; ++dx2) {
                        const int ux = cx + dx2, uy = cy + dy;
                        if (ux < 0 || uy < 0 || ux >= S.cw || uy >= S.ch) continue;
                        const float* o = cout + (S.coarse_offset + (long long)uy * S.cw + ux) * 4;
                        if (o[0] > 0.f && kSurRScale * (1.f + o[1]) < S.r1_max) { g = 1; break; }
                    }
            }
        }
        // audit rays come in runs of 32 consecutive pixels, so that they integrate as coherent warps
        if (!g && audit_hash((unsigned long long)idx >> 5, seed) < audit_threshold) g = 2;
        // empty: the pixel's coarse cell and its eight neighbours all predict no
        // disk crossing (a ray that never crosses the disk carries no light)
        if (!g && empty_skip && S.kerr && S.cw > 0) {
            const FrameDev& F = frames[f];
            const long long pix = idx - F.ray_offset;
            const int cx = int(pix % F.width) / stride, cy = int(pix / F.width / stride);
            bool empty = true;
            for (int dy = -1; dy <= 1 && empty; ++dy)
                for (int dx2 = -1; dx2 <= 1; ++dx2) {
                    const int ux = min(max(cx + dx2, 0), S.cw - 1), uy = min(max(cy + dy, 0), S.ch - 1);
                    if (cout[(S.coarse_offset + (long long)uy * S.cw + ux) * 4] > kEmptyLogit) { empty = false; break; }
                }
            if (empty) g = 3;
        }
        gate[idx] = g;
    }
    // per block: gated, audit and MLP-row counts (class k at block_counts[k * gridDim.x + block])
    __shared__ unsigned warp_counts[3][32];
    const unsigned m1 = __ballot_sync(kFull, g == 1);
    const unsigned m2 = __ballot_sync(kFull, g == 2);
    const unsigned m3 = __ballot_sync(kFull, idx < total && (g == 0 || g == 2));
    if ((threadIdx.x & 31) == 0) {
        warp_counts[0][threadIdx.x >> 5] = __popc(m1);
        warp_counts[1][threadIdx.x >> 5] = __popc(m2);
        warp_counts[2][threadIdx.x >> 5] = __popc(m3);
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        unsigned c = 0;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) c += warp_counts[threadIdx.x][w];
        block_counts[threadIdx.x * gridDim.x + blockIdx.x] = c;
    }
}

// Exclusive prefix sum of the per-block counts (one block of 1024 threads);
// block_counts[n_blocks] receives the total.
__global__ void sur_scan_kernel(unsigned* block_counts, int n_blocks) {
    __shared__ unsigned part[1024];
    const int t = threadIdx.x;
    const int per = (n_blocks + 1023) / 1024;
    const int b0 = t * per, b1 = min(b0 + per, n_blocks);
    unsigned sum = 0;
    for (int b = b0; b < b1; ++b) sum += block_counts[b];
    part[t] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {  // Hillis-Steele inclusive scan
        const unsigned v = t >= off ? part[t - off] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    unsigned run = t > 0 ? part[t - 1] : 0u;
    for (int b = b0; b < b1; ++b) {
        const unsigned c = block_counts[b];
        block_counts[b] = run;
        run += c;
    }
    if (t == 1023) block_counts[n_blocks] = part[1023];
}

// The list of rays to integrate (same blocking as the gate kernel): the gated
// rays in pixel order, kListSkip entries up to the next multiple of 32, then
// the audit rays in pixel order (so each audit run of 32 pixels fills one warp).
// block_offsets: class-1 offsets of the blocks, then their class-2 offsets.
__global__ void sur_scatter_kernel(const unsigned char* gate, long long total, const unsigned* block_offsets,
                                   unsigned* list, int tile_w, unsigned* mlp_rows) {
    __shared__ unsigned warp_base[3][32];
    const long long idx = sur_pixel(tile_w);
    const unsigned char g = idx < total ? gate[idx] : 0;
    const unsigned m1 = __ballot_sync(kFull, g == 1), m2 = __ballot_sync(kFull, g == 2);
    const unsigned m3 = __ballot_sync(kFull, idx < total && (g == 0 || g == 2));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        warp_base[0][warp] = __popc(m1);
        warp_base[1][warp] = __popc(m2);
        warp_base[2][warp] = __popc(m3);
    }
    __syncthreads();
    const unsigned n1 = block_offsets[gridDim.x], pad = (32u - (n1 & 31u)) & 31u;
    const unsigned n12 = block_offsets[2 * gridDim.x];  // the MLP rows' offsets start here
    if (blockIdx.x == 0 && threadIdx.x < pad) list[n1 + threadIdx.x] = kListSkip;
    if (threadIdx.x < 3) {
        unsigned run = block_offsets[threadIdx.x * gridDim.x + blockIdx.x] + (threadIdx.x == 1 ? pad : 0u) -
                       (threadIdx.x == 2 ? n12 : 0u);
        for (int w = 0; w < int(blockDim.x >> 5); ++w) {
            const unsigned c = warp_base[threadIdx.x][w];
            warp_base[threadIdx.x][w] = run;
            run += c;
        }
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
    if (g == 1) list[warp_base[0][warp] + __popc(m1 & below)] = unsigned(idx);
    if (g == 2) list[warp_base[1][warp] + __popc(m2 & below)] = unsigned(idx);
    if (mlp_rows && idx < total && (g == 0 || g == 2)) mlp_rows[warp_base[2][warp] + __popc(m3 & below)] = unsigned(idx);
}

// pixel intensity from the MLP outputs: hit logit, r_1, g_1, higher orders
// Pixels the integrator takes (gate != 0) get only the MLP copy: the
// integrator writes their image value.
__global__ void sur_shade_kernel(const FrameDev* frames, int n_frames, long long total, float* out,
                                 const unsigned char* gate, const float* flux, float* image, float* image_mlp) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const unsigned char g = gate[idx];
    if (g == 3) {  // empty: no disk crossing predicted around it, and no MLP outputs
        image[idx] = 0.f;
        if (image_mlp) image_mlp[idx] = 0.f;
        return;
    }
    if (g == 1 && !image_mlp) return;  // the integrator writes it
    const int f = n_frames > 1 ? find_frame(frames, n_frames, idx) : 0;
    const FrameDev& F = frames[f];
    const float4 o = reinterpret_cast<const float4*>(out)[idx];
    double I = 0.0;
    if (o.x > 0.f) {
        const double r1 = fmin(fmax(double(kSurRScale) * (1.0 + double(o.y)), F.disk_in), F.disk_out);
        const double g1 = fmax(double(o.z), 0.0);
        I = g1 * g1 * g1 * g1 * flux_lookup(flux + size_t(F.flux_slot) * kFluxTable, F, r1);
    }
    I += fmax(double(o.w), 0.0) * double(kSurHigher);
    if (g == 0) image[idx] = float(I);
    if (g == 2) out[idx * 4] = float(I);  // kept for the audit (the outputs are consumed)
    if (image_mlp) image_mlp[idx] = float(I);
}

// The audit's judgement: over the audit pixels, sum |I_mlp - I|, sum I, max
// |I_mlp - I|, max I and their count (acc[0..4], zero on entry; the maxima as
// the bits of non-negative floats).
__global__ void sur_audit_kernel(const unsigned char* gate, const float* image, const float* out, long long total,
                                 float* acc) {
    __shared__ float red[4][32];
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float d = 0.f, v = 0.f, c = 0.f;
    if (idx < total && gate[idx] == 2) {
        v = image[idx];
        d = fabsf(out[idx * 4] - v);
        c = 1.f;
    }
    float sd = d, sv = v, md = d, mv = v, sc = c;
    for (int o = 16; o >= 1; o >>= 1) {
        sd += __shfl_xor_sync(kFull, sd, o);
        sv += __shfl_xor_sync(kFull, sv, o);
        sc += __shfl_xor_sync(kFull, sc, o);
        md = fmaxf(md, __shfl_xor_sync(kFull, md, o));
        mv = fmaxf(mv, __shfl_xor_sync(kFull, mv, o));
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        red[0][warp] = sd;
        red[1][warp] = sv;
        red[2][warp] = sc;
        red[3][warp] = md;
        red[0][16 + warp] = mv;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.f, b = 0.f, k = 0.f, m1 = 0.f, m2 = 0.f;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) {
            a += red[0][w];
            b += red[1][w];
            k += red[2][w];
            m1 = fmaxf(m1, red[3][w]);
            m2 = fmaxf(m2, red[0][16 + w]);
        }
        if (k > 0.f) {
            atomicAdd(acc, a);
            atomicAdd(acc + 1, b);
            atomicMax(reinterpret_cast<int*>(acc + 2), __float_as_int(m1));
            atomicMax(reinterpret_cast<int*>(acc + 3), __float_as_int(m2));
            atomicAdd(acc + 4, k);
        }
    }
}

#include "beam.cuh"

// multi-sample passes: sum += pass (the first pass copies), then out = sum * scale
__global__ void pass_accumulate_kernel(const float* pass, float* sum, long long n, int first) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sum[i] = first ? pass[i] : sum[i] + pass[i];
}
__global__ void pass_scale_kernel(float* v, long long n, float scale) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] *= scale;
}

__global__ void metric_kernel(MetricDev m, const double* pos, long long n, int fp32, double* g, double* dg) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (fp32) {
        float x[4], gg[16], dd[64];
        for (int j = 0; j < 4; ++j) x[j] = float(pos[4 * i + j]);
        metric_full<float>(m, x, gg, dd);
        for (int j = 0; j < 16; ++j) g[16 * i + j] = gg[j];
        for (int j = 0; j < 64; ++j) dg[64 * i + j] = dd[j];
    } else {
        double x[4], gg[16], dd[64];
        for (int j = 0; j < 4; ++j) x[j] = pos[4 * i + j];
        metric_full<double>(m, x, gg, dd);
        for (int j = 0; j < 16; ++j) g[16 * i + j] = gg[j];
        for (int j = 0; j < 64; ++j) dg[64 * i + j] = dd[j];
    }
}

__global__ void dp45_step_kernel(MetricDev m, CfgDev c, double* state, double* h, int* accepted, double* err,
                                 long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x[4], p[4], k1[8], xn[4], pn[4], k7[8];
    for (int j = 0; j < 4; ++j) { x[j] = state[8 * i + j]; p[j] = state[8 * i + 4 + j]; }
    rhs<double>(m, x, p, k1, k1 + 4);
    const double e = dp45_attempt<double>(m, c, x, p, h[i], k1, xn, pn, k7);
    err[i] = e;
    accepted[i] = e <= 1.0 ? 1 : 0;
    if (e <= 1.0)
        for (int j = 0; j < 4; ++j) { state[8 * i + j] = xn[j]; state[8 * i + 4 + j] = pn[j]; }
    h[i] = optimal_step(h[i], e, c);
}

// FMA-chain peak: 8 independent chains per thread, ITER iterations each.
template <class T>
__global__ void fma_peak_kernel(T* out, int iters, T seed) {
    T a0 = seed + T(threadIdx.x), a1 = a0 + T(1), a2 = a0 + T(2), a3 = a0 + T(3);
    T a4 = a0 + T(4), a5 = a0 + T(5), a6 = a0 + T(6), a7 = a0 + T(7);
    const T b = T(0.9999), c = T(1e-7);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
            a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
        }
    }
    const T s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == T(-12345.678)) out[0] = s;  // keeps the chains alive
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Device scratch of one launch: the frame descriptors, the queue cursor and
// counters ([0] cursor, [1..3] counters, [4] launch start), the status word and
// room for the per-frame disk flux tables (kFluxTable floats per frame).
struct LaunchScratch {
    const FrameDev* frames;
    unsigned long long* queue;
    int* status;
    float* flux;
};

struct TrainState;

struct Handle {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    sirius_trace_config cfg{};
    bool configured = false;
    std::string last_error;
    FrameDev* d_frames = nullptr;
    size_t frames_cap = 0;
    sirius_ray_result* d_results = nullptr;
    size_t results_cap = 0;
    float* d_image = nullptr;
    size_t image_cap = 0;
    float* d_spectra = nullptr;
    size_t spectra_cap = 0;
    float* d_flux = nullptr;  // per-frame disk flux tables of the mixed path
    size_t flux_cap = 0;
    sirius_camera_ray* d_rays = nullptr;
    size_t rays_cap = 0;
    unsigned long long* d_queue = nullptr;  // [0] cursor, [1..3] counters
    int* d_status = nullptr;
    cudaEvent_t ev[4] = {};
    sirius_launch_stats stats{};
    // a device-entry launch whose statistics are read on the next sirius_cuda_last_stats
    bool pending = false;
    cudaStream_t pending_stream = nullptr;
    long long pending_total = 0;
    int family_mask = 0;  // bit f: a frame of the last upload is of class f (FrameDev::cls)
    FrameDev frame0{};    // the first frame of the last upload (a one-frame launch's parameter copy)
    std::vector<FrameDev> frames_host;  // the last upload's descriptors (multi-sample passes)
    std::vector<FrameDev> pass_frames_host;  // ... with each pass's sub-pixel offset
    FrameDev* d_pass_frames = nullptr;
    size_t pass_frames_cap = 0;
    // sirius_cuda_prepare_frames: the prepared launch's own scratch (descriptors,
    // queue and counter words, status word, flux tables), released only by the
    // next prepare or by destroy, so a captured graph's pointers stay valid
    unsigned char* d_prep = nullptr;
    LaunchScratch prep{};
    FrameDev prep_frame0{};
    int prep_n_frames = 0, prep_family_mask = 0;
    long long prep_total = 0;
    float* d_pass_image = nullptr;      // multi-sample: one pass's image and spectra, and their sums
    float* d_pass_spectra = nullptr;
    size_t pass_cap = 0;
    unsigned char* d_surrogate = nullptr;  // packed surrogate weight image (surrogate::kImageBytes)
    int* d_sur_err = nullptr;  // [0] the MLP kernel's error flag, [2..3] its tile counter, [8..12] the audit's sums and maxima
    bool sur_failed = false;   // the last call's MLP launches ended with an error: flag and counter start over
    unsigned char* d_tmp = nullptr;        // inputs and outputs of the calls on host buffers (beams, metric, steps)
    size_t tmp_cap = 0;
    // surrogate-gated rendering scratch
    SurFrameDev* d_sur_frames = nullptr;
    SurFrameDev* h_sur_frames = nullptr;  // pinned staging: per-frame basics, then with the curves
    size_t h_sur_frames_cap = 0;
    unsigned* h_list_len = nullptr;       // pinned: gated count, gated + audit count, + MLP rows
    size_t sur_frames_cap = 0;
    float* d_feat = nullptr;
    size_t feat_cap = 0;
    float* d_mlp_out = nullptr;
    size_t mlp_out_cap = 0;
    unsigned* d_list = nullptr;
    size_t list_cap = 0;
    float* d_coarse_feat = nullptr;  // the inner-disk gate's coarse features and MLP outputs
    size_t coarse_feat_cap = 0;
    float* d_coarse_out = nullptr;
    size_t coarse_out_cap = 0;
    long long last_coarse = 0;
    unsigned char* d_gate = nullptr;
    size_t gate_cap = 0;
    unsigned* d_block_counts = nullptr;  // per-block gated, audit and MLP-row counts, then offsets
    unsigned* d_mlp_rows = nullptr;      // pixels the per-pixel MLP evaluates (when empty pixels are skipped)
    int2* d_blocks = nullptr;            // a batch launch's per-frame block table
    size_t blocks_cap = 0;
    size_t mlp_rows_cap = 0;
    bool last_empty_skip = false;        // the last gate launch listed MLP rows (empty pixels skipped)
    size_t block_counts_cap = 0;
    cudaEvent_t sev[5] = {};
    // surrogate rendering: the gated trace (high priority) and the MLP (low priority)
    cudaStream_t sur_stream[2] = {};
    cudaEvent_t fev[4] = {};  // trace done, MLP done, shade done, join
    TrainState* train = nullptr;  // surrogate training state (sirius_cuda_train_init)
    // a one-frame trace into host memory in row pieces: the streams of pieces
    // 1.. (piece 0 runs on the caller's stream); events: [0] fork, [1 + k] piece k
    // traced, [1 + kMaxPieces + k] piece k copied to the host
    cudaStream_t piece_stream[kMaxPieces - 1] = {};
    cudaEvent_t piece_ev[2 * kMaxPieces + 1] = {};
};

// Outputs of a one-frame trace in host memory (the host entry point); done: the
// launch copied them itself, piece by piece, and the stream it was given is
// ordered after the copies.
struct HostOut {
    sirius_ray_result* results;
    float* image;
    float* spectra;
    int nb;
    bool done;
};


int fail(Handle* h, int code, const std::string& msg) {
    if (h) h->last_error = msg;
    cudaGetLastError();  // reported here: the check of the next launch must not find it
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return fail(H, e_ == cudaErrorMemoryAllocation ? SIRIUS_ERR_OUT_OF_MEMORY : SIRIUS_ERR_CUDA, \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                  \
    } while (0)

template <class T>
int ensure(Handle* H, T*& ptr, size_t& cap, size_t count) {
    if (count <= cap && ptr) return SIRIUS_OK;
    if (ptr) CK(cudaFree(ptr));
    ptr = nullptr;
    cap = 0;
    size_t n = std::max<size_t>(count, 1);
    CK(cudaMalloc((void**)&ptr, n * sizeof(T)));
    cap = n;
    return SIRIUS_OK;
}

// The workspace of a call on host buffers (beams, metric, steps), kept for the next call while it
// is at most kTmpKeep (a beam map of 1024^2 and less): a larger one is given back when the call ends.
constexpr size_t kTmpKeep = size_t(64) << 20;
struct TmpGuard {
    Handle* H;
    explicit TmpGuard(Handle* h) : H(h) {}
    TmpGuard(const TmpGuard&) = delete;
    TmpGuard& operator=(const TmpGuard&) = delete;
    ~TmpGuard() {
        if (H->tmp_cap <= kTmpKeep) return;
        cudaFree(H->d_tmp);  // (waits for the device)
        H->d_tmp = nullptr;
        H->tmp_cap = 0;
    }
};

double isco_host(double a_star) {
    const double a = std::min(std::fabs(a_star), 1.0);
    const double Z1 = 1 + std::cbrt(1 - a * a) * (std::cbrt(1 + a) + std::cbrt(1 - a));
    const double Z2 = std::sqrt(3 * a * a + Z1 * Z1);
    return a_star >= 0 ? 3 + Z2 - std::sqrt((3 - Z1) * (3 + Z1 + 2 * Z2))
                       : 3 + Z2 + std::sqrt((3 - Z1) * (3 + Z1 + 2 * Z2));
}

MetricDev make_metric(const sirius_metric& s) { return metric_dev(s); }

// Rays of a frame: its row window (row_count rows), or the whole image.
long long frame_rays(const sirius_frame& f) {
    return (long long)f.camera.width * (f.row_count > 0 ? f.row_count : f.camera.height);
}

// The zero-angular-momentum observer needs a Kerr-Newman metric (Kerr-Schild
// family, Lambda = 0) and a camera outside the outer horizon, off the axis.
int validate_observer(Handle* H, const sirius_frame& f) {
    const sirius_camera& c = f.camera;
    if (c.observer == SIRIUS_OBSERVER_STATIC) return SIRIUS_OK;
    if (c.observer != SIRIUS_OBSERVER_ZAMO) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "unknown camera observer");
    const sirius_metric& m = f.metric;
    if (m.family != SIRIUS_METRIC_KERR_SCHILD || std::fabs(m.Lambda) > 1e-15)
        return fail(H, SIRIUS_ERR_UNSUPPORTED, "the ZAMO observer needs a Kerr-Schild metric with Lambda = 0");
    const double d = m.M * m.M - m.a * m.a - m.Q * m.Q;
    const double rp = d >= 0.0 ? m.M + std::sqrt(d) : 0.0;
    if (!(c.r > rp) || !(c.r * c.r - 2.0 * m.M * c.r + m.a * m.a + m.Q * m.Q > 0.0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "the ZAMO observer must sit outside the outer horizon");
    return SIRIUS_OK;
}

int validate_metric(Handle* H, const sirius_metric& m) {
    if (m.family < 0 || m.family > 2) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "unknown metric family");
    if (!std::isfinite(m.M) || !std::isfinite(m.a) || !std::isfinite(m.Q) || !std::isfinite(m.Lambda))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "non-finite metric parameter");
    if (m.family == SIRIUS_METRIC_MORRIS_THORNE && !(m.b0 > 0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "Morris-Thorne throat radius must be > 0");
    if (m.family == SIRIUS_METRIC_ALCUBIERRE && !(m.sigma > 0 && m.R > 0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "Alcubierre sigma and R must be > 0");
    return SIRIUS_OK;
}

// A frame's camera, projection, observer and row window.
int validate_frame(Handle* H, const sirius_frame& f) {
    int rc = validate_metric(H, f.metric);
    if (rc != SIRIUS_OK) return rc;
    if (f.camera.width <= 0 || f.camera.height <= 0 || !(f.camera.r > 0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "camera needs width, height > 0 and r > 0");
    if (f.camera.projection != SIRIUS_CAMERA_PINHOLE && f.camera.projection != SIRIUS_CAMERA_EQUIRECTANGULAR)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "unknown camera projection");
    if (f.row_count < 0 || f.row_begin < 0 || (f.row_count == 0 && f.row_begin != 0) ||
        (long long)f.row_begin + f.row_count > f.camera.height)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT,
                    "row window must satisfy 0 <= row_begin, row_begin + row_count <= height (row_count 0: the whole frame)");
    return validate_observer(H, f);
}

// The zero-angular-momentum observer at Boyer-Lindquist (r, theta, phi) of a
// Kerr-Newman metric (Bardeen 1972; the FIDO of RDOP002A.cu:2528-2604):
//   rho^2 = r^2 + a^2 cos^2, Delta = r^2 - 2 M r + a^2 + Q^2,
//   Sigma^2 = (r^2 + a^2)^2 - a^2 Delta sin^2, alpha = rho sqrt(Delta) / Sigma,
//   omega = a (2 M r - Q^2) / Sigma^2, varpi = Sigma sin / rho;
//   e_(t) = (d_t + omega d_phi) / alpha, e_(r) = sqrt(Delta) / rho d_r,
//   e_(theta) = d_theta / rho, e_(phi) = d_phi / varpi.
// Boyer-Lindquist to Kerr-Schild: dt' = dt + (2 M r - Q^2) / Delta dr,
// dphi' = dphi + a / Delta dr, x = (r cos phi' - a sin phi') sin, y = (r sin phi'
// + a cos phi') sin, z = r cos (the form whose null vector is l = (1, (r x + a y)
// / (r^2 + a^2), (r y - a x) / (r^2 + a^2), z / r)). phi' = phi - atan2(a, r)
// puts the camera at x = sqrt(r^2 + a^2) sin cos(phi), the oblate map of
// PHCT002A.h:149-169. The tetrad's Kerr-Schild components are J e with J the
// Jacobian d(t', x, y, z) / d(t, r, theta, phi) at the camera.
static void zamo_frame(const sirius_metric& m, double t, double r, double th, double ph, FrameDev& F) {
    const double M = m.M, a = m.a, Q2 = m.Q * m.Q;
    const double st = std::sin(th), ct = std::cos(th);
    const double rho2 = r * r + a * a * ct * ct, rho = std::sqrt(rho2);
    const double Delta = r * r - 2.0 * M * r + a * a + Q2;
    const double Sig2 = (r * r + a * a) * (r * r + a * a) - a * a * Delta * st * st, Sig = std::sqrt(Sig2);
    const double alpha = rho * std::sqrt(Delta) / Sig, omega = a * (2.0 * M * r - Q2) / Sig2;
    const double varpi = Sig * st / rho;
    const double eb[4][4] = {{1.0 / alpha, 0.0, 0.0, omega / alpha},
                             {0.0, std::sqrt(Delta) / rho, 0.0, 0.0},
                             {0.0, 0.0, 1.0 / rho, 0.0},
                             {0.0, 0.0, 0.0, 1.0 / varpi}};
    const double pb = ph - std::atan2(a, r), cp = std::cos(pb), sp = std::sin(pb);
    const double dpb = a / Delta;
    double J[4][4] = {};
    J[0][0] = 1.0;
    J[0][1] = (2.0 * M * r - Q2) / Delta;
    J[1][1] = (cp + (-r * sp - a * cp) * dpb) * st;
    J[1][2] = (r * cp - a * sp) * ct;
    J[1][3] = (-r * sp - a * cp) * st;
    J[2][1] = (sp + (r * cp - a * sp) * dpb) * st;
    J[2][2] = (r * sp + a * cp) * ct;
    J[2][3] = (r * cp - a * sp) * st;
    J[3][1] = ct;
    J[3][2] = -r * st;
    F.zx[0] = t;
    F.zx[1] = (r * cp - a * sp) * st;
    F.zx[2] = (r * sp + a * cp) * st;
    F.zx[3] = r * ct;
    for (int i = 0; i < 4; ++i)
        for (int mu = 0; mu < 4; ++mu) {
            double s = 0.0;
            for (int nu = 0; nu < 4; ++nu) s += J[mu][nu] * eb[i][nu];
            F.ze[4 * i + mu] = s;
        }
}

FrameDev make_frame(const sirius_frame& f, const sirius_trace_config& c) {
    FrameDev F{};
    F.m = make_metric(f.metric);
    F.ray_offset = f.ray_offset;
    F.width = f.camera.width;
    F.height = f.camera.height;
    F.row0 = f.row_count > 0 ? f.row_begin : 0;
    F.n_rays = frame_rays(f);
    F.projection = f.camera.projection;
    // camera (CameraConfig, CMBS001A.h:37-58); theta clamp of initializeLightray (GTRC001A.cpp:25)
    const double th = std::clamp(f.camera.theta, 0.01, kPi - 0.01);
    F.cam_t = f.camera.t; F.cam_r = f.camera.r; F.cam_th = th; F.cam_ph = f.camera.phi;
    F.cam_st = std::sin(th); F.cam_ct = std::cos(th); F.cam_sp = std::sin(f.camera.phi); F.cam_cp = std::cos(f.camera.phi);
    F.aspect = float(f.camera.width) / float(f.camera.height);
    F.tan_half_fov = std::tan(f.camera.fov * float(kPi) / 360.0f);
    F.cY = std::cos(f.camera.yaw); F.sY = std::sin(f.camera.yaw);
    F.cP = std::cos(f.camera.pitch); F.sP = std::sin(f.camera.pitch);
    F.cR = std::cos(f.camera.roll); F.sR = std::sin(f.camera.roll);
    const sirius_metric& m = f.metric;
    const double a_star = m.M != 0 ? m.a / m.M : 0.0;
    F.a_star = a_star;
    F.isco = isco_host(a_star) * m.M;
    F.disk_in = f.disk_inner > 0 ? f.disk_inner : F.isco;
    F.disk_out = f.disk_outer;
    const double d = m.M * m.M - m.a * m.a - m.Q * m.Q;
    F.has_horizon = (m.family == SIRIUS_METRIC_KERR_SCHILD && d >= 0 && m.M > 0) ? 1 : 0;
    const double rp = F.has_horizon ? m.M + std::sqrt(d) : -1.0;
    F.r_hor = F.has_horizon ? rp * c.horizon_factor : -1.0;
    F.r_plus = rp;
    // (r is held at 1e-5; without mass and charge the metric is flat and both forms are zero there)
    const bool ring = m.family == SIRIUS_METRIC_KERR_SCHILD && (m.M != 0.0 || m.Q != 0.0) && !(F.r_hor > 1e-3);
    F.cls = ring ? kClassRing : m.family;
    // the radial-potential gate applies to Kerr-Newman frames (separable: no Lambda term)
    F.gate = (F.has_horizon && std::fabs(m.Lambda) <= 1e-15) ? 1 : 0;
    const double aM = std::clamp(a_star, -0.998, 0.998);
    F.r_ph_pro = 2.0 * m.M * (1.0 + std::cos((2.0 / 3.0) * std::acos(std::clamp(-aM, -1.0, 1.0))));
    const double r_ph_retro = 2.0 * m.M * (1.0 + std::cos((2.0 / 3.0) * std::acos(std::clamp(std::fabs(a_star), -1.0, 1.0))));
    if (m.family == SIRIUS_METRIC_KERR_SCHILD)
        F.island_r = std::max(c.island_factor * r_ph_retro, 2.0 * std::max(rp, 0.0));
    else if (m.family == SIRIUS_METRIC_MORRIS_THORNE)
        F.island_r = c.island_factor * 3.0 * m.b0;
    else
        F.island_r = c.island_factor * (m.R + 3.0 / std::max(m.sigma, 1e-6));
    // static observer at the camera: sqrt(-g_tt) (KS family g_tt = -1 + H - Lambda R^2/3)
    double gtt = -1.0;
    if (m.family == SIRIUS_METRIC_KERR_SCHILD) {
        const double x = f.camera.r * F.cam_st * F.cam_cp, y = f.camera.r * F.cam_st * F.cam_sp, z = f.camera.r * F.cam_ct;
        const double R2 = x * x + y * y + z * z, Rm2 = R2 - m.a * m.a;
        const double sd = std::sqrt(std::max(Rm2 * Rm2 + 4.0 * m.a * m.a * z * z, 1e-20));
        const double r2 = std::max(0.5 * (Rm2 + sd), 1e-10), r = std::sqrt(r2);
        const double H = (2.0 * m.M * r - m.Q * m.Q) * r2 / (r2 * r2 + m.a * m.a * z * z);
        gtt = -1.0 + H - (std::fabs(m.Lambda) > 1e-15 ? m.Lambda * R2 / 3.0 : 0.0);
    } else if (m.family == SIRIUS_METRIC_MORRIS_THORNE) {
        gtt = -std::exp(2.0 * m.Phi0);
    } else {
        const double rs = std::max(f.camera.r, 1e-10);
        const double fs = (std::tanh(m.sigma * (rs + m.R)) - std::tanh(m.sigma * (rs - m.R))) / (2.0 * std::tanh(m.sigma * m.R));
        gtt = -(1.0 - m.vs * m.vs * fs * fs);
    }
    F.sqrt_m_gtt_cam = std::sqrt(std::max(-gtt, 1e-30));
    F.fsqrt_m_gtt_cam = float(F.sqrt_m_gtt_cam);
    F.fdisk_in = float(F.disk_in);
    F.fdisk_out = float(F.disk_out);
    F.fr_ph_pro = float(F.r_ph_pro);
    F.observer = f.camera.observer;
    F.sub_u = 0.5f;
    F.sub_v = 0.5f;
    if (F.observer == SIRIUS_OBSERVER_ZAMO) zamo_frame(m, f.camera.t, f.camera.r, th, f.camera.phi, F);
    return F;
}

CfgDev make_cfg(const sirius_trace_config& c) {
    CfgDev d{};
    // (a scale below 1e-300 has no reciprocal in the kernels' arithmetic)
    d.atol = std::max(c.abs_tolerance, 1e-300); d.rtol = c.rel_tolerance; d.hmin = c.min_step; d.hmax = c.max_step;
    d.h0 = c.initial_step; d.safety = c.safety_factor; d.grow = c.step_grow_max; d.shrink = c.step_shrink_min;
    d.escape_r = c.escape_radius; d.decay = c.crossing_weight_decay;
    d.max_steps = c.max_steps; d.enable_disk = c.enable_disk; d.enable_vol = c.enable_volumetric;
    d.nbins = c.enable_volumetric ? std::min(c.n_bins, SIRIUS_MAX_BINS) : 0;
    d.vol_sub = c.vol_substeps; d.proj_period = c.projection_period; d.spiral = c.spiral_check; d.compat = c.compat;
    d.vol_j0 = c.vol_j0; d.vol_aoj = c.vol_alpha_over_j; d.vol_hz = c.vol_height_ratio; d.vol_s = c.vol_spectral_index;
    d.integrator = c.integrator; d.symp_order = c.symplectic_order; d.symp_step = c.symplectic_step;
    d.crit_band = c.critical_band;
    d.fatol = float(d.atol); d.frtol = float(d.rtol); d.fsafety = float(d.safety); d.fgrow = float(d.grow);
    d.fshrink = float(d.shrink); d.fvol_j0 = float(d.vol_j0); d.fvol_aoj = float(d.vol_aoj);
    d.fvol_hz = float(d.vol_hz); d.fvol_s = float(d.vol_s);
    d.npair = (d.nbins + 1) / 2;
    d.nu_desc = c.vol_spectral_index >= 0.0 ? 1 : 0;
    for (int b = 0; b < d.nbins; ++b) {
        const double nu = d.nbins == 1 ? c.nu_min : c.nu_min * std::pow(c.nu_max / c.nu_min, double(b) / (d.nbins - 1));
        // dtau_b = dtau nu_b^-s, applied as 2^(-dtau_b / ln 2)
        const float w = float(-std::pow(nu, -c.vol_spectral_index) / std::log(2.0));
        if (b & 1) d.nu_l2[b / 2].y = w;
        else d.nu_l2[b / 2] = make_float2(w, 0.f);
    }
    return d;
}

int validate_config(Handle* H, const sirius_trace_config& c) {
    if (!(c.abs_tolerance > 0) || !(c.rel_tolerance >= 0)) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "tolerances must be > 0");
    if (!(c.min_step > 0) || !(c.max_step >= c.min_step) || !(c.initial_step > 0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "step limits must satisfy 0 < min_step <= max_step, initial_step > 0");
    if (c.max_steps <= 0) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "max_steps must be > 0");
    if (c.samples_per_pixel < 0 || c.samples_per_pixel > 4096)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "samples_per_pixel must be in 0..4096");
    if (c.enable_volumetric && (c.n_bins <= 0 || c.n_bins > SIRIUS_MAX_BINS))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "n_bins must be in 1..32 when volumetric transfer is on");
    if (c.enable_volumetric && !(c.nu_min > 0 && c.nu_max >= c.nu_min && c.vol_alpha_over_j > 0 && c.vol_height_ratio > 0))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "invalid volumetric parameters");
    if (c.precision != SIRIUS_PRECISION_FP64 && c.precision != SIRIUS_PRECISION_MIXED)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "unknown precision mode");
    if (c.integrator != SIRIUS_INTEGRATOR_DP45 && c.integrator != SIRIUS_INTEGRATOR_SYMPLECTIC)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "unknown integrator");
    if (c.integrator == SIRIUS_INTEGRATOR_SYMPLECTIC &&
        (!(c.symplectic_step > 0) || (c.symplectic_order != 4 && c.symplectic_order != 6 && c.symplectic_order != 8)))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "symplectic_step must be > 0 and symplectic_order 4, 6 or 8");
    if (c.compat) return fail(H, SIRIUS_ERR_UNSUPPORTED, "reference-compatible mode is not available on the GPU path");
    if (c.block_size != 0 && c.block_size != 32 && c.block_size != 64 && c.block_size != 128)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "block_size must be 0, 32, 64 or 128");
    if (c.refill_threshold < 0 || c.refill_threshold > 32)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "refill_threshold must be in 0..32");
    if (c.max_registers != 0 && c.max_registers != 128 && c.max_registers != 168 && c.max_registers != 255)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "max_registers must be 0, 128, 168 or 255");
    if (c.rays_per_thread < 0 || c.rays_per_thread > 2)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "rays_per_thread must be 0, 1 or 2");
    return SIRIUS_OK;
}

// The streams of launches 1..n-1 and the events of n launches (copies: and of their copies to the
// host); those a handle has not yet, so that a batch's first call makes one or two streams, where
// a frame in pieces needs 7 and 17 events (about 0.7 ms).
int ensure_piece_streams(Handle* H, int n, bool copies) {
    auto event = [&](cudaEvent_t& e) { return e ? cudaSuccess : cudaEventCreateWithFlags(&e, cudaEventDisableTiming); };
    CK(event(H->piece_ev[0]));
    for (int k = 0; k < n; ++k) {
        if (k > 0 && !H->piece_stream[k - 1])
            CK(cudaStreamCreateWithFlags(&H->piece_stream[k - 1], cudaStreamNonBlocking));
        if (k > 0 || copies) CK(event(H->piece_ev[1 + k]));
        if (copies) CK(event(H->piece_ev[1 + kMaxPieces + k]));
    }
    return SIRIUS_OK;
}

// Launches on the piece streams within one call: an error exit waits for them, since what the caller
// does next is ordered after its own stream alone.
struct PieceGuard {
    Handle* H;
    bool armed = false;
    explicit PieceGuard(Handle* h) : H(h) {}
    PieceGuard(const PieceGuard&) = delete;
    PieceGuard& operator=(const PieceGuard&) = delete;
    ~PieceGuard() {
        if (!armed) return;
        for (auto& q : H->piece_stream)
            if (q) cudaStreamSynchronize(q);
        cudaGetLastError();  // (the call has its error)
    }
};

// Launch the tracer over [0, total) of already-uploaded frames.
int launch_trace(Handle* H, int n_frames, long long total, sirius_ray_result* d_results, float* d_image,
                 float* d_spectra, const sirius_camera_ray* d_rays, cudaStream_t st, bool timed,
                 const LaunchScratch* scratch = nullptr, const unsigned* d_list = nullptr, bool flux_ready = false,
                 HostOut* host = nullptr) {
    const sirius_trace_config& c = H->cfg;
    if (!scratch && (c.precision == SIRIUS_PRECISION_MIXED)) {
        const int rc = ensure(H, H->d_flux, H->flux_cap, size_t(n_frames) * kFluxTable);
        if (rc != SIRIUS_OK) return rc;
    }
    const LaunchScratch own{H->d_frames, H->d_queue, H->d_status, H->d_flux};
    const LaunchScratch& S = scratch ? *scratch : own;
    Params P{};
    P.frames = S.frames;
    P.n_frames = n_frames;
    P.total = total;
    P.results = d_results;
    P.image = d_image;
    P.spectra = d_spectra;
    P.host_rays = d_rays;
    P.list = d_list;
    if (n_frames == 1) P.f0 = H->frame0;
    P.queue = S.queue;
    P.counters = S.queue + 1;
    P.clock0 = S.queue + 4;
    P.status = S.status;
    P.c = make_cfg(c);
    const bool mixed = c.precision == SIRIUS_PRECISION_MIXED;
    // one thread per ray unless blocks_per_sm != 0 (persistent warps pulling rays
    // from a queue). Consecutive rays are neighbouring pixels, whose geodesics
    // take the same branches: a warp refilled lane by lane mixes rays at
    // different stages of their paths and diverges, so refills default to whole warps.
    P.persistent = c.blocks_per_sm != 0 ? 1 : 0;
    P.refill_threshold = c.refill_threshold > 0 ? c.refill_threshold : 1;
    // 32, 64 or 128 threads per block (__launch_bounds__ allows 128): small
    // launches (a list of gated rays) spread over more SMs with smaller blocks
    const int block = (c.block_size == 32 || c.block_size == 64) ? c.block_size : 128;
    const size_t shmem = size_t(2) * P.c.npair * block * sizeof(float2);
    // register budget: the kernel compiled for blocks_per_sm resident 128-thread
    // blocks per SM (persistent), or for max_registers (one thread per ray);
    // fewer registers, possibly spills. The default was measured on the 1024^2
    // bench frame in the tiled layout: mixed DP45 runs fastest at 128 registers
    // (16 warps per SM; 16.7 ms against 18.1 at 168 and 18.4 at 255), FP64 DP45 at
    // 168 (19.8 ms against 20.2 at 128 and 21.0 at 255); the symplectic
    // integrator keeps 255. The choice depends on the configuration
    // only, never on the launch's size or contents: the budgets' FP32 roundings
    // differ, and a ray's result must not depend on what else shares its launch.
    const bool symp = c.integrator == SIRIUS_INTEGRATOR_SYMPLECTIC;
    const bool mixed_dp45 = mixed && !symp;
    const int minb = c.blocks_per_sm > 0      ? std::min(c.blocks_per_sm, 4)
                     : c.max_registers == 128 ? 4
                     : c.max_registers == 168 ? 3
                     : c.max_registers == 255 ? 2
                     : mixed_dp45             ? kDefaultMinBlocksMixed
                     : !mixed && !symp        ? kDefaultMinBlocksFp64
                                              : kDefaultMinBlocks;
    // the classes present: one -> its specialised kernel; several -> one launch per
    // class (each thread skips the rays of others), so a ray's result never
    // depends on what else shares the batch; the persistent queue serves every
    // class from one generic kernel
    int fams[4], n_fams = 0;
    for (int f = 0; f < 4; ++f)
        if (H->family_mask & (1 << f)) fams[n_fams++] = f;
    P.family = -1;
    TraceFn launch_fn[4];
    int launch_family[4], n_launches = 0;
    if (n_fams == 1) {
        launch_fn[0] = pick_kernel(mixed, minb, fams[0], symp, n_frames == 1);
        launch_family[0] = -1;
        n_launches = 1;
    } else if (!P.persistent) {
        for (int i = 0; i < n_fams; ++i) {
            launch_fn[i] = pick_kernel(mixed, minb, fams[i], symp);
            launch_family[i] = fams[i];
        }
        n_launches = n_fams;
    } else {
        launch_fn[0] = pick_kernel(mixed, minb, kAnyFamily, symp);
        launch_family[0] = -1;
        n_launches = 1;
    }
    // two rays per thread (packed FP32 pairs): mixed DP45 over Kerr-Schild frames,
    // one-thread-per-ray launch shape, rays generated on the device
    const int rpt = c.rays_per_thread > 0 ? c.rays_per_thread : kDefaultRaysPerThread;
    const bool pair = rpt == 2 && mixed_dp45 && !P.persistent && !d_rays && n_fams == 1 &&
                      fams[0] == SIRIUS_METRIC_KERR_SCHILD;
    if (pair) {
        const int pminb = c.max_registers == 168 ? 3 : 2;
        launch_fn[0] = pick_ks_mixed_pair(pminb, n_frames == 1);
    }
    const int rays_per_block = pair ? 2 * block : block;
    const size_t shmem_launch = pair ? 2 * shmem : shmem;
    if (shmem_launch > 48 * 1024)
        CK(cudaFuncSetAttribute((const void*)launch_fn[0], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(shmem_launch)));
    // a one-frame launch of camera rays traces 8 x 4 pixel tiles per warp (tile_ray:
    // blocks of 32, 64 and 128 threads cover 8 x 4, 16 x 4 and 16 x 8 pixels; tiles
    // at the right and bottom edges are cut by the frame)
    const int tile_x = block >= 64 ? 16 : 8, tile_y = block == 128 ? 8 : 4;
    P.tiled = (n_frames == 1 && !d_list && !d_rays && !P.persistent && !pair && H->frame0.ray_offset == 0 &&
               H->frame0.width > 0 && total == H->frame0.n_rays && total % H->frame0.width == 0)
                  ? 1 : 0;
    const long long tiled_blocks =
        P.tiled ? ((H->frame0.width + tile_x - 1) / tile_x) * ((total / H->frame0.width + tile_y - 1) / tile_y) : 0;
    int grid;
    if (P.persistent) {
        int per_sm = c.blocks_per_sm;
        if (per_sm < 0) {
            int occ = 0;
            CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, launch_fn[0], block, shmem));
            per_sm = std::max(occ, 1);
        }
        grid = H->num_sms * per_sm;
        const long long need = (total + block - 1) / block;
        if (grid > need) grid = int(std::max<long long>(need, 1));
    } else {
        grid = P.tiled ? int(tiled_blocks) : int((total + rays_per_block - 1) / rays_per_block);
    }
    // a batch of frames launched one thread per ray: each block traces one pixel
    // tile of one frame (edge tiles cut by the frame), and a launch for one family
    // covers only that family's frames. Per launch i: frame entries [tab_off[i], tab_off[i+1])
    // of the table (x: first block, y: frame), grid tab_grid[i].
    std::vector<int2> tab;
    int tab_off[5] = {0, 0, 0, 0, 0}, tab_grid[4] = {grid, grid, grid, grid};
    const bool use_table = n_frames > 1 && !P.persistent && !d_list && !d_rays && !pair && !scratch &&
                           int(H->frames_host.size()) == n_frames;
    if (use_table) {
        for (int i = 0; i < n_launches; ++i) {
            tab_off[i] = int(tab.size());
            int b0 = 0;
            for (int f = 0; f < n_frames; ++f) {
                const FrameDev& F = H->frames_host[size_t(f)];
                if (launch_family[i] >= 0 && F.cls != launch_family[i]) continue;
                tab.push_back(make_int2(b0, f));
                const long long rows = F.n_rays / F.width;
                b0 += int(((F.width + tile_x - 1) / tile_x) * ((rows + tile_y - 1) / tile_y));
            }
            tab_grid[i] = b0;
        }
        tab_off[n_launches] = int(tab.size());
        int rc = ensure(H, H->d_blocks, H->blocks_cap, tab.size());
        if (rc != SIRIUS_OK) return rc;
        CK(cudaMemcpyAsync(H->d_blocks, tab.data(), tab.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
    }
    // [0] queue cursor, [1..3] counters, [4] launch start: all start at zero
    CK(cudaMemsetAsync(S.queue, 0, 5 * sizeof(unsigned long long), st));
    CK(cudaMemsetAsync(S.status, 0, sizeof(int), st));
    // whole-launch bound on the device clock, measured from the first warp's start
    P.watchdog_ns = c.watchdog_ms > 0 ? (unsigned long long)c.watchdog_ms * 1000000ull : ~0ull;
    if (timed) CK(cudaEventRecord(H->ev[1], st));
    // the mixed path reads the disk flux from per-frame tables
    P.flux = nullptr;
    int extra_launches = 0;
    if (mixed && c.enable_disk && (H->family_mask & ((1 << SIRIUS_METRIC_KERR_SCHILD) | (1 << kClassRing))) && S.flux) {
        if (!flux_ready) {  // else the caller built this upload's tables ahead of this stream
            flux_table_kernel<<<n_frames, kFluxN, 0, st>>>(S.frames, S.flux);
            CK(cudaGetLastError());
            extra_launches = 1;
        }
        P.flux = S.flux;
    }
    // A one-frame tiled launch whose outputs go to host memory traces its tile
    // rows in pieces, each on its own stream (all queued at once, so the next
    // piece's blocks fill the SMs as the previous piece drains, as in one launch),
    // and copies each piece's rays (whole pixel rows, contiguous in every output)
    // to the host on the piece's stream as soon as it is traced, while the other
    // pieces trace (pieces end out of order: the rows of the shadow and the disk
    // cost most). The kernel and each ray's result are those of the single launch.
    const int tiles_x = P.tiled ? (H->frame0.width + tile_x - 1) / tile_x : 1;
    const int tile_rows = P.tiled ? int(tiled_blocks / tiles_x) : 0;
    const int n_pieces = (host && P.tiled && n_launches == 1 && tiled_blocks >= kPieceMinBlocks)
                             ? std::min(kMaxPieces, tile_rows) : 0;
    PieceGuard pieces(H);
    if (n_pieces > 1) {
        const int rc = ensure_piece_streams(H, n_pieces, true);
        if (rc != SIRIUS_OK) return rc;
        pieces.armed = true;
        cudaEvent_t* E = H->piece_ev;
        CK(cudaEventRecord(E[0], st));
        for (int k = 1; k < n_pieces; ++k) CK(cudaStreamWaitEvent(H->piece_stream[k - 1], E[0], 0));
        const long long width = H->frame0.width, rows = total / width;
        const size_t nb = size_t(host->nb);
        P.family = launch_family[0];
        for (int k = 0; k < n_pieces; ++k) {
            const int t0 = int((long long)tile_rows * k / n_pieces), t1 = int((long long)tile_rows * (k + 1) / n_pieces);
            cudaStream_t sk = k == 0 ? st : H->piece_stream[k - 1];
            P.block0 = t0 * tiles_x;
            launch_fn[0]<<<(t1 - t0) * tiles_x, block, shmem_launch, sk>>>(P);
            CK(cudaGetLastError());
            CK(cudaEventRecord(E[1 + k], sk));
            const long long r0 = (long long)t0 * tile_y * width;
            const long long r1 = std::min<long long>((long long)t1 * tile_y, rows) * width;
            const size_t n = size_t(r1 - r0);
            if (host->results)
                CK(cudaMemcpyAsync(host->results + r0, d_results + r0, n * sizeof(sirius_ray_result),
                                   cudaMemcpyDeviceToHost, sk));
            if (host->image)
                CK(cudaMemcpyAsync(host->image + r0, d_image + r0, n * sizeof(float), cudaMemcpyDeviceToHost, sk));
            if (host->spectra && nb)
                CK(cudaMemcpyAsync(host->spectra + size_t(r0) * nb, d_spectra + size_t(r0) * nb, n * nb * sizeof(float),
                                   cudaMemcpyDeviceToHost, sk));
            CK(cudaEventRecord(E[1 + kMaxPieces + k], sk));
        }
        P.block0 = 0;
        for (int k = 1; k < n_pieces; ++k) CK(cudaStreamWaitEvent(st, E[1 + k], 0));
        host->done = true;
        n_launches = 0;  // the pieces were the launch
    }
    // a batch's per-family launches side by side, each after the first on a stream of its
    // own: the next family's blocks fill the SMs as one family's last wave drains (12
    // frames of 64^2 to 320^2: 9.73 -> 7.48 ms). Launches from prepared or static scratch, which
    // may be captured, stay on the caller's stream.
    const bool side = n_launches > 1 && !scratch;
    if (side) {
        const int rc = ensure_piece_streams(H, n_launches, false);
        if (rc != SIRIUS_OK) return rc;
        pieces.armed = true;
        CK(cudaEventRecord(H->piece_ev[0], st));
    }
    for (int i = 0; i < n_launches; ++i) {
        P.family = launch_family[i];
        int g = grid;
        if (use_table) {
            P.blocks = H->d_blocks + tab_off[i];
            P.n_block_frames = tab_off[i + 1] - tab_off[i];
            g = tab_grid[i];
            if (g == 0) continue;
        }
        cudaStream_t si = side && i > 0 ? H->piece_stream[i - 1] : st;
        if (si != st) CK(cudaStreamWaitEvent(si, H->piece_ev[0], 0));
        launch_fn[i]<<<g, block, shmem_launch, si>>>(P);
        CK(cudaGetLastError());
        if (si != st) CK(cudaEventRecord(H->piece_ev[1 + i], si));
    }
    if (side)
        for (int i = 1; i < n_launches; ++i)
            if (!use_table || tab_grid[i] != 0) CK(cudaStreamWaitEvent(st, H->piece_ev[1 + i], 0));
    if (timed) CK(cudaEventRecord(H->ev[2], st));
    // the pieces' copies: after the end event, which times the kernels alone
    for (int k = 1; k < n_pieces; ++k) CK(cudaStreamWaitEvent(st, H->piece_ev[1 + kMaxPieces + k], 0));
    pieces.armed = false;
    H->stats.grid_blocks = grid;
    H->stats.block_size = block;
    H->stats.kernel_launches = (n_pieces > 1 ? n_pieces : n_launches) + extra_launches;
    return SIRIUS_OK;
}

int samples_grid(const sirius_trace_config& c) {
    int g = 1;
    while ((g + 1) * (g + 1) <= c.samples_per_pixel) ++g;
    return g;
}

// Multi-sample pass buffers and the g x g variants of the uploaded frame
// descriptors (one per sub-pixel offset, row by row) on the device.
int prepare_passes(Handle* H, long long total, cudaStream_t st) {
    const int g = samples_grid(H->cfg);
    if (g == 1) return SIRIUS_OK;
    if (H->pass_cap < size_t(total)) {
        cudaFree(H->d_pass_image);
        cudaFree(H->d_pass_spectra);
        H->d_pass_image = H->d_pass_spectra = nullptr;
        H->pass_cap = 0;
        CK(cudaMalloc((void**)&H->d_pass_image, size_t(total) * sizeof(float)));
        CK(cudaMalloc((void**)&H->d_pass_spectra, size_t(total) * SIRIUS_MAX_BINS * sizeof(float)));
        H->pass_cap = size_t(total);
    }
    const size_t n = H->frames_host.size();
    H->pass_frames_host.resize(size_t(g) * g * n);
    for (int s = 0; s < g * g; ++s) {
        const float u = (float(s % g) + 0.5f) / float(g), v = (float(s / g) + 0.5f) / float(g);
        for (size_t i = 0; i < n; ++i) {
            FrameDev f = H->frames_host[i];
            f.sub_u = u;
            f.sub_v = v;
            H->pass_frames_host[size_t(s) * n + i] = f;
        }
    }
    int rc = ensure(H, H->d_pass_frames, H->pass_frames_cap, H->pass_frames_host.size());
    if (rc != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(H->d_pass_frames, H->pass_frames_host.data(), H->pass_frames_host.size() * sizeof(FrameDev),
                       cudaMemcpyHostToDevice, st));
    return SIRIUS_OK;
}

// The trace of the uploaded frames into the given outputs; with
// samples_per_pixel > 1, one launch per sub-pixel offset of the g x g grid
// (row by row), each into pass buffers, summed in that order and scaled by
// 1/g^2. prepared: the pass descriptors are already on the device
// (sirius_cuda_prepare_frames), so only stream work is issued.
int launch_frames(Handle* H, int n_frames, long long total, sirius_ray_result* d_results, float* d_image,
                  float* d_spectra, cudaStream_t st, bool timed, bool prepared = false, HostOut* host = nullptr) {
    const int g = samples_grid(H->cfg);
    if (g == 1)
        return launch_trace(H, n_frames, total, d_results, d_image, d_spectra, nullptr, st, timed, nullptr, nullptr,
                            false, host);
    if (d_results) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "per-ray results need samples_per_pixel <= 1");
    if (!d_image && !d_spectra) return SIRIUS_OK;
    const int nb = H->cfg.enable_volumetric ? std::min(H->cfg.n_bins, SIRIUS_MAX_BINS) : 0;
    if (!prepared) {
        const int rc = prepare_passes(H, total, st);
        if (rc != SIRIUS_OK) return rc;
    }
    const size_t n = size_t(n_frames);
    const int blocks = int((total + 255) / 256), sblocks = int((total * std::max(nb, 1) + 255) / 256);
    if (timed) CK(cudaEventRecord(H->ev[1], st));
    for (int s = 0; s < g * g; ++s) {
        H->frame0 = H->pass_frames_host[size_t(s) * n];
        CK(cudaMemcpyAsync(H->d_frames, H->d_pass_frames + size_t(s) * n, n * sizeof(FrameDev),
                           cudaMemcpyDeviceToDevice, st));
        int rc = launch_trace(H, n_frames, total, nullptr, d_image ? H->d_pass_image : nullptr,
                              (d_spectra && nb) ? H->d_pass_spectra : nullptr, nullptr, st, false);
        if (rc != SIRIUS_OK) return rc;
        if (d_image) pass_accumulate_kernel<<<blocks, 256, 0, st>>>(H->d_pass_image, d_image, total, s == 0);
        if (d_spectra && nb)
            pass_accumulate_kernel<<<sblocks, 256, 0, st>>>(H->d_pass_spectra, d_spectra, total * nb, s == 0);
        CK(cudaGetLastError());
    }
    const float scale = 1.0f / float(g * g);
    if (d_image) pass_scale_kernel<<<blocks, 256, 0, st>>>(d_image, total, scale);
    if (d_spectra && nb) pass_scale_kernel<<<sblocks, 256, 0, st>>>(d_spectra, total * nb, scale);
    CK(cudaGetLastError());
    if (timed) CK(cudaEventRecord(H->ev[2], st));
    H->frame0 = H->frames_host[0];
    return SIRIUS_OK;
}

int finish_stats(Handle* H, cudaStream_t st, long long total, bool timed) {
    unsigned long long cnt[4] = {};
    int status = 0;
    CK(cudaMemcpyAsync(cnt, H->d_queue, sizeof(cnt), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&status, H->d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    H->stats.rays = total;
    H->stats.accepted_steps = (long long)cnt[1];
    H->stats.rejected_steps = (long long)cnt[2];
    H->stats.fp64_steps = (long long)cnt[3];
    H->stats.status_flags = status;
    if (timed) {
        float k = 0, t = 0;
        CK(cudaEventElapsedTime(&k, H->ev[1], H->ev[2]));
        CK(cudaEventElapsedTime(&t, H->ev[0], H->ev[3]));
        H->stats.kernel_ms = k;
        H->stats.total_ms = t;
    }
    if (status & 1) return fail(H, SIRIUS_ERR_TIMEOUT, "trace kernel stopped by its watchdog");
    return SIRIUS_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Library-owned scratch of sirius_cuda_trace_frames_static: a file-scope
// device array, so that entry point allocates nothing. Its queue/counter words
// and status word must be zero when a launch starts (the entry point zeroes
// them on its stream before each launch); the frame descriptors are rewritten
// by every call. One array per device: calls in flight at the same time on one
// device (other streams, other handles, other host threads) share it and race.
// ---------------------------------------------------------------------------
namespace {
struct StaticScratch {
    FrameDev frames[SIRIUS_STATIC_MAX_FRAMES];
    unsigned long long queue[8];  // [0] cursor, [1..3] counters, [4] launch start
    int status;
    float flux[SIRIUS_STATIC_MAX_FRAMES * kFluxTable];  // the mixed path's disk flux tables
};
constexpr int kStaticMaxDevices = 64;
}  // namespace

static __device__ __align__(256) unsigned char g_static_scratch[sizeof(StaticScratch)];
static_assert(sizeof(StaticScratch) <= 168 * 1024, "static scratch stays modest");

namespace {
// The device address of g_static_scratch on `device`, resolved once per device
// (the first call per device should come before any stream capture).
StaticScratch* static_scratch(int device) {
    static void* addr[kStaticMaxDevices] = {};
    static std::once_flag once[kStaticMaxDevices];
    std::call_once(once[device], [device] {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_scratch) == cudaSuccess) addr[device] = p;
        else cudaGetLastError();
    });
    return static_cast<StaticScratch*>(addr[device]);
}
}  // namespace

// ---------------------------------------------------------------------------
// Surrogate training (train.cuh): device state, the launch sequence of one
// optimiser step, and its captured graph.
// ---------------------------------------------------------------------------
namespace {
struct TrainState {
    sirius_train_config cfg{};
    float* params = nullptr;  // FP32 master weights
    float* grad = nullptr;
    float* m1 = nullptr;
    float* m2 = nullptr;
    __nv_bfloat16* wbf = nullptr;  // BF16 copies the GEMMs read (train::kBfTotal elements)
    train::StepState* st = nullptr;
    int* err = nullptr;  // [0] error flag, [2..3] the forward kernel's tile counter (which it leaves at zero)
    CUtensorMap wmap[4] = {};  // W2, W3, W4, W5 of wbf for the forward kernel
    bool tma = false;          // whether the driver encoded them
    bool ready = false;        // an initialisation has succeeded: the parameters are there
    long long cap = 0;  // rows the activation buffers hold
    unsigned char* rows = nullptr;  // the allocation that holds them, x0 to y
    __nv_bfloat16* x0 = nullptr;
    __nv_bfloat16* h[4] = {};
    __nv_bfloat16* dy = nullptr;
    __nv_bfloat16* dz[4] = {};        // dZ of layers 4, 3, 2, 1
    cudaStream_t side = nullptr;      // the weight gradients' branch of the step
    cudaEvent_t fork = nullptr, join = nullptr;
    float* t = nullptr;
    float* w = nullptr;
    float* z[4] = {};
    float* y = nullptr;
    cudaGraphExec_t graph = nullptr;  // one optimiser step
    const void* key[3] = {};          // the training set the graph was captured for
    long long key_rows = 0;
};

void train_free_rows(TrainState* T) {
    cudaFree(T->rows);
    T->rows = nullptr;
    T->cap = 0;
}

void train_drop_graph(TrainState* T) {
    if (T->graph) cudaGraphExecDestroy(T->graph);
    T->graph = nullptr;
    T->key[0] = T->key[1] = T->key[2] = nullptr;
    T->key_rows = 0;
}

void train_free(TrainState* T) {
    if (!T) return;
    train_drop_graph(T);
    train_free_rows(T);
    cudaFree(T->params); cudaFree(T->grad); cudaFree(T->m1); cudaFree(T->m2); cudaFree(T->wbf);
    cudaFree(T->st); cudaFree(T->err);
    if (T->side) cudaStreamDestroy(T->side);
    if (T->fork) cudaEventDestroy(T->fork);
    if (T->join) cudaEventDestroy(T->join);
    delete T;
}

// The buffers of a batch, carved from one allocation (15 of their own took 0.8 ms more to make
// and to release; each begins on a 1024-byte boundary).
int train_rows(Handle* H, TrainState* T, long long rows) {
    if (rows <= T->cap) return SIRIUS_OK;
    train_drop_graph(T);
    train_free_rows(T);
    using namespace train;
    size_t total = 0;
    auto carve = [&](auto*& p, long long width) {  // (before the allocation: sizes alone)
        p = T->rows ? reinterpret_cast<std::remove_reference_t<decltype(p)>>(T->rows + total) : nullptr;
        total += (size_t(rows) * width * sizeof(*p) + 1023) / 1024 * 1024;
    };
    auto carve_all = [&] {
        total = 0;
        carve(T->x0, kInPad);
        carve(T->dy, kOutPad);
        for (auto& p : T->h) carve(p, kHid);
        for (auto& p : T->dz) carve(p, kHid);
        for (auto& p : T->z) carve(p, kHid);
        carve(T->t, 4);
        carve(T->w, 1);
        carve(T->y, kOut);
    };
    carve_all();
    CK(cudaMalloc((void**)&T->rows, total));
    carve_all();
    T->cap = rows;
    return SIRIUS_OK;
}

// Whether a step can run: the parameters are there, and the buffers of the configured batch (an
// initialisation for a larger one may have run out of memory).
bool train_ready(const TrainState* T) { return T && T->ready && T->cap >= T->cfg.batch; }

unsigned long long train_wait_limit(const Handle* H) {
    return (unsigned long long)(H->configured && H->cfg.watchdog_ms > 0 ? H->cfg.watchdog_ms : 30000) * 1000000ull;
}

template <int BN, int E>
void gemm_launch(const train::GemmArgs& g0, cudaStream_t s) {
    train::GemmArgs g = g0;
    // a TMA operand moves whole 64-wide K boxes: other K splits take the register path
    if (g.K % train::kBK != 0 || g.k_per_cta % train::kBK != 0) g.tma_a = g.tma_b = 0;
    const dim3 grid((g.M + train::kBM - 1) / train::kBM, (g.N + BN - 1) / BN, (g.K + g.k_per_cta - 1) / g.k_per_cta);
    if (g.tma_a || g.tma_b)
        train::gemm_kernel<BN, E, true><<<grid, train::kGemmThreads, train::GemmSmem<BN>::Bytes, s>>>(g);
    else
        train::gemm_kernel<BN, E, false><<<grid, train::kGemmThreads, train::GemmSmem<BN>::Bytes, s>>>(g);
}

int train_set_attributes(Handle* H) {
    using namespace train;
    CK(cudaFuncSetAttribute(surrogate::train_forward_kernel<surrogate::kTrainTma>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, surrogate::kPairSmBytes));
    CK(cudaFuncSetAttribute(surrogate::train_forward_kernel<surrogate::kTrainPlain>,
                            cudaFuncAttributeMaxDynamicSharedMemorySize, surrogate::kPairSmBytes));
    CK(cudaFuncSetAttribute(gemm_kernel<256, kEpiDHidden, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            GemmSmem<256>::Bytes));
    CK(cudaFuncSetAttribute(gemm_kernel<256, kEpiDHidden, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            GemmSmem<256>::Bytes));
    CK(cudaFuncSetAttribute(gemm_kernel<256, kEpiDWeight, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            GemmSmem<256>::Bytes));
    CK(cudaFuncSetAttribute(gemm_kernel<256, kEpiDWeight, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            GemmSmem<256>::Bytes));
    return SIRIUS_OK;
}

constexpr long long kTrainBf[4] = {train::kBfW1, train::kBfW2, train::kBfW3, train::kBfW4};

// cuTensorMapEncodeTiled from the driver, through the runtime's entry-point query
// (the library links no driver library)
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();  // (answered here, by the register path)
            return EncodeTiledFn(nullptr);
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// A K-major BF16 operand (rows x K, row stride ld elements) as a TMA map of
// 64 x box_rows boxes with the 128-byte swizzle (rows beyond `rows` read as
// zeros). False when the driver has no encoder or refuses the map; the operand
// then goes through registers.
bool kmajor_map(CUtensorMap* m, const __nv_bfloat16* p, long long rows, long long K, long long ld, int box_rows) {
    const EncodeTiledFn fn = encode_tiled();
    if (!fn || K % 64 != 0 || (ld * 2) % 16 != 0 || (reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
    const cuuint64_t dims[2] = {cuuint64_t(K), cuuint64_t(rows)};
    const cuuint64_t strides[1] = {cuuint64_t(ld) * 2};
    const cuuint32_t box[2] = {64u, cuuint32_t(box_rows)};
    const cuuint32_t es[2] = {1u, 1u};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// An MN-major BF16 operand (element (row, k) at p[k * ld + row]: K rows of ld
// elements, `rows` of them used) as a TMA map of 64 (MN) x 64 (K) boxes with the
// 128-byte swizzle.
bool mnmajor_map(CUtensorMap* m, const __nv_bfloat16* p, long long rows, long long K, long long ld) {
    const EncodeTiledFn fn = encode_tiled();
    if (!fn || K % 64 != 0 || (ld * 2) % 16 != 0 || (reinterpret_cast<uintptr_t>(p) & 15) != 0) return false;
    const cuuint64_t dims[2] = {cuuint64_t(rows), cuuint64_t(K)};
    const cuuint64_t strides[1] = {cuuint64_t(ld) * 2};
    const cuuint32_t box[2] = {64u, 64u};
    const cuuint32_t es[2] = {1u, 1u};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// TMA for the operands whose K is a multiple of 64: K-major ones as rows x 64
// boxes, MN-major ones (the weight-gradient products' dZ^T and H, the dH products'
// W) as 64 x 64 boxes when their tile extent (kBM, or BN) is a multiple of 64; the
// 16-wide input layer and the 16-wide MN-major operands stay on the register path
int tma_mode(const train::Operand& op, int tile_rows, long long K, CUtensorMap* m) {
    if (K % 64 != 0) return 0;
    if (op.kmajor) return kmajor_map(m, op.p, op.rows, K, op.ld, tile_rows) ? 1 : 0;
    if (tile_rows % 64 != 0) return 0;
    return mnmajor_map(m, op.p, op.rows, K, op.ld) ? 2 : 0;
}

void use_tma(train::GemmArgs& g, int bn, bool a, bool b) {
    g.tma_a = a ? tma_mode(g.a, train::kBM, g.K, &g.ta) : 0;
    g.tma_b = b ? tma_mode(g.b, bn, g.K, &g.tb) : 0;
}

// forward over the first `rows` gathered rows: Z_l, H_l (l = 1..4) and Y
void train_forward(const Handle* H, TrainState* T, int rows, cudaStream_t s) {
    using namespace train;
    surrogate::TrainForward f{};
    f.x0 = T->x0;
    f.w1 = T->wbf + kBfW1;
    for (int l = 0; l < 5; ++l) f.bias[l] = T->params + kOffB[l];
    for (int l = 0; l < 4; ++l) {
        f.z[l] = T->z[l];
        f.h[l] = T->h[l];
    }
    for (int l = 0; l < 4; ++l) {
        f.w[l] = T->wmap[l];
        f.wp[l] = T->wbf + (l < 3 ? kTrainBf[l + 1] : kBfW5);
    }
    const int tiles = (rows + 2 * surrogate::kTileM - 1) / (2 * surrogate::kTileM);
    const int grid = 2 * std::min(tiles, std::max(H->num_sms / 2, 1));
    // (without tensor maps as the GEMMs do: operands through registers)
    const auto kernel = T->tma ? surrogate::train_forward_kernel<surrogate::kTrainTma>
                               : surrogate::train_forward_kernel<surrogate::kTrainPlain>;
    kernel<<<grid, surrogate::kPairThreads, surrogate::kPairSmBytes, s>>>(
        f, rows, T->y, T->err, reinterpret_cast<unsigned long long*>(T->err + 2), train_wait_limit(H));
}

void train_loss(TrainState* T, int rows, bool with_grad, cudaStream_t s) {
    const int blocks = (rows + 255) / 256;
    train::loss_sums_kernel<<<blocks, 256, 0, s>>>(T->t, T->w, rows, T->st);
    train::loss_grad_kernel<<<blocks, 256, 0, s>>>(T->y, T->t, T->w, rows, T->st, T->dy,
                                                   with_grad ? T->grad + train::kOffB[4] : nullptr);
}

// gradient of the batch loss into T->grad (which must hold zeros); rows a multiple of 128.
// A layer's weight gradient and the next dH both need its dZ and not one another: the
// weight gradients run on a side stream (a parallel branch of the captured step), where
// their 128 CTAs fill the slots that the dH products' 256 leave of 296 and cover their
// start and end (32768 rows: 0.265 -> 0.245 ms a step). Each dZ has a buffer of its own.
void train_backward(const Handle* H, TrainState* T, int rows, cudaStream_t s) {
    using namespace train;
    auto side_after = [&]() {
        cudaEventRecord(T->fork, s);
        cudaStreamWaitEvent(T->side, T->fork, 0);
    };
    GemmArgs g{};
    g.err = T->err;
    g.wait_limit_ns = train_wait_limit(H);
    const int kpc = std::max(64, ((rows / 64 + 63) / 64) * 64);  // batch rows per CTA in the weight gradients
    // dW5^T = H4^T dY
    g.a = Operand{T->h[3], kHid, 0, kHid};
    g.b = Operand{T->dy, kOutPad, 0, kOutPad};
    g.M = kHid; g.N = kOutPad; g.K = rows; g.k_per_cta = kpc;
    g.e = EpiArgs{};
    g.e.grad = T->grad + kOffW[4]; g.e.ldg = kHid; g.e.ng = kOut;
    use_tma(g, 16, true, true);
    side_after();
    gemm_launch<16, kEpiDWeightT>(g, T->side);
    // dH4 = dY W5 -> dZ4 (and the b4 gradient)
    g.a = Operand{T->dy, kOutPad, 1, rows};
    g.b = Operand{T->wbf + kBfW5, kHid, 0, kHid};
    g.M = rows; g.N = kHid; g.K = g.k_per_cta = kOutPad;
    g.e = EpiArgs{};
    g.e.z = T->z[3]; g.e.ldz = kHid; g.e.h = T->dz[0]; g.e.ldh = kHid; g.e.grad = T->grad + kOffB[3];
    use_tma(g, 256, true, true);
    gemm_launch<256, kEpiDHidden>(g, s);
    for (int l = 3; l >= 1; --l) {  // layers 4, 3, 2
        __nv_bfloat16* cur = T->dz[3 - l];
        __nv_bfloat16* nxt = T->dz[4 - l];
        // dW_l = dZ_l^T H_{l-1}
        g.a = Operand{cur, kHid, 0, kHid};
        g.b = Operand{T->h[l - 1], kHid, 0, kHid};
        g.M = kHid; g.N = kHid; g.K = rows; g.k_per_cta = kpc;
        g.e = EpiArgs{};
        g.e.grad = T->grad + kOffW[l]; g.e.ldg = kHid; g.e.ng = kHid;
        use_tma(g, 256, true, true);
        side_after();
        gemm_launch<256, kEpiDWeight>(g, T->side);
        // dH_{l-1} = dZ_l W_l -> dZ_{l-1} (and the b_{l-1} gradient)
        g.a = Operand{cur, kHid, 1, rows};
        g.b = Operand{T->wbf + kTrainBf[l], kHid, 0, kHid};
        g.M = rows; g.N = kHid; g.K = g.k_per_cta = kHid;
        g.e = EpiArgs{};
        g.e.z = T->z[l - 1]; g.e.ldz = kHid; g.e.h = nxt; g.e.ldh = kHid; g.e.grad = T->grad + kOffB[l - 1];
        use_tma(g, 256, true, true);
        gemm_launch<256, kEpiDHidden>(g, s);
    }
    // dW1 = dZ1^T X0: the 2 x 5 input columns (high and low BF16 terms of each
    // feature) folded onto the 5 weights they share
    g.a = Operand{T->dz[3], kHid, 0, kHid};
    g.b = Operand{T->x0, kInPad, 0, kInPad};
    g.M = kHid; g.N = kInPad; g.K = rows; g.k_per_cta = kpc;
    g.e = EpiArgs{};
    g.e.grad = T->grad + kOffW[0]; g.e.ldg = kIn; g.e.ng = 2 * kIn; g.e.fold = kIn;
    use_tma(g, 16, true, true);
    gemm_launch<16, kEpiDWeight>(g, s);
    cudaEventRecord(T->join, T->side);
    cudaStreamWaitEvent(s, T->join, 0);
}

void train_step(const Handle* H, TrainState* T, const float* feat, const float* targets, const float* weights,
                long long n_rows, cudaStream_t s) {
    const int B = T->cfg.batch;
    const int spe = int(n_rows / B);
    train::gather_kernel<<<(B + 255) / 256, 256, 0, s>>>(feat, targets, weights, n_rows, B, spe, T->cfg.seed, 0, 0,
                                                         T->st, T->x0, T->t, T->w);
    train_forward(H, T, B, s);
    train_loss(T, B, true, s);
    train_backward(H, T, B, s);
    const train::AdamConfig c{T->cfg.max_lr, T->cfg.warmup_fraction, T->cfg.beta1, T->cfg.beta2,
                              T->cfg.eps,    T->cfg.weight_decay,    T->cfg.total_steps};
    train::adam_kernel<<<H->num_sms * 2, 256, 0, s>>>(T->params, T->grad, T->m1, T->m2, T->wbf, T->st, c);
}

int train_check_err(Handle* H, TrainState* T) {
    int err = 0;
    CK(cudaMemcpyAsync(&err, T->err, sizeof(int), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaStreamSynchronize(H->stream));
    if (err) return fail(H, SIRIUS_ERR_TIMEOUT, "training GEMM stopped by its wait bound");
    return SIRIUS_OK;
}
}  // namespace

extern "C" {

int sirius_cuda_abi_version(void) { return SIRIUS_CUDA_ABI_VERSION; }

int sirius_cuda_default_config(sirius_trace_config* c) {
    if (!c) return SIRIUS_ERR_INVALID_ARGUMENT;
    std::memset(c, 0, sizeof(*c));
    // IntegratorConfig / TracerConfig as RenderSession sets them (SNRS001A.cpp:103-129)
    c->abs_tolerance = 5e-6; c->rel_tolerance = 5e-6; c->min_step = 1e-5; c->max_step = 2.0; c->initial_step = 0.1;
    c->safety_factor = 0.9; c->step_grow_max = 2.0; c->step_shrink_min = 0.1;
    c->escape_radius = 200.0; c->horizon_factor = 1.05; c->max_steps = 20000; c->enable_disk = 1;
    c->disk_temperature_inner = 1.0; c->crossing_weight_decay = kPi;
    c->enable_volumetric = 0; c->n_bins = 0; c->nu_min = 1e-2; c->nu_max = 1e2; c->vol_j0 = 1.0;
    c->vol_alpha_over_j = 0.1; c->vol_height_ratio = 0.1; c->vol_spectral_index = 0.7; c->vol_substeps = 4;
    c->integrator = SIRIUS_INTEGRATOR_DP45; c->precision = SIRIUS_PRECISION_FP64; c->compat = 0;
    c->projection_period = 1; c->spiral_check = 0; c->island_factor = 1.5; c->critical_band = 0.05; c->symplectic_step = 0.01;
    c->symplectic_order = 4; c->block_size = 0; c->refill_threshold = 0; c->blocks_per_sm = 0; c->watchdog_ms = 30000;
    return SIRIUS_OK;
}

int sirius_cuda_create(int device, sirius_cuda_handle* out) {
    if (!out) return SIRIUS_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) { cudaGetLastError(); return SIRIUS_ERR_NO_DEVICE; }
    if (device < 0 || device >= n) return SIRIUS_ERR_INVALID_ARGUMENT;
    Handle* H = new (std::nothrow) Handle();
    if (!H) return SIRIUS_ERR_OUT_OF_MEMORY;
    H->device = device;
    auto bail = [&](int code) { delete H; return code; };
    if (cudaSetDevice(device) != cudaSuccess) return bail(SIRIUS_ERR_CUDA);
    // (two attributes: the whole property record takes 2.5 ms, and up to a hundred times that while
    // other processes keep the driver busy)
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&H->num_sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return bail(SIRIUS_ERR_CUDA);
    if (major < 10) return bail(SIRIUS_ERR_UNSUPPORTED);
    if (cudaStreamCreateWithFlags(&H->stream, cudaStreamNonBlocking) != cudaSuccess) return bail(SIRIUS_ERR_CUDA);
    for (auto& e : H->ev)
        if (cudaEventCreate(&e) != cudaSuccess) return bail(SIRIUS_ERR_CUDA);
    if (cudaMalloc((void**)&H->d_queue, 8 * sizeof(unsigned long long)) != cudaSuccess) return bail(SIRIUS_ERR_OUT_OF_MEMORY);
    if (cudaMalloc((void**)&H->d_status, sizeof(int)) != cudaSuccess) return bail(SIRIUS_ERR_OUT_OF_MEMORY);
    sirius_cuda_default_config(&H->cfg);
    H->configured = true;
    *out = H;
    return SIRIUS_OK;
}

int sirius_cuda_destroy(sirius_cuda_handle h) {
    Handle* H = static_cast<Handle*>(h);
    if (!H) return SIRIUS_ERR_INVALID_ARGUMENT;
    cudaSetDevice(H->device);
    if (H->stream) cudaStreamSynchronize(H->stream);
    cudaFree(H->d_frames); cudaFree(H->d_results); cudaFree(H->d_image); cudaFree(H->d_spectra);
    cudaFree(H->d_flux);
    cudaFree(H->d_rays); cudaFree(H->d_queue); cudaFree(H->d_status);
    cudaFree(H->d_surrogate); cudaFree(H->d_sur_err);
    cudaFree(H->d_sur_frames); cudaFree(H->d_feat); cudaFree(H->d_mlp_out); cudaFree(H->d_list); cudaFree(H->d_gate);
    cudaFree(H->d_coarse_feat); cudaFree(H->d_coarse_out);
    cudaFree(H->d_block_counts);
    cudaFree(H->d_mlp_rows);
    cudaFree(H->d_blocks);
    cudaFree(H->d_pass_image); cudaFree(H->d_pass_spectra); cudaFree(H->d_pass_frames); cudaFree(H->d_prep);
    if (H->h_sur_frames) cudaFreeHost(H->h_sur_frames);
    if (H->h_list_len) cudaFreeHost(H->h_list_len);
    cudaFree(H->d_tmp);
    train_free(H->train);
    for (auto& e : H->sev) if (e) cudaEventDestroy(e);
    for (auto& e : H->fev) if (e) cudaEventDestroy(e);
    for (auto& q : H->sur_stream) if (q) cudaStreamDestroy(q);
    for (auto& e : H->piece_ev) if (e) cudaEventDestroy(e);
    for (auto& q : H->piece_stream) if (q) cudaStreamDestroy(q);
    for (auto& e : H->ev) if (e) cudaEventDestroy(e);
    if (H->stream) cudaStreamDestroy(H->stream);
    delete H;
    return SIRIUS_OK;
}

const char* sirius_cuda_get_last_error(sirius_cuda_handle h) {
    Handle* H = static_cast<Handle*>(h);
    return H ? H->last_error.c_str() : "invalid handle";
}

int sirius_cuda_configure(sirius_cuda_handle h, const sirius_trace_config* c) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !c) return SIRIUS_ERR_INVALID_ARGUMENT;
    const int rc = validate_config(H, *c);
    if (rc != SIRIUS_OK) return rc;
    H->cfg = *c;
    H->configured = true;
    return SIRIUS_OK;
}

static int upload_frames(Handle* H, const sirius_frame* frames, int n, long long* total_out) {
    std::vector<FrameDev> fd(n);
    long long total = 0;
    for (int i = 0; i < n; ++i) {
        const sirius_frame& f = frames[i];
        int rc = validate_frame(H, f);
        if (rc != SIRIUS_OK) return rc;
        if (f.ray_offset != total)
            return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "frames must be contiguous: ray_offset[i] = sum of previous pixel counts");
        fd[i] = make_frame(f, H->cfg);
        fd[i].flux_slot = i;
        total += fd[i].n_rays;
    }
    H->family_mask = 0;
    for (int i = 0; i < n; ++i) H->family_mask |= 1 << fd[i].cls;
    H->frame0 = fd[0];
    H->frames_host = fd;
    int rc = ensure(H, H->d_frames, H->frames_cap, size_t(n));
    if (rc != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(H->d_frames, fd.data(), n * sizeof(FrameDev), cudaMemcpyHostToDevice, H->stream));
    *total_out = total;
    return SIRIUS_OK;
}

int sirius_cuda_trace_frames(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                             sirius_ray_result* results, float* image, float* spectra) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    cudaStream_t st = H->stream;
    CK(cudaEventRecord(H->ev[0], st));
    long long total = 0;
    int rc = upload_frames(H, frames, n_frames, &total);
    if (rc != SIRIUS_OK) return rc;
    const int nb = H->cfg.enable_volumetric ? std::min(H->cfg.n_bins, SIRIUS_MAX_BINS) : 0;
    if (results && (rc = ensure(H, H->d_results, H->results_cap, size_t(total))) != SIRIUS_OK) return rc;
    if (image && (rc = ensure(H, H->d_image, H->image_cap, size_t(total))) != SIRIUS_OK) return rc;
    if (spectra && nb && (rc = ensure(H, H->d_spectra, H->spectra_cap, size_t(total) * nb)) != SIRIUS_OK) return rc;
    // copies overlap the trace only into page-locked memory (a copy into pageable
    // memory returns once it is done, which would hold back the next piece's launch)
    auto page_locked = [](const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeHost;
    };
    const bool overlap = (!results || page_locked(results)) && (!image || page_locked(image)) &&
                         (!(spectra && nb) || page_locked(spectra));
    HostOut host{results, image, (spectra && nb) ? spectra : nullptr, nb, false};
    rc = launch_frames(H, n_frames, total, results ? H->d_results : nullptr, image ? H->d_image : nullptr,
                       (spectra && nb) ? H->d_spectra : nullptr, st, true, false, overlap ? &host : nullptr);
    if (rc != SIRIUS_OK) return rc;
    if (!host.done) {  // else copied piece by piece during the trace
        if (results) CK(cudaMemcpyAsync(results, H->d_results, size_t(total) * sizeof(sirius_ray_result), cudaMemcpyDeviceToHost, st));
        if (image) CK(cudaMemcpyAsync(image, H->d_image, size_t(total) * sizeof(float), cudaMemcpyDeviceToHost, st));
        if (spectra && nb) CK(cudaMemcpyAsync(spectra, H->d_spectra, size_t(total) * nb * sizeof(float), cudaMemcpyDeviceToHost, st));
    }
    CK(cudaEventRecord(H->ev[3], st));
    return finish_stats(H, st, total, true);
}

int sirius_cuda_trace_frames_device(sirius_cuda_handle h, const sirius_frame* d_frames_user, int32_t n_frames,
                                    int64_t total_rays, sirius_ray_result* d_results, float* d_image, float* d_spectra,
                                    void* stream) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_frames_user || n_frames <= 0 || total_rays <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    // frames arrive in device memory: bring the small descriptors to the host to derive constants
    std::vector<sirius_frame> hf(n_frames);
    CK(cudaMemcpyAsync(hf.data(), d_frames_user, n_frames * sizeof(sirius_frame), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    long long total = 0;
    cudaStream_t keep = H->stream;
    H->stream = st;
    int rc = upload_frames(H, hf.data(), n_frames, &total);
    H->stream = keep;
    if (rc != SIRIUS_OK) return rc;
    if (total != total_rays) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "total_rays does not match the frames");
    CK(cudaEventRecord(H->ev[0], st));
    rc = launch_frames(H, n_frames, total, d_results, d_image, d_spectra, st, true);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaEventRecord(H->ev[3], st));
    H->pending = true;
    H->pending_stream = st;
    H->pending_total = total;
    return SIRIUS_OK;
}

int sirius_cuda_prepare_frames(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                               int64_t* total_rays) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (!H->configured) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_configure has not been called");
    if (H->cfg.samples_per_pixel > 1)
        return fail(H, SIRIUS_ERR_UNSUPPORTED, "prepared frames trace one sample per pixel");
    CK(cudaSetDevice(H->device));
    long long total = 0;
    int rc = upload_frames(H, frames, n_frames, &total);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaStreamSynchronize(H->stream));
    // one allocation: descriptors | queue words | status | flux tables (256-byte aligned parts)
    auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t o_q = up(size_t(n_frames) * sizeof(FrameDev)), o_s = o_q + up(8 * sizeof(unsigned long long)),
                 o_f = o_s + up(sizeof(int)), bytes = o_f + size_t(n_frames) * kFluxTable * sizeof(float);
    if (H->d_prep) CK(cudaFree(H->d_prep));
    H->d_prep = nullptr;
    H->prep_n_frames = 0;
    CK(cudaMalloc((void**)&H->d_prep, bytes));
    H->prep.frames = reinterpret_cast<FrameDev*>(H->d_prep);
    H->prep.queue = reinterpret_cast<unsigned long long*>(H->d_prep + o_q);
    H->prep.status = reinterpret_cast<int*>(H->d_prep + o_s);
    H->prep.flux = reinterpret_cast<float*>(H->d_prep + o_f);
    CK(cudaMemcpy(const_cast<FrameDev*>(H->prep.frames), H->frames_host.data(), size_t(n_frames) * sizeof(FrameDev),
                  cudaMemcpyHostToDevice));
    H->prep_frame0 = H->frames_host[0];
    H->prep_n_frames = n_frames;
    H->prep_family_mask = H->family_mask;
    H->prep_total = total;
    if (total_rays) *total_rays = total;
    return SIRIUS_OK;
}

int sirius_cuda_launch_prepared(sirius_cuda_handle h, sirius_ray_result* d_results, float* d_image, float* d_spectra,
                                void* stream) {
    Handle* H = static_cast<Handle*>(h);
    if (!H) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (H->prep_n_frames <= 0) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_prepare_frames has not been called");
    if (H->cfg.samples_per_pixel > 1)
        return fail(H, SIRIUS_ERR_UNSUPPORTED, "prepared frames trace one sample per pixel");
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    H->frame0 = H->prep_frame0;
    H->family_mask = H->prep_family_mask;
    return launch_trace(H, H->prep_n_frames, H->prep_total, d_results, d_image, d_spectra, nullptr, st, false,
                        &H->prep);
}

int sirius_cuda_trace_beams(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                            sirius_beam_result* results) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0 || !results) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (!H->configured) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_configure has not been called");
    for (int i = 0; i < n_frames; ++i)
        if (frames[i].metric.family != SIRIUS_METRIC_KERR_SCHILD)
            return fail(H, SIRIUS_ERR_UNSUPPORTED, "beams are traced for the Kerr-Schild family");
    CK(cudaSetDevice(H->device));
    long long total = 0;
    int rc = upload_frames(H, frames, n_frames, &total);
    if (rc != SIRIUS_OK) return rc;
    TmpGuard tmp(H);
    if ((rc = ensure(H, H->d_tmp, H->tmp_cap, size_t(total) * sizeof(sirius_beam_result))) != SIRIUS_OK) return rc;
    sirius_beam_result* d_out = reinterpret_cast<sirius_beam_result*>(H->d_tmp);
    BeamParams B{};
    B.frames = H->d_frames;
    B.n_frames = n_frames;
    B.total = total;
    B.c = make_cfg(H->cfg);
    B.out = d_out;
    B.watchdog_ns = H->cfg.watchdog_ms > 0 ? (unsigned long long)H->cfg.watchdog_ms * 1000000ull : ~0ull;
    B.status = H->d_status;
    cudaError_t e = cudaMemsetAsync(H->d_status, 0, sizeof(int), H->stream);
    if (e == cudaSuccess) {
        const int grid = int((total + 31) / 32);  // two lanes per beam
        if (H->family_mask & (1 << SIRIUS_METRIC_KERR_SCHILD)) beam_kernel<false><<<grid, 64, 0, H->stream>>>(B);
        if (H->family_mask & (1 << kClassRing)) beam_kernel<true><<<grid, 64, 0, H->stream>>>(B);
        e = cudaGetLastError();
    }
    int status = 0;
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(results, d_out, size_t(total) * sizeof(sirius_beam_result), cudaMemcpyDeviceToHost,
                            H->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&status, H->d_status, sizeof(int), cudaMemcpyDeviceToHost, H->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(H->stream);
    if (e != cudaSuccess) return fail(H, SIRIUS_ERR_CUDA, std::string("beam trace: ") + cudaGetErrorString(e));
    if (status & 1) return fail(H, SIRIUS_ERR_TIMEOUT, "beam kernel stopped by its watchdog");
    return SIRIUS_OK;
}

int sirius_cuda_trace_frames_static(sirius_cuda_handle h, const sirius_frame* d_frames_user, int32_t n_frames,
                                    int64_t total_rays, sirius_ray_result* d_results, float* d_image, float* d_spectra,
                                    void* stream) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_frames_user || n_frames <= 0 || total_rays <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (n_frames > SIRIUS_STATIC_MAX_FRAMES)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "sirius_cuda_trace_frames_static takes at most "
                                                    "SIRIUS_STATIC_MAX_FRAMES (64) frames per call");
    if (H->device < 0 || H->device >= kStaticMaxDevices)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "device ordinal beyond the static scratch table");
    if (H->cfg.samples_per_pixel > 1)
        return fail(H, SIRIUS_ERR_UNSUPPORTED, "sirius_cuda_trace_frames_static traces one sample per pixel");
    CK(cudaSetDevice(H->device));
    StaticScratch* scratch = static_scratch(H->device);
    if (!scratch) return fail(H, SIRIUS_ERR_CUDA, "cudaGetSymbolAddress failed for the static scratch");
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    // frame descriptors: device -> host (stack) -> per-frame constants -> static scratch
    sirius_frame hf[SIRIUS_STATIC_MAX_FRAMES];
    FrameDev fd[SIRIUS_STATIC_MAX_FRAMES];
    CK(cudaMemcpyAsync(hf, d_frames_user, n_frames * sizeof(sirius_frame), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    long long total = 0;
    int mask = 0;
    for (int i = 0; i < n_frames; ++i) {
        const sirius_frame& f = hf[i];
        int rc = validate_frame(H, f);
        if (rc != SIRIUS_OK) return rc;
        if (f.ray_offset != total)
            return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "frames must be contiguous: ray_offset[i] = sum of previous pixel counts");
        fd[i] = make_frame(f, H->cfg);
        fd[i].flux_slot = i;
        total += fd[i].n_rays;
        mask |= 1 << fd[i].cls;
    }
    if (total != total_rays) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "total_rays does not match the frames");
    // a pageable source: the copy has been staged when cudaMemcpyAsync returns
    CK(cudaMemcpyAsync(scratch->frames, fd, n_frames * sizeof(FrameDev), cudaMemcpyHostToDevice, st));
    // the launch reads the family mask and the one-frame parameter copy from the
    // handle; the handle's own upload and the statistics of its last traced call
    // are left as they were
    const int saved_mask = H->family_mask;
    const FrameDev saved_frame0 = H->frame0;
    const sirius_launch_stats saved_stats = H->stats;
    H->family_mask = mask;
    H->frame0 = fd[0];
    const LaunchScratch ls{scratch->frames, scratch->queue, &scratch->status, scratch->flux};
    const int rc = launch_trace(H, n_frames, total, d_results, d_image, d_spectra, nullptr, st, false, &ls);
    H->family_mask = saved_mask;
    H->frame0 = saved_frame0;
    H->stats = saved_stats;
    return rc;
}

int sirius_cuda_trace_rays(sirius_cuda_handle h, const sirius_metric* metric, double disk_inner, double disk_outer,
                           const sirius_camera_ray* rays, int64_t n_rays, sirius_ray_result* results) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !metric || !rays || !results || n_rays <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    // All rays of one call share the camera origin of the first ray (the CameraRay batch of a frame).
    for (int64_t i = 1; i < n_rays; ++i)
        for (int j = 0; j < 4; ++j)
            if (rays[i].origin[j] != rays[0].origin[j])
                return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "all rays of one call must share the camera origin");
    sirius_frame f{};
    f.metric = *metric;
    f.camera.t = rays[0].origin[0];
    f.camera.r = rays[0].origin[1];
    f.camera.theta = rays[0].origin[2];
    f.camera.phi = rays[0].origin[3];
    f.camera.width = 1;
    f.camera.height = 1;
    f.camera.fov = 30.f;
    f.disk_inner = disk_inner;
    f.disk_outer = disk_outer;
    f.ray_offset = 0;
    cudaStream_t st = H->stream;
    CK(cudaEventRecord(H->ev[0], st));
    long long dummy = 0;
    int rc = upload_frames(H, &f, 1, &dummy);
    if (rc != SIRIUS_OK) return rc;
    if ((rc = ensure(H, H->d_rays, H->rays_cap, size_t(n_rays))) != SIRIUS_OK) return rc;
    if ((rc = ensure(H, H->d_results, H->results_cap, size_t(n_rays))) != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(H->d_rays, rays, size_t(n_rays) * sizeof(sirius_camera_ray), cudaMemcpyHostToDevice, st));
    rc = launch_trace(H, 1, n_rays, H->d_results, nullptr, nullptr, H->d_rays, st, true);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(results, H->d_results, size_t(n_rays) * sizeof(sirius_ray_result), cudaMemcpyDeviceToHost, st));
    CK(cudaEventRecord(H->ev[3], st));
    return finish_stats(H, st, n_rays, true);
}

int sirius_cuda_metric_evaluate(sirius_cuda_handle h, const sirius_metric* metric, const double* positions, int64_t n,
                                int32_t precision, double* g, double* dg) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !metric || !positions || !g || !dg || n <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    int rc = validate_metric(H, *metric);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaSetDevice(H->device));
    TmpGuard tmp(H);
    if ((rc = ensure(H, H->d_tmp, H->tmp_cap, size_t(n) * 84 * sizeof(double))) != SIRIUS_OK) return rc;
    double* dp = reinterpret_cast<double*>(H->d_tmp);
    double *dgp = dp + 4 * size_t(n), *ddg = dgp + 16 * size_t(n);
    cudaStream_t st = H->stream;
    CK(cudaMemcpyAsync(dp, positions, size_t(n) * 4 * sizeof(double), cudaMemcpyHostToDevice, st));
    metric_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(make_metric(*metric), dp, n, precision == SIRIUS_PRECISION_MIXED,
                                                               dgp, ddg);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(g, dgp, size_t(n) * 16 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(dg, ddg, size_t(n) * 64 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return SIRIUS_OK;
}

int sirius_cuda_dp45_step(sirius_cuda_handle h, const sirius_metric* metric, double* state, double* hh, int32_t* accepted,
                          double* err, int64_t n) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !metric || !state || !hh || !accepted || !err || n <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    int rc = validate_metric(H, *metric);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaSetDevice(H->device));
    TmpGuard tmp(H);
    if ((rc = ensure(H, H->d_tmp, H->tmp_cap, size_t(n) * (10 * sizeof(double) + sizeof(int)))) != SIRIUS_OK) return rc;
    double* ds = reinterpret_cast<double*>(H->d_tmp);
    double *dh = ds + 8 * size_t(n), *de = dh + n;
    int* da = reinterpret_cast<int*>(de + n);
    cudaStream_t st = H->stream;
    CK(cudaMemcpyAsync(ds, state, size_t(n) * 8 * sizeof(double), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dh, hh, size_t(n) * sizeof(double), cudaMemcpyHostToDevice, st));
    dp45_step_kernel<<<unsigned((n + 127) / 128), 128, 0, st>>>(make_metric(*metric), make_cfg(H->cfg), ds, dh, da, de, n);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(state, ds, size_t(n) * 8 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(hh, dh, size_t(n) * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(err, de, size_t(n) * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(accepted, da, size_t(n) * sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return SIRIUS_OK;
}

int sirius_cuda_last_stats(sirius_cuda_handle h, sirius_launch_stats* out) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !out) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (H->pending) {  // a stream-ordered launch: wait for it and read its counters and events
        H->pending = false;
        CK(cudaSetDevice(H->device));
        const int rc = finish_stats(H, H->pending_stream, H->pending_total, true);
        *out = H->stats;
        return rc;
    }
    *out = H->stats;
    return SIRIUS_OK;
}

int sirius_cuda_autotune(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames, sirius_trace_config* out) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    long long total = 0;
    int rc = upload_frames(H, frames, n_frames, &total);
    if (rc != SIRIUS_OK) return rc;
    if ((rc = ensure(H, H->d_image, H->image_cap, size_t(total))) != SIRIUS_OK) return rc;
    const sirius_trace_config base = H->cfg;
    // (blocks/SM, threshold, register cap, rays per thread): blocks/SM 0 is the
    // one-thread-per-ray launch at a register cap (0: the default), with one ray
    // or two packed rays per thread (mixed DP45 over Kerr-Schild frames)
    const int candidates[][4] = {{0, 1, 0, 1},   {0, 1, 255, 1}, {0, 1, 168, 1}, {0, 1, 128, 1}, {0, 1, 255, 2},
                                 {0, 1, 168, 2}, {1, 1, 0, 1},   {2, 1, 0, 1},   {3, 1, 0, 1},   {4, 1, 0, 1},
                                 {2, 4, 0, 1},   {2, 8, 0, 1},   {3, 4, 0, 1}};
    const bool pairs = base.precision == SIRIUS_PRECISION_MIXED && base.integrator == SIRIUS_INTEGRATOR_DP45 &&
                       H->family_mask == (1 << SIRIUS_METRIC_KERR_SCHILD);
    double best = 1e300;
    sirius_trace_config best_cfg = base;
    for (const auto& cand : candidates) {
        if (cand[3] == 2 && !pairs) continue;
        H->cfg = base;
        H->cfg.blocks_per_sm = cand[0];
        H->cfg.refill_threshold = cand[1];
        H->cfg.max_registers = cand[2];
        H->cfg.rays_per_thread = cand[3];
        CK(cudaEventRecord(H->ev[0], H->stream));
        rc = launch_trace(H, n_frames, total, nullptr, H->d_image, nullptr, nullptr, H->stream, true);
        if (rc != SIRIUS_OK) { H->cfg = base; return rc; }
        CK(cudaEventRecord(H->ev[3], H->stream));
        rc = finish_stats(H, H->stream, total, true);
        if (rc != SIRIUS_OK) { H->cfg = base; return rc; }
        if (H->stats.kernel_ms < best) { best = H->stats.kernel_ms; best_cfg = H->cfg; }
    }
    H->cfg = best_cfg;
    if (out) *out = best_cfg;
    return SIRIUS_OK;
}

int sirius_cuda_measure_fma_peak(sirius_cuda_handle h, int32_t precision, double* flops_per_s) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !flops_per_s) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    const int block = 256, iters = 2048;
    const int grid = H->num_sms * 8;
    double* dout = nullptr;
    CK(cudaMalloc((void**)&dout, sizeof(double)));
    float best = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        CK(cudaEventRecord(H->ev[0], H->stream));
        if (precision == 0) fma_peak_kernel<double><<<grid, block, 0, H->stream>>>(dout, iters, 1.0);
        else fma_peak_kernel<float><<<grid, block, 0, H->stream>>>((float*)dout, iters, 1.0f);
        CK(cudaGetLastError());
        CK(cudaEventRecord(H->ev[1], H->stream));
        CK(cudaEventSynchronize(H->ev[1]));
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, H->ev[0], H->ev[1]));
        if (rep > 0) best = std::min(best, ms);
    }
    cudaFree(dout);
    const double flops = 2.0 * 8.0 * 16.0 * double(iters) * double(grid) * double(block);
    *flops_per_s = flops / (double(best) * 1e-3);
    return SIRIUS_OK;
}

int sirius_cuda_surrogate_load(sirius_cuda_handle h, const float* params, int64_t n_params) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !params) return SIRIUS_ERR_INVALID_ARGUMENT;
    if (n_params != surrogate::kParams)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "surrogate parameter count must be SIRIUS_SURROGATE_PARAMS");
    CK(cudaSetDevice(H->device));
    std::vector<unsigned char> img(surrogate::kImageBytes);
    surrogate::pack_weights(params, img.data());
    // (kept by the handle once all of it is there: a first load that failed leaves no weights)
    using Buffer = std::unique_ptr<unsigned char, cudaError_t (*)(void*)>;
    Buffer w(nullptr, cudaFree), e(nullptr, cudaFree);
    unsigned char* d_w = H->d_surrogate;
    if (!d_w) {
        void* p = nullptr;
        if (cudaMalloc(&p, surrogate::kImageBytes) != cudaSuccess)
            return fail(H, SIRIUS_ERR_OUT_OF_MEMORY, "cudaMalloc surrogate weights");
        w.reset(d_w = static_cast<unsigned char*>(p));
        if (cudaMalloc(&p, 16 * sizeof(int)) != cudaSuccess)
            return fail(H, SIRIUS_ERR_OUT_OF_MEMORY, "cudaMalloc surrogate status");
        e.reset(static_cast<unsigned char*>(p));
        CK(cudaMemsetAsync(p, 0, 16 * sizeof(int), H->stream));
        CK(cudaFuncSetAttribute(surrogate::mlp_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                surrogate::kPairSmBytes));
    }
    CK(cudaMemcpyAsync(d_w, img.data(), surrogate::kImageBytes, cudaMemcpyHostToDevice, H->stream));
    CK(cudaStreamSynchronize(H->stream));
    if (w) {
        H->d_surrogate = w.release();
        H->d_sur_err = reinterpret_cast<int*>(e.release());
    }
    return SIRIUS_OK;
}

// bound on any wait inside the MLP kernel: the configured watchdog (default 30 s)
static unsigned long long surrogate_wait_ns(const Handle* H) {
    return (unsigned long long)(H->cfg.watchdog_ms > 0 ? H->cfg.watchdog_ms : 30000) * 1000000ull;
}

// launches the MLP on n feature rows (device buffers) on stream st
static int surrogate_launch(Handle* H, const float* d_features, long long n, float* d_out, cudaStream_t st,
                            const unsigned* rows = nullptr) {
    if (!H->d_surrogate) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "no surrogate weights loaded");
    if (n <= 0) return SIRIUS_OK;
    const long long tiles = (n + 2 * surrogate::kTileM - 1) / (2 * surrogate::kTileM);
    const int grid = 2 * int(std::min<long long>(tiles, std::max(H->num_sms / 2, 1)));  // a pair of CTAs per tile
    // (the kernel leaves the counter at zero)
    unsigned long long* counter = reinterpret_cast<unsigned long long*>(H->d_sur_err + 2);
    surrogate::mlp_pair_kernel<<<grid, surrogate::kPairThreads, surrogate::kPairSmBytes, st>>>(
        H->d_surrogate, d_features, n, d_out, H->d_sur_err, counter, surrogate_wait_ns(H), rows);
    CK(cudaGetLastError());
    return SIRIUS_OK;
}

// The MLP launches of one call. None of the handle's others is in flight when it begins: every call
// waits for its own, also where it ends early with an error (the destructor).
struct SurrogateCall {
    Handle* H;
    cudaStream_t st;
    bool open = false;
    std::chrono::steady_clock::time_point start{};

    SurrogateCall(Handle* h, cudaStream_t s) : H(h), st(s) {}
    SurrogateCall(const SurrogateCall&) = delete;
    SurrogateCall& operator=(const SurrogateCall&) = delete;

    // before the launches: after an error the flag and the tile counter start over
    int begin() {
        if (!H->d_sur_err) return SIRIUS_OK;
        if (H->sur_failed) CK(cudaMemsetAsync(H->d_sur_err, 0, 16 * sizeof(int), st));
        H->sur_failed = false;
        open = true;
        start = std::chrono::steady_clock::now();
        return SIRIUS_OK;
    }

    // The kernels' error flag, once their stream has been waited for. A wait that runs out takes
    // its whole bound, and it began after the call did: a call that ended within half the bound
    // (the two clocks are not compared any closer) has no flag to read. That saves the copy (with the
    // memsets, which the kernel's own counter made needless, 1000 rows 36 -> 27 us) without page-locked
    // memory for the flag (1.4 to 3 ms to allocate with a new handle's weights). Bounds below 100 ms
    // always read it.
    int finish() {
        if (!open) return SIRIUS_OK;
        const double limit = double(surrogate_wait_ns(H));
        const double took = std::chrono::duration<double, std::nano>(std::chrono::steady_clock::now() - start).count();
        int err = 0;
        if (limit < 1e8 || took >= 0.5 * limit) {
            CK(cudaMemcpyAsync(&err, H->d_sur_err, sizeof(int), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
        }
        open = false;
        if (!err) return SIRIUS_OK;
        H->sur_failed = true;
        return fail(H, SIRIUS_ERR_TIMEOUT, "surrogate MLP kernel stopped by its wait bound");
    }

    ~SurrogateCall() {
        if (!open) return;
        H->sur_failed = true;
        cudaStreamSynchronize(st);
        for (auto& q : H->sur_stream)
            if (q) cudaStreamSynchronize(q);
        cudaGetLastError();  // (the call has its error)
    }
};

int sirius_cuda_surrogate_infer(sirius_cuda_handle h, const float* d_features, int64_t n, float* d_out,
                                void* stream) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_features || !d_out || n < 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    SurrogateCall mlp(H, st);
    int rc = mlp.begin();
    if (rc != SIRIUS_OK) return rc;
    if ((rc = surrogate_launch(H, d_features, n, d_out, st)) != SIRIUS_OK) return rc;
    CK(cudaStreamSynchronize(st));
    return mlp.finish();
}

// ---- surrogate training ----
void sirius_cuda_default_train_config(sirius_train_config* c) {
    if (!c) return;
    std::memset(c, 0, sizeof(*c));
    c->batch = 16384;
    c->total_steps = 1;
    c->max_lr = 2e-3f;
    c->warmup_fraction = 0.05f;
    c->beta1 = 0.9f;
    c->beta2 = 0.999f;
    c->eps = 1e-8f;
    c->weight_decay = 0.f;
    c->seed = 0;
}

int sirius_cuda_train_init(sirius_cuda_handle h, const float* params, const sirius_train_config* cfg) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !params || !cfg) return SIRIUS_ERR_INVALID_ARGUMENT;
    const sirius_train_config& c = *cfg;
    if (c.batch <= 0 || c.batch % 128 != 0 || c.batch > (1 << 20))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "batch must be a positive multiple of 128, at most 2^20");
    if (c.total_steps < 1) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "total_steps must be >= 1");
    if (!(c.max_lr > 0.f) || !std::isfinite(c.max_lr) || !(c.warmup_fraction >= 0.f && c.warmup_fraction <= 1.f) ||
        !(c.beta1 >= 0.f && c.beta1 < 1.f) || !(c.beta2 >= 0.f && c.beta2 < 1.f) || !(c.eps > 0.f) ||
        !(c.weight_decay >= 0.f))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "invalid optimiser settings");
    for (long long i = 0; i < surrogate::kParams; ++i)
        if (!std::isfinite(params[i])) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "non-finite initial parameter");
    CK(cudaSetDevice(H->device));
    if (!H->train) {
        std::unique_ptr<TrainState, void (*)(TrainState*)> T(new (std::nothrow) TrainState, train_free);
        if (!T) return fail(H, SIRIUS_ERR_OUT_OF_MEMORY, "training state");
        const size_t pb = surrogate::kParams * sizeof(float);
        CK(cudaMalloc((void**)&T->params, pb));
        CK(cudaMalloc((void**)&T->grad, pb));
        CK(cudaMalloc((void**)&T->m1, pb));
        CK(cudaMalloc((void**)&T->m2, pb));
        CK(cudaMalloc((void**)&T->wbf, train::kBfTotal * sizeof(__nv_bfloat16)));
        CK(cudaMalloc((void**)&T->st, sizeof(train::StepState)));
        CK(cudaMalloc((void**)&T->err, 4 * sizeof(int)));
        CK(cudaStreamCreateWithFlags(&T->side, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&T->fork, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&T->join, cudaEventDisableTiming));
        const int rc = train_set_attributes(H);
        if (rc != SIRIUS_OK) return rc;
        H->train = T.release();
    }
    TrainState* T = H->train;
    const long long w[4] = {train::kBfW2, train::kBfW3, train::kBfW4, train::kBfW5};
    T->tma = true;
    for (int l = 0; l < 4; ++l)
        T->tma = T->tma && kmajor_map(&T->wmap[l], T->wbf + w[l], l < 3 ? 256 : 16, 256, 256, l < 3 ? 128 : 8);
    train_drop_graph(T);  // the captured step embeds the configuration
    T->cfg = c;
    const int rc = train_rows(H, T, c.batch);
    if (rc != SIRIUS_OK) return rc;
    const size_t pb = surrogate::kParams * sizeof(float);
    CK(cudaMemcpyAsync(T->params, params, pb, cudaMemcpyHostToDevice, H->stream));
    CK(cudaMemsetAsync(T->grad, 0, pb, H->stream));
    CK(cudaMemsetAsync(T->m1, 0, pb, H->stream));
    CK(cudaMemsetAsync(T->m2, 0, pb, H->stream));
    CK(cudaMemsetAsync(T->wbf, 0, train::kBfTotal * sizeof(__nv_bfloat16), H->stream));
    CK(cudaMemsetAsync(T->st, 0, sizeof(train::StepState), H->stream));
    CK(cudaMemsetAsync(T->err, 0, 4 * sizeof(int), H->stream));
    train::weights_to_bf16_kernel<<<H->num_sms, 256, 0, H->stream>>>(T->params, T->wbf);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(H->stream));
    T->ready = true;
    return SIRIUS_OK;
}

int sirius_cuda_train_steps(sirius_cuda_handle h, const float* d_features, const float* d_targets,
                            const float* d_weights, int64_t n_rows, int64_t n_steps, float* device_ms) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_features || !d_targets || !d_weights || n_steps < 0) return SIRIUS_ERR_INVALID_ARGUMENT;
    TrainState* T = H->train;
    if (!train_ready(T)) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_train_init has not succeeded");
    if (n_rows < T->cfg.batch || n_rows > (1LL << 40))
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "n_rows must hold at least one batch");
    CK(cudaSetDevice(H->device));
    if (T->graph && (T->key[0] != d_features || T->key[1] != d_targets || T->key[2] != d_weights ||
                     T->key_rows != n_rows))
        train_drop_graph(T);
    if (!T->graph) {
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(H->stream, cudaStreamCaptureModeThreadLocal));
        train_step(H, T, d_features, d_targets, d_weights, n_rows, H->stream);
        const cudaError_t e1 = cudaStreamEndCapture(H->stream, &g);
        const cudaError_t e0 = cudaGetLastError();
        if (e1 != cudaSuccess || e0 != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            return fail(H, SIRIUS_ERR_CUDA, std::string("capturing the training step: ") +
                                                cudaGetErrorString(e1 != cudaSuccess ? e1 : e0));
        }
        const cudaError_t e2 = cudaGraphInstantiate(&T->graph, g, 0);
        cudaGraphDestroy(g);
        if (e2 != cudaSuccess) {
            T->graph = nullptr;
            return fail(H, SIRIUS_ERR_CUDA, std::string("instantiating the training step: ") + cudaGetErrorString(e2));
        }
        T->key[0] = d_features;
        T->key[1] = d_targets;
        T->key[2] = d_weights;
        T->key_rows = n_rows;
    }
    for (auto& e : H->ev)
        if (!e) CK(cudaEventCreate(&e));
    CK(cudaEventRecord(H->ev[1], H->stream));
    for (int64_t i = 0; i < n_steps; ++i) CK(cudaGraphLaunch(T->graph, H->stream));
    CK(cudaEventRecord(H->ev[2], H->stream));
    const int rc = train_check_err(H, T);
    if (rc == SIRIUS_OK && device_ms) CK(cudaEventElapsedTime(device_ms, H->ev[1], H->ev[2]));
    return rc;
}

int sirius_cuda_train_evaluate(sirius_cuda_handle h, const float* d_features, const float* d_targets,
                               const float* d_weights, int64_t n_rows, float* loss_parts) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_features || !d_targets || !d_weights || !loss_parts || n_rows <= 0)
        return SIRIUS_ERR_INVALID_ARGUMENT;
    TrainState* T = H->train;
    if (!train_ready(T)) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_train_init has not succeeded");
    CK(cudaSetDevice(H->device));
    double acc[4] = {0, 0, 0, 0};
    for (long long r0 = 0; r0 < n_rows; r0 += T->cfg.batch) {
        const int rows = int(std::min<long long>(T->cfg.batch, n_rows - r0));
        train::gather_kernel<<<(rows + 255) / 256, 256, 0, H->stream>>>(d_features, d_targets, d_weights, n_rows,
                                                                        rows, 1, 0, 1, r0, T->st, T->x0, T->t, T->w);
        train_forward(H, T, rows, H->stream);
        train_loss(T, rows, false, H->stream);
        CK(cudaGetLastError());
        float sums[8];
        CK(cudaMemcpyAsync(sums, T->st->sums, sizeof(sums), cudaMemcpyDeviceToHost, H->stream));
        CK(cudaStreamSynchronize(H->stream));
        for (int j = 0; j < 4; ++j) acc[j] += double(sums[2 + j]) * rows;
    }
    for (int j = 0; j < 4; ++j) loss_parts[j] = float(acc[j] / double(n_rows));
    return train_check_err(H, T);
}

int sirius_cuda_train_gradient(sirius_cuda_handle h, const float* d_features, const float* d_targets,
                               const float* d_weights, int64_t n_rows, float* loss_parts, float* grad) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !d_features || !d_targets || !d_weights || !grad) return SIRIUS_ERR_INVALID_ARGUMENT;
    TrainState* T = H->train;
    if (!train_ready(T)) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_train_init has not succeeded");
    if (n_rows <= 0 || n_rows % 128 != 0 || n_rows > T->cfg.batch)
        return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "n_rows must be a positive multiple of 128, at most the batch");
    CK(cudaSetDevice(H->device));
    const int rows = int(n_rows);
    train::gather_kernel<<<(rows + 255) / 256, 256, 0, H->stream>>>(d_features, d_targets, d_weights, n_rows, rows,
                                                                    1, 0, 1, 0, T->st, T->x0, T->t, T->w);
    train_forward(H, T, rows, H->stream);
    train_loss(T, rows, true, H->stream);
    train_backward(H, T, rows, H->stream);
    CK(cudaGetLastError());
    float sums[8];
    CK(cudaMemcpyAsync(sums, T->st->sums, sizeof(sums), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaMemcpyAsync(grad, T->grad, surrogate::kParams * sizeof(float), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaMemsetAsync(T->grad, 0, surrogate::kParams * sizeof(float), H->stream));
    const int rc = train_check_err(H, T);
    if (rc != SIRIUS_OK) return rc;
    if (loss_parts)
        for (int j = 0; j < 4; ++j) loss_parts[j] = sums[2 + j];
    return SIRIUS_OK;
}

int sirius_cuda_train_params(sirius_cuda_handle h, float* params, int64_t* steps) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !params) return SIRIUS_ERR_INVALID_ARGUMENT;
    TrainState* T = H->train;
    if (!T || !T->ready) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "sirius_cuda_train_init has not succeeded");
    CK(cudaSetDevice(H->device));
    long long st = 0;
    CK(cudaMemcpyAsync(params, T->params, surrogate::kParams * sizeof(float), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaMemcpyAsync(&st, &T->st->step, sizeof(st), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaStreamSynchronize(H->stream));
    if (steps) *steps = st;
    return SIRIUS_OK;
}

// Per-frame constants of the surrogate gate: the camera's Boyer-Lindquist
// polar angle and the critical curve (Bardeen 1973: spherical photon orbits
// r in [r_ph,pro, r_ph,retro] give xi = L/E, eta = Q/E^2; alpha = -xi/sin(theta_o),
// beta = +-sqrt(eta + a^2 cos^2 theta_o - xi^2 cot^2 theta_o)), resampled at
// kCurveN angles about its centre.
static SurFrameDev make_sur_frame(const sirius_frame& f, const FrameDev& F, bool curve = true) {
    SurFrameDev S{};
    const sirius_metric& m = f.metric;
    const double x = F.cam_r * F.cam_st * F.cam_cp, y = F.cam_r * F.cam_st * F.cam_sp, z = F.cam_r * F.cam_ct;
    const double a = m.a, M = m.M;
    const double R2 = x * x + y * y + z * z, Rm2 = R2 - a * a;
    const double rk = std::sqrt(std::max(0.5 * (Rm2 + std::sqrt(Rm2 * Rm2 + 4.0 * a * a * z * z)), 1e-20));
    const double th = std::acos(std::clamp(z / rk, -1.0, 1.0));
    S.sin_o = std::max(std::sin(th), 1e-6);
    S.theta_deg = th * 180.0 / kPi;
    // the MLP was fitted to static-observer Kerr frames; other frames are integrated in full
    S.kerr = (m.family == SIRIUS_METRIC_KERR_SCHILD && F.has_horizon && m.Q == 0.0 && m.Lambda == 0.0 &&
              F.observer == SIRIUS_OBSERVER_STATIC) ? 1 : 0;
    if (!S.kerr || !curve) return S;
    std::vector<std::pair<double, double>> pts;
    const double co = std::cos(th), cot = co / S.sin_o;
    if (std::fabs(a) < 1e-6 * M) {
        const double R = std::sqrt(27.0) * M;
        for (int i = 0; i < 1024; ++i) {
            const double t = 2.0 * kPi * i / 1024.0;
            pts.push_back({R * std::cos(t), R * std::sin(t)});
        }
    } else {
        const double as = std::clamp(std::fabs(a) / M, 0.0, 1.0);
        const double r0 = 2.0 * M * (1.0 + std::cos((2.0 / 3.0) * std::acos(-as)));
        const double r1 = 2.0 * M * (1.0 + std::cos((2.0 / 3.0) * std::acos(as)));
        for (int i = 0; i <= 1024; ++i) {
            const double r = r0 + (r1 - r0) * i / 1024.0;
            const double xi = (r * r * (3.0 * M - r) - a * a * (r + M)) / (a * (r - M));
            const double eta = r * r * r * (4.0 * a * a * M - r * (r - 3.0 * M) * (r - 3.0 * M)) / (a * a * (r - M) * (r - M));
            const double b2 = eta + a * a * co * co - xi * xi * cot * cot;
            if (b2 < 0.0) continue;
            const double al = -xi / S.sin_o, be = std::sqrt(b2);
            pts.push_back({al, be});
            pts.push_back({al, -be});
        }
    }
    if (pts.size() < 64) { S.kerr = 0; return S; }
    double amin = 1e300, amax = -1e300;
    for (auto& q : pts) { amin = std::min(amin, q.first); amax = std::max(amax, q.first); }
    const double ac = 0.5 * (amin + amax);
    S.ac = float(ac);
    std::vector<std::pair<double, std::pair<double, double>>> polar;
    for (auto& q : pts) polar.push_back({std::atan2(q.second, q.first - ac), q});
    std::sort(polar.begin(), polar.end(), [](const auto& u, const auto& v) { return u.first < v.first; });
    const size_t np = polar.size();
    size_t k = 0;
    for (int j = 0; j < kCurveN; ++j) {
        const double phi = -kPi + 2.0 * kPi * (j + 0.5) / kCurveN;
        while (k < np && polar[k].first < phi) ++k;
        const auto& hi = polar[k % np];
        const auto& lo = polar[(k + np - 1) % np];
        double p0 = lo.first, p1 = hi.first;
        if (k == 0) p0 -= 2.0 * kPi;
        if (k == np) p1 += 2.0 * kPi;
        const double w = p1 > p0 ? (phi - p0) / (p1 - p0) : 0.0;
        S.ca[j] = float(lo.second.first + w * (hi.second.first - lo.second.first));
        S.cb[j] = float(lo.second.second + w * (hi.second.second - lo.second.second));
    }
    return S;
}

// Stage 1 for the uploaded frames: the per-frame constants the features need
// (camera inclination) and the features kernel. Its upload comes from pinned
// memory, so the host returns at once and computes the critical curves while
// the kernel runs.
static int surrogate_features_launch(Handle* H, const sirius_frame* frames, int n_frames, long long total,
                                     cudaStream_t st) {
    int rc;
    if (H->h_sur_frames_cap < size_t(2 * n_frames)) {
        if (H->h_sur_frames) CK(cudaFreeHost(H->h_sur_frames));
        H->h_sur_frames = nullptr;
        H->h_sur_frames_cap = 0;
        CK(cudaMallocHost((void**)&H->h_sur_frames, 2 * size_t(n_frames) * sizeof(SurFrameDev)));
        H->h_sur_frames_cap = 2 * size_t(n_frames);
    }
    if ((rc = ensure(H, H->d_sur_frames, H->sur_frames_cap, size_t(n_frames))) != SIRIUS_OK) return rc;
    if ((rc = ensure(H, H->d_feat, H->feat_cap, size_t(total) * 5)) != SIRIUS_OK) return rc;
    for (int i = 0; i < n_frames; ++i) H->h_sur_frames[i] = make_sur_frame(frames[i], make_frame(frames[i], H->cfg), false);
    CK(cudaMemcpyAsync(H->d_sur_frames, H->h_sur_frames, n_frames * sizeof(SurFrameDev), cudaMemcpyHostToDevice, st));
    sur_features_kernel<<<int((total + 255) / 256), 256, 0, st>>>(H->d_frames, H->d_sur_frames, n_frames, total,
                                                                  H->d_feat);
    CK(cudaGetLastError());
    return SIRIUS_OK;
}

// Stage 2: the critical curves (host), the gate, and the list of rays to
// integrate (gated rays, padding to a multiple of 32, audit rays); the two
// list counts are copied into pinned memory (read them once the stream has
// passed this point).
static int surrogate_gate_launch(Handle* H, const sirius_frame* frames, int n_frames, long long total,
                                 const sirius_surrogate_config* sc, unsigned char* d_gate, cudaStream_t st,
                                 bool allow_empty = false) {
    int rc;
    SurFrameDev* full = H->h_sur_frames + n_frames;
    for (int i = 0; i < n_frames; ++i) full[i] = make_sur_frame(frames[i], make_frame(frames[i], H->cfg));
    if ((rc = ensure(H, H->d_list, H->list_cap, size_t(total) + 32)) != SIRIUS_OK) return rc;
    const int block = 256;
    const int n_blocks = int((total + block - 1) / block);
    // per block: gated, audit and MLP-row counts; after the scan, offsets, with
    // [n_blocks] = gated total, [2 n_blocks] = gated + audit, [3 n_blocks] = + MLP rows
    if ((rc = ensure(H, H->d_block_counts, H->block_counts_cap, 3 * size_t(n_blocks) + 1)) != SIRIUS_OK) return rc;
    if (!d_gate) {
        if ((rc = ensure(H, H->d_gate, H->gate_cap, size_t(total))) != SIRIUS_OK) return rc;
        d_gate = H->d_gate;
    }
    if (!H->h_list_len) CK(cudaMallocHost((void**)&H->h_list_len, 3 * sizeof(unsigned)));
    const double band = sc ? sc->gate_band : 0.3;
    const double audit = sc ? std::clamp(sc->audit_fraction, 0.0, 1.0) : 0.01;
    const unsigned thr = unsigned(std::min(audit * 4294967296.0, 4294967295.0));
    const unsigned seed = sc ? sc->audit_seed : 0u;
    // the coarse MLP pass of the inner-disk gate and of the empty pixels (after the
    // descriptors above reach the device)
    const double inner = sc ? (sc->inner_gate == 0.f ? kInnerGateDefault : double(sc->inner_gate)) : kInnerGateDefault;
    const bool empty = allow_empty && H->d_surrogate && !(sc && sc->empty_skip < 0);
    H->last_empty_skip = empty;
    const int stride = (sc && sc->coarse_stride > 0) ? sc->coarse_stride : kCoarseStrideDefault;
    long long n_coarse = 0;
    if ((inner > 0.0 || empty) && H->d_surrogate) {  // without weights (features only) there is no coarse pass
        for (int i = 0; i < n_frames; ++i) {
            const FrameDev F = make_frame(frames[i], H->cfg);
            const long long rows = F.n_rays / F.width;
            full[i].coarse_offset = n_coarse;
            full[i].cw = (F.width + stride - 1) / stride;
            full[i].ch = int((rows + stride - 1) / stride);
            full[i].r1_max = full[i].kerr && inner > 0.0 ? float(inner * F.disk_in) : 0.f;
            n_coarse += (long long)full[i].cw * full[i].ch;
        }
    }
    CK(cudaMemcpyAsync(H->d_sur_frames, full, n_frames * sizeof(SurFrameDev), cudaMemcpyHostToDevice, st));
    if (n_coarse > 0) {
        if ((rc = ensure(H, H->d_coarse_feat, H->coarse_feat_cap, size_t(n_coarse) * 5)) != SIRIUS_OK) return rc;
        if ((rc = ensure(H, H->d_coarse_out, H->coarse_out_cap, size_t(n_coarse) * 4)) != SIRIUS_OK) return rc;
        sur_coarse_gather_kernel<<<int((n_coarse + 255) / 256), 256, 0, st>>>(H->d_frames, H->d_sur_frames, n_frames,
                                                                            stride, n_coarse, H->d_feat,
                                                                            H->d_coarse_feat);
        CK(cudaGetLastError());
        if ((rc = surrogate_launch(H, H->d_coarse_feat, n_coarse, H->d_coarse_out, st)) != SIRIUS_OK) return rc;
    }
    H->last_coarse = n_coarse;
    // one frame in 16 x 16 pixel tiles: the list of gated rays in tile order
    int tile_w = 0;
    if (n_frames == 1) {
        const FrameDev F = make_frame(frames[0], H->cfg);
        if (F.width % 16 == 0 && F.n_rays == total && (total / F.width) % 16 == 0) tile_w = F.width;
    }
    sur_gate_kernel<<<n_blocks, block, 0, st>>>(H->d_frames, H->d_sur_frames, n_frames, total, float(band), thr, seed,
                                                H->d_feat, stride, H->d_coarse_out, d_gate, H->d_block_counts, tile_w,
                                                n_coarse > 0 && empty ? 1 : 0);
    CK(cudaGetLastError());
    sur_scan_kernel<<<1, 1024, 0, st>>>(H->d_block_counts, 3 * n_blocks);
    CK(cudaGetLastError());
    unsigned* rows = nullptr;
    if (empty && n_coarse > 0) {
        if ((rc = ensure(H, H->d_mlp_rows, H->mlp_rows_cap, size_t(total))) != SIRIUS_OK) return rc;
        rows = H->d_mlp_rows;
    }
    H->last_empty_skip = rows != nullptr;
    sur_scatter_kernel<<<n_blocks, block, 0, st>>>(d_gate, total, H->d_block_counts, H->d_list, tile_w, rows);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(H->h_list_len, H->d_block_counts + n_blocks, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(H->h_list_len + 1, H->d_block_counts + 2 * size_t(n_blocks), sizeof(unsigned),
                       cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(H->h_list_len + 2, H->d_block_counts + 3 * size_t(n_blocks), sizeof(unsigned),
                       cudaMemcpyDeviceToHost, st));
    return SIRIUS_OK;
}

static int render_surrogate_pass(Handle* H, const sirius_frame* frames, int n_frames,
                                 const sirius_surrogate_config* sc, float* d_image, float* d_image_mlp,
                                 unsigned char* d_gate, cudaStream_t st, sirius_surrogate_stats* stats) {
    if (!H->d_surrogate) return fail(H, SIRIUS_ERR_NOT_CONFIGURED, "no surrogate weights loaded");
    for (auto& e : H->sev)
        if (!e) CK(cudaEventCreate(&e));
    long long total = 0;
    cudaStream_t keep = H->stream;
    H->stream = st;
    int rc = upload_frames(H, frames, n_frames, &total);
    H->stream = keep;
    if (rc != SIRIUS_OK) return rc;
    if (total > 0xFFFFFFFFll) return fail(H, SIRIUS_ERR_INVALID_ARGUMENT, "surrogate rendering takes < 2^32 rays");
    if ((rc = ensure(H, H->d_mlp_out, H->mlp_out_cap, size_t(total) * 4)) != SIRIUS_OK) return rc;
    if (!d_gate) {
        if ((rc = ensure(H, H->d_gate, H->gate_cap, size_t(total))) != SIRIUS_OK) return rc;
        d_gate = H->d_gate;
    }
    // 1. features, the inner-disk gate's coarse MLP pass, the gate and the
    // compacted list of rays to integrate
    SurrogateCall mlp(H, st);
    if ((rc = mlp.begin()) != SIRIUS_OK) return rc;
    CK(cudaEventRecord(H->sev[0], st));
    if ((rc = surrogate_features_launch(H, frames, n_frames, total, st)) != SIRIUS_OK) return rc;
    if ((rc = surrogate_gate_launch(H, frames, n_frames, total, sc, d_gate, st, d_image_mlp == nullptr)) != SIRIUS_OK)
        return rc;
    // 2. the integrator on the compacted list of gated and audit rays, beside
    // 3. the MLP on every pixel and the shading of the ungated ones. The trace
    // goes first, from a high-priority stream, so its blocks take every free
    // slot; the MLP (low priority, tiles from a counter) fills the SMs that the
    // trace's tail leaves idle, a few long near-critical warps. The shading
    // writes only ungated pixels, so the two never write the same pixel.
    if (!H->sur_stream[0]) {
        int least = 0, greatest = 0;
        CK(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        CK(cudaStreamCreateWithPriority(&H->sur_stream[0], cudaStreamNonBlocking, greatest));
        CK(cudaStreamCreateWithPriority(&H->sur_stream[1], cudaStreamNonBlocking, least));
        for (auto& e : H->fev) CK(cudaEventCreate(&e));
    }
    cudaStream_t s_trace = H->sur_stream[0], s_mlp = H->sur_stream[1];
    if ((rc = ensure(H, H->d_flux, H->flux_cap, size_t(n_frames) * kFluxTable)) != SIRIUS_OK) return rc;
    flux_table_kernel<<<n_frames, kFluxN, 0, st>>>(H->d_frames, H->d_flux);
    CK(cudaGetLastError());
    CK(cudaEventRecord(H->sev[1], st));
    CK(cudaStreamWaitEvent(s_trace, H->sev[1], 0));
    CK(cudaStreamWaitEvent(s_mlp, H->sev[1], 0));
    CK(cudaEventSynchronize(H->sev[1]));
    const unsigned n_gated = H->h_list_len[0], n_int = H->h_list_len[1];
    const long long n_mlp = H->last_empty_skip ? (long long)(H->h_list_len[2] - H->h_list_len[1]) : total;
    const long long n_list = (long long)n_int + ((32 - (n_gated & 31u)) & 31u);
    if (n_int > 0) {
        rc = launch_trace(H, n_frames, n_list, nullptr, d_image, nullptr, nullptr, s_trace, false, nullptr, H->d_list,
                          true);
        if (rc != SIRIUS_OK) return rc;
    }
    CK(cudaEventRecord(H->fev[0], s_trace));
    if ((rc = surrogate_launch(H, H->d_feat, n_mlp, H->d_mlp_out, s_mlp,
                               H->last_empty_skip ? H->d_mlp_rows : nullptr)) != SIRIUS_OK)
        return rc;
    CK(cudaEventRecord(H->fev[1], s_mlp));
    sur_shade_kernel<<<int((total + 255) / 256), 256, 0, s_mlp>>>(H->d_frames, n_frames, total, H->d_mlp_out, d_gate,
                                                                  H->d_flux, d_image, d_image_mlp);
    CK(cudaGetLastError());
    CK(cudaEventRecord(H->fev[2], s_mlp));
    CK(cudaStreamWaitEvent(st, H->fev[0], 0));
    CK(cudaStreamWaitEvent(st, H->fev[2], 0));
    float* audit = reinterpret_cast<float*>(H->d_sur_err + 8);
    CK(cudaMemsetAsync(audit, 0, 5 * sizeof(float), st));
    sur_audit_kernel<<<int((total + 255) / 256), 256, 0, st>>>(d_gate, d_image, H->d_mlp_out, total, audit);
    CK(cudaGetLastError());
    CK(cudaEventRecord(H->sev[4], st));
    int status = 0;
    float aud[5] = {};
    CK(cudaMemcpyAsync(aud, audit, sizeof(aud), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&status, H->d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if ((rc = mlp.finish()) != SIRIUS_OK) return rc;
    if (n_int > 0 && (status & 1)) return fail(H, SIRIUS_ERR_TIMEOUT, "trace kernel stopped by its watchdog");
    if (stats) {
        *stats = sirius_surrogate_stats{};
        stats->rays = total;
        stats->integrated = n_int;
        float tt = 0.f;
        CK(cudaEventElapsedTime(&stats->ms_features, H->sev[0], H->sev[1]));
        CK(cudaEventElapsedTime(&stats->ms_trace, H->sev[1], H->fev[0]));   // concurrent with the MLP
        CK(cudaEventElapsedTime(&stats->ms_mlp, H->sev[1], H->fev[1]));
        CK(cudaEventElapsedTime(&stats->ms_shade, H->fev[1], H->fev[2]));
        CK(cudaEventElapsedTime(&tt, H->sev[0], H->sev[4]));
        stats->ms_total = tt;
        stats->audit_count = int32_t(aud[4]);
        stats->audit_rel_l1 = aud[1] > 0.f ? aud[0] / aud[1] : 0.f;
        stats->audit_rel_max = aud[3] > 0.f ? aud[2] / aud[3] : 0.f;
        stats->coarse_rays = int32_t(std::min<long long>(H->last_coarse, 0x7fffffff));
    }
    return SIRIUS_OK;
}

// The render and the audit's judgement of it: above the caller's budget, one
// more render with the critical-curve band and the inner-disk gate widened.
static int render_surrogate(Handle* H, const sirius_frame* frames, int n_frames, const sirius_surrogate_config* sc,
                            float* d_image, float* d_image_mlp, unsigned char* d_gate, cudaStream_t st,
                            sirius_surrogate_stats* stats) {
    sirius_surrogate_stats first{};
    int rc = render_surrogate_pass(H, frames, n_frames, sc, d_image, d_image_mlp, d_gate, st, &first);
    if (rc != SIRIUS_OK) return rc;
    if (sc && sc->audit_budget > 0.f && first.audit_rel_max > sc->audit_budget) {
        sirius_surrogate_config wide = *sc;
        wide.gate_band = 1.5 * sc->gate_band;
        const float inner = sc->inner_gate == 0.f ? float(kInnerGateDefault) : sc->inner_gate;
        wide.inner_gate = inner > 0.f ? 1.5f * inner : inner;
        sirius_surrogate_stats second{};
        rc = render_surrogate_pass(H, frames, n_frames, &wide, d_image, d_image_mlp, d_gate, st, &second);
        if (rc != SIRIUS_OK) return rc;
        second.rerendered = 1;
        second.ms_total += first.ms_total;
        if (stats) *stats = second;
        return SIRIUS_OK;
    }
    if (stats) *stats = first;
    return SIRIUS_OK;
}

int sirius_cuda_surrogate_features(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                                   const sirius_surrogate_config* sc, float* d_features, uint8_t* d_gate,
                                   void* stream) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0 || !d_features) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    long long total = 0;
    cudaStream_t keep = H->stream;
    H->stream = st;
    int rc = upload_frames(H, frames, n_frames, &total);
    H->stream = keep;
    if (rc != SIRIUS_OK) return rc;
    SurrogateCall mlp(H, st);
    if ((rc = mlp.begin()) != SIRIUS_OK) return rc;
    if ((rc = surrogate_features_launch(H, frames, n_frames, total, st)) != SIRIUS_OK) return rc;
    if ((rc = surrogate_gate_launch(H, frames, n_frames, total, sc, d_gate, st)) != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(d_features, H->d_feat, size_t(total) * 5 * sizeof(float), cudaMemcpyDeviceToDevice, st));
    CK(cudaStreamSynchronize(st));
    return mlp.finish();
}

int sirius_cuda_render_surrogate_device(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                                        const sirius_surrogate_config* sc, float* d_image, float* d_image_mlp,
                                        uint8_t* d_gate, void* stream, sirius_surrogate_stats* stats) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0 || !d_image) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : cudaStreamLegacy;
    return render_surrogate(H, frames, n_frames, sc, d_image, d_image_mlp, d_gate, st, stats);
}

int sirius_cuda_render_surrogate(sirius_cuda_handle h, const sirius_frame* frames, int32_t n_frames,
                                 const sirius_surrogate_config* sc, float* image, float* image_mlp, uint8_t* gate,
                                 sirius_surrogate_stats* stats) {
    Handle* H = static_cast<Handle*>(h);
    if (!H || !frames || n_frames <= 0 || !image) return SIRIUS_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(H->device));
    long long total = 0;
    for (int i = 0; i < n_frames; ++i) total += frame_rays(frames[i]);
    int rc;
    if ((rc = ensure(H, H->d_image, H->image_cap, size_t(total) * (image_mlp ? 2 : 1))) != SIRIUS_OK) return rc;
    if ((rc = ensure(H, H->d_gate, H->gate_cap, size_t(total))) != SIRIUS_OK) return rc;
    float* d_img = H->d_image;
    float* d_mlp = image_mlp ? H->d_image + total : nullptr;
    rc = render_surrogate(H, frames, n_frames, sc, d_img, d_mlp, H->d_gate, H->stream, stats);
    if (rc != SIRIUS_OK) return rc;
    CK(cudaMemcpyAsync(image, d_img, size_t(total) * sizeof(float), cudaMemcpyDeviceToHost, H->stream));
    if (image_mlp) CK(cudaMemcpyAsync(image_mlp, d_mlp, size_t(total) * sizeof(float), cudaMemcpyDeviceToHost, H->stream));
    if (gate) CK(cudaMemcpyAsync(gate, H->d_gate, size_t(total), cudaMemcpyDeviceToHost, H->stream));
    CK(cudaStreamSynchronize(H->stream));
    return SIRIUS_OK;
}

}  // extern "C"
