// Particle-path kernels for sm_100a: geometry (once per camera), Poisson counts fused with a
// single-pass decoupled-lookback scan (per ensemble), the persistent particle kernel with one
// packed 64-bit atomicMin per particle, the splat-parallel validation path, and resolve.
//
// Arithmetic follows shaders/gps_splat.wgsl expression by expression (left-to-right, IEEE f32,
// no contraction: this file is compiled with --fmad=false) with the deterministic
// transcendentals of fmath.h, so results are bit-identical to the CPU mirror oracle.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "internal.h"

#include "devmath.cuh"
#include "pdl.cuh"

// Resident blocks per SM the particle kernel is compiled for (register budget).
#ifndef GPSB_FAST_MIN_BLOCKS
#define GPSB_FAST_MIN_BLOCKS 4  // resident blocks per SM of the PBVR fast-decision variant
#endif
#ifndef GPSB_PARTICLE_MIN_BLOCKS
#define GPSB_PARTICLE_MIN_BLOCKS 5
#endif

namespace gpsb {

typedef unsigned long long ull;

// ---------------------------------------------------------------- fast decisions
// Particles whose effect bounded approximate maths settles skip the exact path; the bounds and the
// decisions of the PBVR methods are in pbvr_fast.h, those of GPS and ScreenOccupancy below. The
// approximations are the MUFU forms (lg2 / rsqrt / sin / cos / ex2 / rcp, flush-to-zero).
using gxf::kErMax;
using gxf::kLn2;
using gxf::kLogAbs;
using gxf::kLogRel;
using gxf::kRMax;
using gxf::kSinCos;
using gxf::kU;
using gxf::kXMin;
constexpr float kSafe = 1.01f;
constexpr float kExpA = 6e-7f, kExpB = 1.5e-7f;     // |mexp(a) - exp(a)| <= (kExpA + kExpB |a|) mexp(a) + kExpTiny, a <= 0
constexpr float kExpTiny = 1.5e-38f;
constexpr float kLog2e = 1.44269502f;

__device__ __forceinline__ float mufu(float x, int op) {
    float y;
    switch (op) {
        case 0: asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
        case 1: asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
        case 2: asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
        case 3: asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
        case 4: asm("sin.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
        default: asm("cos.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); break;
    }
    return y;
}
__device__ __forceinline__ float mlog(float x) { return mufu(x, 0) * kLn2; }
__device__ __forceinline__ float mexp(float a) { return mufu(a * kLog2e, 1); }

// The approximations of the PBVR decisions on the GPU.
struct Mufu {
    // sqrt(x), x = -2 log u1 (one rounding: scaling by a power of two commutes with it)
    __device__ __forceinline__ float radius(float u1, float& x) const {
        x = mufu(u1, 0) * (-F_(2.0) * kLn2);
        return x * mufu(x, 2);
    }
    __device__ __forceinline__ float cos(float t) const { return mufu(t, 5); }
    __device__ __forceinline__ float sin(float t) const { return mufu(t, 4); }
    __device__ __forceinline__ float rcp(float x) const { return mufu(x, 3); }
    __device__ __forceinline__ float ex2(float x) const { return mufu(x, 1); }
    __device__ __forceinline__ float lg2(float x) const { return mufu(x, 0); }
    __device__ __forceinline__ bool every(bool b) const { return b; }
};
struct MufuWarp : Mufu {  // for a whole warp that decides together
    __device__ __forceinline__ bool every(bool b) const { return __all_sync(0xffffffffu, b); }
};

// ---------------------------------------------------------------- fast decisions (GPS): position bound
// gps_fast computes a particle's image position with the MUFU forms. r = sqrt(-2 log(1 - u1)) is
// within kErMax of the exact path's (checked over every uniform); the radius table is continuous
// and piecewise linear in w = r 128 / (4.123 sqrt 2), its largest step 0.04874 <= kLutSlope, and w is
// within 1.3e-4 (kErMax and the roundings of both paths at w <= 127), so the radius is within
// kLutSlope 1.3e-4 + 4e-6 (the interpolation's roundings in both paths); times sine or cosine, with
// radii up to 5.84, within kGpsEw.
constexpr float kLutSlope = 0.049f;
constexpr float kGpsEw = kLutSlope * 1.3e-4f + 4e-6f + 5.84f * (kSinCos + 2.0f * kU) + 6e-7f;
using gxf::kCellBias;
// Half a subpixel minus the bound of |position - exact position| in subpixels, along x and y; a
// sample nearer than that to a subpixel edge is undecided. Per unit of the factor's row sum S:
// kGpsEw and the products' roundings (below 6e-6); the sums' roundings at the magnitude of the
// mean and of the grid coordinate; 2e-6 for the subpixel arithmetic.
__device__ __forceinline__ float2 gps_limits(const FrameConst& f, float mx, float my, float l00, float l10, float l11) {
    const float side = (float)f.side, sx = fabsf(l00), sy = fabsf(l10) + fabsf(l11);
    if (max(f.W, f.H) > (1u << 20)) return make_float2(F_(-1.0), F_(-1.0));  // kCellBias holds grids below 2^22
    const float ex = (sx * (kGpsEw + 6e-6f) + F_(3e-7) * fabsf(mx)) * side * F_(1.02) + F_(2e-6);
    const float ey = (sy * (kGpsEw + 6e-6f) + F_(3e-7) * fabsf(my)) * side * F_(1.02) + F_(2e-6);
    return make_float2(F_(0.5) - ex, F_(0.5) - ey);  // not positive, or NaN: never decides
}

// ============================================================================ geometry
// Once per camera: projection, opacity clamp, per-method count descriptor and particle record,
// and the view-dependent SH colour (prepare/prepare_gps/prepare_pbvr without the seed-dependent
// Poisson draw, gps_splat.wgsl:535-642; splat_colour :210-251). It also zeroes the scratch of the first
// batch's count scan, which saves that batch a memset.
//
// The kernels of a frame (this one, k_count_scan, k_particles, k_resolve, k_features and the accumulator's
// clear) are launched with programmatic stream serialisation and wait for the previous grid as their
// first instruction, so each is resident when the one before it ends. With the clears inside kernels a frame of
// one batch is four launches (10k splats, 256x256, one ensemble: 24.5 -> 18.5 us; frames
// of milliseconds the same).
__global__ void __launch_bounds__(128) k_geometry(FrameConst f, const float4* __restrict__ splats,
                                                   const float* __restrict__ sh, float4* __restrict__ rec,
                                                   uint2* __restrict__ cdesc, float4* __restrict__ colour,
                                                   uint64_t* __restrict__ scratch, uint32_t scratch_words) {
    grid_dependency_wait();
    launch_dependents();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t k = i; k < scratch_words; k += gridDim.x * blockDim.x) scratch[k] = 0ull;
    if (i >= f.N) return;
    float4 g0 = __ldg(&splats[4 * (size_t)i]);
    float4 g1 = __ldg(&splats[4 * (size_t)i + 1]);
    float4 g2 = __ldg(&splats[4 * (size_t)i + 2]);
    float4 g3 = __ldg(&splats[4 * (size_t)i + 3]);
    uint2 cd = make_uint2(0u, CD_NONE);
    Proj pr = project(f, g0, g1, g2);
    float o = clamp_(g0.w, F_(0.0), F_(1.0));
    float4* R = rec + (size_t)i * kRecF4;
    if (pr.ok && o > F_(0.0)) {
        float l00 = sqrt_(fmax_(pr.a, F_(1e-30)));
        float l10 = div_(pr.b, l00);
        float l11 = sqrt_(fmax_(pr.c - l10 * l10, F_(1e-30)));
        float4 r0 = make_float4(pr.mx, pr.my, pr.depth, o);
        const uint32_t method = f.method;
        const float S = (float)f.S;
        if (method == 0u && f.fp_fixed <= 1u && !(f.fp_kappa > F_(0.0))) {
            float ex = gxc::kOffscreenSigma * sqrt_(pr.a), ey = gxc::kOffscreenSigma * sqrt_(pr.c);
            bool off = pr.mx + ex < F_(0.0) || pr.mx - ex >= (float)f.W || pr.my + ey < F_(0.0) || pr.my - ey >= (float)f.H;
            if (!off) {
                float det = pr.a * pr.c - pr.b * pr.b;
                float li2 = dilog(o);
                float en = f.density * S * F_(2.0) * gxc::kPi * sqrt_(det) * li2;
                if (en > F_(0.0)) cd = make_uint2(f2b(en), CD_POISSON_CAP);
                float fo = (F_(1.0) - sqrt_(fmax_(F_(1.0) - fmin_(o, F_(1.0)), F_(0.0)))) * F_(64.0);
                uint32_t i0 = min(f2u(fo), 63u);
                float a = fo - (float)i0;
                R[0] = r0;
                R[1] = make_float4(l00, l10, l11, a);
                R[2] = make_float4(__uint_as_float(i0), li2, F_(0.0), F_(0.0));
                const float2 lim = gps_limits(f, pr.mx, pr.my, l00, l10, l11);
                R[3] = make_float4(lim.x, lim.y, F_(0.0), F_(0.0));
            }
        } else if (method == 0u) {
            // footprint-subpixel mode (render_monte_carlo, oracle.rs:240-310): footprint s per splat
            // (fixed, or adaptive from the smallest standard deviation in subpixels), the expected
            // count divided by s^2, the sampling covariance optionally shrunk by the block's blur
            // (s / spp_side)^2 / 12, and the off-screen skip only for s = 1
            float det = pr.a * pr.c - pr.b * pr.b;
            uint32_t fp = max(f.fp_fixed, 1u);
            if (f.fp_kappa > F_(0.0)) {
                float tr = pr.a + pr.c;
                float disc = sqrt_(fmax_(F_(0.25) * tr * tr - det, F_(0.0)));
                float smin = sqrt_(fmax_(F_(0.5) * tr - disc, F_(0.0))) * (float)f.side;
                float sfp = floorf(f.fp_kappa * smin);
                fp = !(smin > F_(0.0)) || !(sfp >= F_(1.0)) ? 1u : (sfp >= (float)f.fp_max ? f.fp_max : (uint32_t)sfp);
            }
            float sa = pr.a, sb = pr.b, sc = pr.c;
            if (f.fp_comp && fp > 1u) {
                float q = (float)fp / (float)f.side;
                float v = q * q / F_(12.0);
                float ta = pr.a - v, tc = pr.c - v;
                float t = ta + tc, d = ta * tc - pr.b * pr.b;
                if (d > F_(0.0) && t > F_(0.0) && F_(0.5) * t - sqrt_(fmax_(F_(0.25) * t * t - d, F_(0.0))) >= v) {
                    sa = ta;
                    sc = tc;
                }
            }
            bool off = false;
            if (fp == 1u) {
                float ex = gxc::kOffscreenSigma * sqrt_(sa), ey = gxc::kOffscreenSigma * sqrt_(sc);
                off = pr.mx + ex < F_(0.0) || pr.mx - ex >= (float)f.W || pr.my + ey < F_(0.0) || pr.my - ey >= (float)f.H;
            }
            if (!off) {
                float li2 = dilog(o);
                float en = f.density * S * F_(2.0) * gxc::kPi * sqrt_(det) * li2 / (float)(fp * fp);
                if (en > F_(0.0)) cd = make_uint2(f2b(en), CD_POISSON_CAP);
                float fo = (F_(1.0) - sqrt_(fmax_(F_(1.0) - fmin_(o, F_(1.0)), F_(0.0)))) * F_(64.0);
                uint32_t i0 = min(f2u(fo), 63u);
                float a = fo - (float)i0;
                float m00 = sqrt_(fmax_(sa, F_(1e-30)));
                float m10 = div_(sb, m00);
                float m11 = sqrt_(fmax_(sc - m10 * m10, F_(1e-30)));
                R[0] = r0;
                R[1] = make_float4(m00, m10, m11, a);
                R[2] = make_float4(__uint_as_float(i0), li2, (float)fp, F_(0.0));
            }
        } else if (method == 4u) {
            float density = fmax_(f.density, F_(1e-8));
            float amin = fmax_(F_(1.0) - gx::exp(div_(gxc::kLn254over255, density)), F_(1e-8));
            if (o > amin) {
                float radius = sqrt_(F_(2.0) * gx::log(div_(o, amin)));
                float ext_x = radius * sqrt_(pr.a), ext_y = radius * sqrt_(pr.c);
                float lo_x = clamp_(floorf(pr.mx - ext_x), F_(0.0), (float)f.W);
                float lo_y = clamp_(floorf(pr.my - ext_y), F_(0.0), (float)f.H);
                float hi_x = clamp_(ceilf(pr.mx + ext_x), F_(0.0), (float)f.W);
                float hi_y = clamp_(ceilf(pr.my + ext_y), F_(0.0), (float)f.H);
                float sz_x = fmax_(hi_x - lo_x, F_(0.0)), sz_y = fmax_(hi_y - lo_y, F_(0.0));
                uint32_t count = f2u(sz_x) * f2u(sz_y) * f.side * f.side;
                if (count != 0u) {
                    float invdet = div_(F_(1.0), fmax_(pr.a * pr.c - pr.b * pr.b, F_(1e-30)));
                    float peak_tau = -gx::log(F_(1.0) - fmin_(o, gxc::kOneMinus1e6));
                    bool sparse = density * peak_tau < F_(1.0);
                    if (sparse) cd = make_uint2(f2b((float)count * density * peak_tau), CD_POISSON);
                    else cd = make_uint2(count, CD_FIXED);
                    R[0] = r0;
                    R[1] = make_float4(__uint_as_float(f2u(lo_x)), __uint_as_float(f2u(lo_y)), sz_x, sz_y);
                    R[2] = make_float4(pr.c * invdet, F_(2.0) * (-pr.b * invdet), pr.a * invdet, peak_tau);
                    R[3] = make_float4(__uint_as_float(0xFFFFFFFFu / f2u(sz_x)), __uint_as_float(f2u(sz_x)), __uint_as_float(count - 1u),
                                       sparse ? F_(1.0) : F_(0.0));
                }
            }
        } else {
            // pbvr_lambda (gps_splat.wgsl:441-460)
            float g = extinction_term(o);
            if (method == 1u) g = fmin_(o, gxc::kOneMinus1e6);
            float scale = f.base_k;
            if (method != 3u) {
                uint32_t level = f.calibration;
                if (level == 1u) scale = scale * pixel_density_scale(f, f.object_depth);
                else if (level == 2u) scale = scale * pixel_density_scale(f, pr.depth);
                else if (level == 3u) scale = S * F_(2.0) * gxc::kPi * sqrt_(pr.a * pr.c - pr.b * pr.b);
            }
            float lambda = f.density * g * scale;
            if (!(lambda > F_(0.0)) || lambda > F_(3.0e38)) lambda = F_(0.0);
            if (lambda > F_(0.0)) {
                float det = pr.a * pr.c - pr.b * pr.b;
                float keep = F_(1.0);
                uint32_t flags = CD_POISSON_CAP;
                if (method == 3u) {
                    float target = f.density * S * F_(2.0) * gxc::kPi * sqrt_(det) * dilog(o);
                    if (lambda > F_(0.5)) keep = clamp_(div_(target, lambda), F_(0.0), F_(1.0)); else keep = F_(0.0);
                    if (target > lambda) flags |= CD_UNDERCOVERED;
                }
                cd = make_uint2(f2b(lambda), flags);
                float idet = div_(F_(1.0), fmax_(det, F_(1e-30)));
                // chol_of (gps_splat.wgsl:464-485)
                float c0[3], c1[3], c2[3];
                rot_cols(g2, c0, c1, c2);
                float s2x = gx::exp(F_(2.0) * g1.x), s2y = gx::exp(F_(2.0) * g1.y), s2z = gx::exp(F_(2.0) * g1.z);
                float a00 = s2x * c0[0] * c0[0] + s2y * c1[0] * c1[0] + s2z * c2[0] * c2[0];
                float a10 = s2x * c0[1] * c0[0] + s2y * c1[1] * c1[0] + s2z * c2[1] * c2[0];
                float a20 = s2x * c0[2] * c0[0] + s2y * c1[2] * c1[0] + s2z * c2[2] * c2[0];
                float a11 = s2x * c0[1] * c0[1] + s2y * c1[1] * c1[1] + s2z * c2[1] * c2[1];
                float a21 = s2x * c0[2] * c0[1] + s2y * c1[2] * c1[1] + s2z * c2[2] * c2[1];
                float a22 = s2x * c0[2] * c0[2] + s2y * c1[2] * c1[2] + s2z * c2[2] * c2[2];
                float k00 = sqrt_(fmax_(a00, F_(1e-30)));
                float k10 = div_(a10, k00);
                float k20 = div_(a20, k00);
                float k11 = sqrt_(fmax_(a11 - k10 * k10, F_(1e-30)));
                float k21 = div_(a21 - k20 * k10, k11);
                float k22 = sqrt_(fmax_(a22 - k20 * k20 - k21 * k21, F_(1e-30)));
                const float oo = fmin_(o, gxc::kOneMinus1e6), h = eol(oo);
                R[0] = r0;
                R[1] = make_float4(keep, h, F_(0.0), F_(0.0));
                R[2] = make_float4(g0.x, g0.y, g0.z, pr.c * idet);
                R[3] = make_float4(-pr.b * idet, pr.a * idet, F_(0.0), F_(0.0));
                R[4] = make_float4(k00, k10, k11, F_(0.0));
                R[5] = make_float4(k20, k21, k22, F_(0.0));
                if (f.fast_mode) {
                    const float g[3] = {g0.x, g0.y, g0.z};
                    float q[24];
                    gxf::make_record(f.ff, f.rot0, f.rot1, f.rot2, f.pos, f.fx, f.fy, g, k00, k10, k11, k20, k21, k22,
                                     pr.c * idet, -pr.b * idet, pr.a * idet, pr.mx, pr.my, oo, h, q);
#pragma unroll
                    for (int c = 0; c < 6; ++c) R[6 + c] = make_float4(q[4 * c], q[4 * c + 1], q[4 * c + 2], q[4 * c + 3]);
                }
            }
        }
    }
    cdesc[i] = cd;
    if ((cd.y & 3u) != CD_NONE) colour[i] = splat_colour(f, sh, i, g0, g3);
}

void launch_geometry(const FrameConst& fc, const float4* splats, const float* sh, const float* lut, float4* rec,
                     uint2* cdesc, float4* colour, const ScanScratch& sc, size_t scratch_bytes, cudaStream_t st) {
    (void)lut;
    if (fc.N == 0) return;
    launch_pdl(k_geometry, dim3((fc.N + 127) / 128), dim3(128), 0, st, fc, splats, sh, rec, cdesc, colour, (uint64_t*)sc.mem,
               (uint32_t)(scratch_bytes / 8));
}

// ============================================================================ count + scan
__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t sat_add(uint64_t a, uint64_t b) {
    uint64_t s = a + b;
    return s > kLbSumSat ? kLbSumSat : s;
}
__device__ __forceinline__ uint64_t lb_pack(uint64_t status, uint64_t sum, uint32_t nz) {
    return status | ((sum > kLbSumSat ? kLbSumSat : sum) << 24) | (uint64_t)nz;
}

// Per ensemble e and tile t of 256 x ITEMS splats: Poisson count of every splat with the stream
// particle_seed(i, 0, first_seed + e) (gps_splat.wgsl:539-548, 593-602, 573-574), the per-splat cap,
// the statistics of prepare, then a block scan and a decoupled lookback over the tiles of the
// ensemble. Splats with a non-zero count are written, in splat order, to the compact list
// clist[e * N + j] = (splat id, exclusive particle offset). The last tile writes the ensemble
// total; a total above 2^32 - 1 marks the ensemble skipped (gps_splat.wgsl:635-639, 648-654).
// Bound: the draws of small means, one uniform per event (poisson): a thread draws for all its splats in
// one loop, going on to its next splat when one is done, so a warp runs as long as its largest sum of counts
// instead of the sum of each round's largest count (560k splats, far view, 64 ensembles: 1.06 -> 1.03 ms; mid view, 8: 0.156 -> 0.130).
// The draws leave the memory idle, so the blocks also clear the batch's subpixels, an equal share each
// (the same far view's scan 1032 -> 1062 us,
// a memset of 83 us saved; 560k splats, 4 ensembles of 1280x720 2x2: a memset of 20 us saved).
template <int ITEMS>
__global__ void __launch_bounds__(kScanThreads) k_count_scan(FrameConst f, const uint2* cdesc,
                                                             uint32_t first_seed, uint32_t tiles_per_e, uint32_t tiles,
                                                             ull* __restrict__ sub, uint64_t sub_words, uint64_t* lookback, uint32_t* tile_counter,
                                                             uint2* __restrict__ clist, EnsTotal* etot, ull* stats,
                                                             uint32_t* err) {
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_wsum[kScanThreads / 32];
    __shared__ uint32_t s_wnz[kScanThreads / 32];
    __shared__ uint64_t s_excl_sum;
    __shared__ uint32_t s_excl_nz;
    __shared__ ull s_stat[6];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // its dependent, the particle kernel, reads the list through the read-only path: it may start when this
    // kernel's blocks exit, not before (plain loads and an earlier start: a GPS frame of 773M particles 1.2 % longer)
    grid_dependency_wait();
    {
        const uint64_t pairs = sub_words / 2u, per = (pairs + gridDim.x - 1u) / gridDim.x, first = blockIdx.x * per;
        const uint64_t end = first + per < pairs ? first + per : pairs;
        for (uint64_t k = first + tid; k < end; k += kScanThreads)
            reinterpret_cast<uint4*>(sub)[k] = make_uint4(gxc::kEmpty, gxc::kEmpty, gxc::kEmpty, gxc::kEmpty);
        if (blockIdx.x == 0 && tid == 0 && (sub_words & 1u)) sub[sub_words - 1u] = ~0ull;
    }
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    if (tid < 6) s_stat[tid] = 0ull;
    __syncthreads();
    const uint32_t id = s_tile;
    if (id >= tiles) return;  // a block that was only there to clear
    const uint32_t e = id / tiles_per_e, t = id % tiles_per_e;
    const uint32_t seed = first_seed + e;
    const uint32_t N = f.N, cap = f.cap;
    const bool gps = f.method == 0u;
    const uint32_t base = (t * kScanThreads + tid) * ITEMS;

    uint32_t cnt[ITEMS];
    ull st_pts = 0, st_trunc = 0, st_drop = 0, st_vis = 0, st_cand = 0, st_under = 0;
    uint64_t tsum = 0;
    uint32_t tnz = 0;
    // raw counts: fixed ones, and the normal approximation of large means; small means are left to the loop below
    __shared__ float s_l[ITEMS][kScanThreads];        // exp(-lambda)
    __shared__ uint32_t s_rs[ITEMS][kScanThreads];    // stream state, then the count
    uint32_t todo = 0u, modes = 0u;
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t i = base + q;
        const uint2 cd = i < N ? cdesc[i] : make_uint2(0u, CD_NONE);
        const uint32_t mode = cd.y & 3u;
        uint32_t n = 0;
        if (mode == CD_FIXED) {
            n = cd.x;
        } else if (mode != CD_NONE) {
            uint32_t rs = gx::particle_seed(i, 0u, seed);
            const float lambda = __uint_as_float(cd.x);
            if (lambda > F_(0.0) && lambda < F_(30.0)) {
                s_l[q][tid] = gx::exp(-lambda);
                n = rs;
                todo |= 1u << q;
            } else {
                n = poisson(lambda, &rs);
            }
        }
        s_rs[q][tid] = n;
        modes |= mode << (2 * q);
        if (cd.y & CD_UNDERCOVERED) st_under += 1;
    }
    // gps_splat.wgsl:142-150 (poisson): uniforms until their product is at most exp(-lambda)
    {
        int q = todo ? __ffs(todo) - 1 : 0;
        float l = todo ? s_l[q][tid] : F_(0.0), p = F_(1.0);
        uint32_t rs = s_rs[q][tid], k = 0u;
        while (todo) {
            p = p * gx::next_u(&rs);
            if (p <= l) {
                s_rs[q][tid] = k;
                todo &= todo - 1u;
                q = todo ? __ffs(todo) - 1 : q;
                l = s_l[q][tid];
                rs = s_rs[q][tid];
                p = F_(1.0);
                k = 0u;
            } else {
                k += 1u;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t mode = (modes >> (2 * q)) & 3u;
        uint32_t n = s_rs[q][tid];
        if (mode != CD_NONE) {
            st_vis += 1;
            if (gps && mode != CD_FIXED) st_pts += n; else st_cand += n;
            if (mode == CD_POISSON_CAP && n > cap) {
                st_trunc += 1;
                st_drop += n - cap;
                n = cap;
            }
        }
        cnt[q] = n;
        tsum += n;
        tnz += n ? 1u : 0u;
    }
    // statistics: warp reduce, then shared, then one atomic per non-zero word per block
    ull sv[6] = {st_pts, st_trunc, st_drop, st_vis, st_cand, st_under};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        ull v = sv[k];
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(&s_stat[k], v);
    }
    // block scan of (tsum, tnz)
    uint64_t isum = tsum;
    uint32_t inz = tnz;
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t a = __shfl_up_sync(0xffffffffu, isum, o);
        uint32_t b = __shfl_up_sync(0xffffffffu, inz, o);
        if (lane >= o) { isum += a; inz += b; }
    }
    if (lane == 31) { s_wsum[warp] = isum; s_wnz[warp] = inz; }
    __syncthreads();
    uint64_t wpre = 0;
    uint32_t wpre_nz = 0, agg_nz = 0;
    uint64_t agg = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) {
        if (w < warp) { wpre += s_wsum[w]; wpre_nz += s_wnz[w]; }
        agg += s_wsum[w];
        agg_nz += s_wnz[w];
    }
    // decoupled lookback over the tiles of ensemble e
    uint64_t* lb = lookback + (size_t)e * tiles_per_e;
    if (warp == 0) {
        uint64_t excl = 0;
        uint32_t excl_nz = 0;
        if (t == 0) {
            if (lane == 0) st_relaxed(&lb[0], lb_pack(kLbPrefix, agg, agg_nz));
        } else {
            if (lane == 0) st_relaxed(&lb[t], lb_pack(kLbAggregate, agg, agg_nz));
            int32_t pred = (int32_t)t - 1;
            uint32_t spins = 0;
            bool failed = false;
            while (true) {
                int32_t j = pred - lane;
                uint64_t w = 0;
                if (j >= 0) {
                    w = ld_relaxed(&lb[j]);
                    while ((w >> 62) == 0ull) {
                        if (++spins > (1u << 20)) { failed = true; break; }
                        __nanosleep(64);
                        w = ld_relaxed(&lb[j]);
                    }
                } else {
                    w = kLbPrefix;  // before tile 0: an empty inclusive prefix
                }
                if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
                uint32_t is_prefix = __ballot_sync(0xffffffffu, (w >> 62) == 2ull);
                int first = is_prefix ? __ffs(is_prefix) - 1 : 32;  // closest predecessor with a prefix
                uint64_t v_sum = (lane <= first) ? ((w >> 24) & kLbSumSat) : 0ull;
                uint32_t v_nz = (lane <= first) ? (uint32_t)(w & 0xFFFFFFull) : 0u;
                for (int o = 16; o; o >>= 1) {
                    v_sum += __shfl_xor_sync(0xffffffffu, v_sum, o);
                    v_nz += __shfl_xor_sync(0xffffffffu, v_nz, o);
                }
                excl = sat_add(excl, v_sum);
                excl_nz += v_nz;
                if (first < 32) break;
                pred -= 32;
            }
            if (failed) {
                if (lane == 0) {
                    atomicOr(err, ERR_SCAN_LOOKBACK);
                    atomicOr(&etot[e].flags, 2u);
                }
                excl = 0;
                excl_nz = 0;
            }
            if (lane == 0) st_relaxed(&lb[t], lb_pack(kLbPrefix, sat_add(excl, agg), excl_nz + agg_nz));
        }
        if (lane == 0) { s_excl_sum = excl; s_excl_nz = excl_nz; }
    }
    __syncthreads();
    // compact list of non-zero splats
    uint64_t off = s_excl_sum + wpre + (isum - tsum);
    uint32_t j = s_excl_nz + wpre_nz + (inz - tnz);
    uint2* out = clist + (size_t)e * N;
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        if (cnt[q]) {
            out[j] = make_uint2(base + q, (uint32_t)off);
            off += cnt[q];
            ++j;
        }
    }
    if (tid < 6 && s_stat[tid]) {
        const int word[6] = {ST_POINTS, ST_TRUNCATED, ST_DROPPED, ST_VISIBLE, ST_CANDIDATES, ST_UNDERCOVERED};
        atomicAdd(&stats[word[tid]], s_stat[tid]);
    }
    if (t == tiles_per_e - 1 && tid == 0) {
        uint64_t total = sat_add(s_excl_sum, agg);
        etot[e].particles = total;
        etot[e].nonzero = s_excl_nz + agg_nz;
        atomicAdd(&stats[ST_ENTRIES], (ull)(s_excl_nz + agg_nz));
        atomicAdd(&stats[ST_ENSEMBLES], 1ull);
        if (total > 0xFFFFFFFFull) {
            atomicOr(&etot[e].flags, 1u);
            atomicAdd(&stats[ST_SKIPPED], 1ull);
        } else {
            atomicAdd(&stats[ST_PARTICLES], (ull)total);
        }
    }
}

// few tiles of eight splats a thread leave most SMs idle: one splat a thread
static bool scan_small(uint32_t n, uint32_t E) { return (uint64_t)((n + kScanTile - 1) / kScanTile) * E < kScanSmallTiles; }
static uint32_t count_scan_tiles(uint32_t n, uint32_t E) {
    return scan_small(n, E) ? (n + kScanThreads - 1) / kScanThreads : (n + kScanTile - 1) / kScanTile;
}
size_t count_scan_bytes(uint32_t n, uint32_t E) { return scan_scratch_bytes(E, (uint64_t)E * count_scan_tiles(n, E)); }

void launch_count_scan(const FrameConst& fc, const uint2* cdesc, uint32_t first_seed, uint32_t E, const ScanScratch& sc,
                       bool cleared, uint2* clist, unsigned long long* sub, unsigned long long* stats, uint32_t* err,
                       cudaStream_t st) {
    if (!cleared) cudaMemsetAsync(sc.mem, 0, count_scan_bytes(fc.N, E), st);
    if (fc.N == 0 || E == 0) return;
    const uint32_t per_e = count_scan_tiles(fc.N, E), tiles = per_e * E;
    const uint64_t sub_words = (uint64_t)E * fc.W * fc.H * fc.S;
    // with few tiles, more blocks that only clear: 32 KB each, up to two rounds of resident blocks
    const uint32_t grid = std::max(tiles, (uint32_t)std::min<uint64_t>((sub_words + 4095u) / 4096u, 148u * 16u));
    auto go = [&](auto kernel) {
        launch_pdl(kernel, dim3(grid), dim3(kScanThreads), 0, st, fc, cdesc, first_seed, per_e, tiles, sub, sub_words,
                   sc.lookback(E), sc.counters(), clist, sc.totals(), stats, err);
    };
    if (scan_small(fc.N, E)) go(k_count_scan<1>);
    else go(k_count_scan<kScanItems>);
}

// ============================================================================ particles
constexpr int kLutN = 65 * 129;

__device__ __forceinline__ void splat_write(ull* sub, uint32_t idx, float depth_z, uint32_t id) {
    ull packed = ((ull)(f2b(depth_z) | 0x80000000u) << 32) | (ull)id;
    ull cur = __ldcg(sub + idx);
    if (packed < cur) atomicMin(sub + idx, packed);
}

constexpr uint32_t kNoCell = 0xFFFFFFFFu;  // "not written" of the locate functions

// emit_particle (gps_splat.wgsl:259-282): the image position of a GPS particle, its random numbers
// taken from rs (kIter: the iterated radius and footprint blocks may be asked for)
template <bool kIter>
__device__ __forceinline__ float2 gps_position(const FrameConst& f, const FTabs& T, const float* lut, uint32_t& rs, float4 r0,
                                               float4 r1, float4 r2) {
    float u = gx::next_u(&rs);
    float r = kIter && f.exact_radius ? corrected_radius_exact(r0.w, r2.y, u)
                                      : corrected_radius_lut(lut, __float_as_uint(r2.x), r1.w, u, T.lg);
    float th = gxc::kTwoPi * gx::next_u(&rs);
    float sn, cs;
    gx::sincos_t(th, T.sc, &sn, &cs);
    float wx = r * cs, wy = r * sn;
    return make_float2(r0.x + r1.x * wx, r0.y + (r1.y * wx + r1.z * wy));
}
// subpixel of an image position, kNoCell off screen
__device__ __forceinline__ uint32_t subpixel_of(const FrameConst& f, float2 q) {
    if (q.x < F_(0.0) || q.x >= (float)f.W || q.y < F_(0.0) || q.y >= (float)f.H) return kNoCell;
    uint32_t px = f2u(q.x), py = f2u(q.y);
    uint32_t sx = min(f.side - 1u, f2u((q.x - (float)px) * (float)f.side));
    uint32_t sy = min(f.side - 1u, f2u((q.y - (float)py) * (float)f.side));
    return (py * f.W + px) * f.S + sy * f.side + sx;
}

// a GPS particle with the packed winner rule; returns whether it was written
template <bool kIter = true>
__device__ __forceinline__ uint32_t emit_gps(const FrameConst& f, const FTabs& T, const float* lut, uint32_t i, uint32_t& rs,
                                             float4 r0, float4 r1, float4 r2, ull* sub) {
    const float2 q = gps_position<kIter>(f, T, lut, rs, r0, r1, r2);
    if (kIter && r2.z > F_(1.0)) {
        // footprint block (write_block, oracle.rs:156-173): the s x s subpixels around the sample
        const int s = (int)r2.z, side = (int)f.side;
        const int gx0 = (int)floorf(q.x * (float)side - F_(0.5) * (float)s + F_(0.5));
        const int gy0 = (int)floorf(q.y * (float)side - F_(0.5) * (float)s + F_(0.5));
        const int gw = (int)f.W * side, gh = (int)f.H * side;
        uint32_t wrote = 0u;
        for (int gy = max(gy0, 0); gy < min(gy0 + s, gh); ++gy)
            for (int gx = max(gx0, 0); gx < min(gx0 + s, gw); ++gx) {
                const uint32_t qx = (uint32_t)(gx / side), qy = (uint32_t)(gy / side);
                splat_write(sub, (qy * f.W + qx) * f.S + (uint32_t)(gy % side) * f.side + (uint32_t)(gx % side), r0.z, i);
                wrote = 1u;
            }
        return wrote;
    }
    const uint32_t cell = subpixel_of(f, q);
    if (cell == kNoCell) return 0u;
    splat_write(sub, cell, r0.z, i);
    return 1u;
}

struct Normal {
    uint32_t* st;
    const FTabs& T;
    bool has;
    float spare;
    __device__ __forceinline__ float next() {
        if (has) { has = false; return spare; }
        float u1 = fmax_(gx::next_u(st), gxc::kUMin);
        float u2 = gx::next_u(st);
        float r = sqrt_(-F_(2.0) * gx::log_t_pos(u1, T.lg));  // u1 >= kUMin
        float sn, cs;
        gx::sincos_t(gxc::kTwoPi * u2, T.sc, &sn, &cs);
        spare = r * sn;
        has = true;
        return r * cs;
    }
};

// emit_particle_pbvr (gps_splat.wgsl:490-532); returns bit 0 = counts as a point, bit 1 = on screen, at
// `cell` with depth `depth_z`
__device__ __forceinline__ uint32_t pbvr_eval(const FrameConst& f, const FTabs& T, uint32_t& rs, const float4* R,
                                              uint32_t& cell, float& depth_z) {
    Normal nm{&rs, T, false, F_(0.0)};
    float uz = nm.next();
    float uy = nm.next();
    float ux = nm.next();
    float4 r1 = R[1];
    if (f.method == 3u) {
        if (gx::next_u(&rs) >= r1.x) return 0u;
    }
    float4 r2 = R[2], r4 = R[4], r5 = R[5];
    float wx = r2.x + r4.x * ux;
    float wy = r2.y + (r4.y * ux + r4.z * uy);
    float wz = r2.z + (r5.x * ux + r5.y * uy + r5.z * uz);
    float px = wx - f.pos[0], py = wy - f.pos[1], pz = wz - f.pos[2];
    float cx = dot3(f.rot0[0], f.rot0[1], f.rot0[2], px, py, pz);
    float cy = dot3(f.rot1[0], f.rot1[1], f.rot1[2], px, py, pz);
    float cz = dot3(f.rot2[0], f.rot2[1], f.rot2[2], px, py, pz);
    if (cz <= f.near_z) return 0u;
    float pix_x = div_(f.fx * cx, cz) + f.cx;
    float pix_y = div_(f.fy * cy, cz) + f.cy;
    const uint32_t flags = f.flags;
    if (flags & FLAG_JITTER) {
        float jy = nm.next();
        float jx = nm.next();
        pix_x = pix_x + f.jitter_sd * jx;
        pix_y = pix_y + f.jitter_sd * jy;
    }
    float4 r0 = R[0];
    if (flags & FLAG_RADIAL) {
        float4 r3 = R[3];
        float dvx = pix_x - r0.x, dvy = pix_y - r0.y;
        float r2v = r2.w * dvx * dvx + F_(2.0) * r3.x * dvx * dvy + r3.y * dvy * dvy;
        // radial_keep (gps_splat.wgsl:434-438) with h(min(o, 1-1e-6)) hoisted per splat
        float oo = fmin_(r0.w, gxc::kOneMinus1e6);
        float y = oo * gx::exp_t(-F_(0.5) * fmax_(r2v, F_(0.0)), T.ex);
        float keep = clamp_(div_(eol(y, T.lg), r1.y), F_(0.0), F_(1.0));
        if (gx::next_u(&rs) >= keep) return 0u;
    }
    depth_z = (flags & FLAG_CENTRE) ? r0.z : cz;
    if (pix_x < F_(0.0) || pix_x >= (float)f.W || pix_y < F_(0.0) || pix_y >= (float)f.H) return 1u;
    uint32_t ipx = f2u(pix_x), ipy = f2u(pix_y);
    uint32_t sx = min(f.side - 1u, f2u((pix_x - (float)ipx) * (float)f.side));
    uint32_t sy = min(f.side - 1u, f2u((pix_y - (float)ipy) * (float)f.side));
    cell = (ipy * f.W + ipx) * f.S + sy * f.side + sx;
    return 3u;
}
__device__ __forceinline__ uint32_t emit_pbvr(const FrameConst& f, const FTabs& T, uint32_t i, uint32_t& rs, const float4* R,
                                              ull* sub) {
    uint32_t cell;
    float z;
    const uint32_t r = pbvr_eval(f, T, rs, R, cell, z);
    if (r & 2u) splat_write(sub, cell, z, i);
    return r;
}

// grid coordinates (cx, cy) of a subpixel -> its index
__device__ __forceinline__ uint32_t cell_of(const FrameConst& f, uint32_t cx, uint32_t cy) {
    if (f.side == 1u) return cy * f.W + cx;
    uint32_t qx, qy;
    if (f.side == 3u) {
        qx = __umulhi(cx, 0x55555556u);
        qy = __umulhi(cy, 0x55555556u);
    } else {
        const uint32_t sh = f.side >> 1;  // 2 -> 1, 4 -> 2
        qx = cx >> sh;
        qy = cy >> sh;
    }
    return qy * ((f.W - 1u) * f.S) + cy * f.side + qx * (f.S - f.side) + cx;
}

// Exhaustive check of the constants of the fast decisions: the largest |approximation - exact| /
// bound over every input the approximations get, out[0..5] as float bits (ratios <= 1 hold the
// bounds): log over the uniforms k 2^-24; log over every float in [1e-6, 1); sin and cos over
// 2 pi k 2^-24; |r - r_exact| / kErMax over the uniforms with x >= kXMin; r / kRMax; exp over
// every float in [-128, 0]. NaN shows as infinity.
__device__ __forceinline__ void upd_ratio(float& m, float v) { m = v != v ? __int_as_float(0x7F800000) : fmaxf(m, v); }

__global__ void __launch_bounds__(256) k_fast_bounds(uint32_t* out) {
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    float m[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t k = tid; k < (1u << 24); k += nth) {
        const float u = (float)k * (1.0f / 16777216.0f);
        const float u1 = fmax_(u, gxc::kUMin);
        const float L = mlog(u1), Le = gx::log(u1);
        upd_ratio(m[0], fabsf(L - Le) / __fmaf_rn(kLogRel, fabsf(L), kLogAbs));
        // r exactly as fast_pair and Normal::next compute it
        const float x = -F_(2.0) * L;
        const float r = x * mufu(x, 2);
        const float re = sqrt_(-F_(2.0) * Le);
        if (x >= kXMin) {
            upd_ratio(m[3], fabsf(r - re) / kErMax);
            upd_ratio(m[4], r / kRMax);
        }
        const float t = gxc::kTwoPi * u;
        float se, ce;
        gx::sincos(t, &se, &ce);
        upd_ratio(m[2], fmaxf(fabsf(mufu(t, 4) - se), fabsf(mufu(t, 5) - ce)) / kSinCos);
    }
    for (uint32_t b = __float_as_uint(1e-6f) + tid; b < 0x3F800000u; b += nth) {
        const float v = __uint_as_float(b);
        const float L = mlog(v);
        upd_ratio(m[1], fabsf(L - gx::log(v)) / __fmaf_rn(kLogRel, fabsf(L), kLogAbs));
    }
    for (uint32_t b = 0x80000000u + tid; b <= 0xC3000000u; b += nth) {
        const float a = __uint_as_float(b);
        const float y = mexp(a);
        upd_ratio(m[5], fabsf(y - gx::exp(a)) / __fmaf_rn(__fmaf_rn(kExpB, fabsf(a), kExpA), y, kExpTiny));
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m[c]));
        if ((threadIdx.x & 31) == 0 && w) atomicMax(&out[c], w);
    }
}

void launch_fast_bounds(uint32_t* out, cudaStream_t st) {
    cudaMemsetAsync(out, 0, 6 * sizeof(uint32_t), st);
    k_fast_bounds<<<148 * 8, 256, 0, st>>>(out);
}

// The subpixel a ScreenOccupancy particle tests, its offset from the splat's centre and the acceptance
// draw's squared distance (particle_pass, gps_splat.wgsl:686-703): integer arithmetic and single
// roundings in the shader's order, shared by the exact and the fast decision. Divisions by the
// rectangle's width and by the subpixel count are multiplications by their reciprocals: R[3].x
// holds floor((2^32 - 1) / width), whose quotient is at most one too small; R[1].xy, R[3].y and R[3].z hold the
// rectangle's corner, its width and its last sample as integers.
struct SoCell {
    uint32_t cell;  // subpixel index
    float r2;       // squared Mahalanobis distance of the jittered sample
};
__device__ __forceinline__ SoCell so_cell(const FrameConst& f, uint32_t k, uint32_t& rs, const float4* R) {
    const float4 r0 = R[0], b = R[1], inv = R[2], r3 = R[3];
    const uint32_t side = f.side, samples = f.S;
    const uint32_t bz = __float_as_uint(r3.y);
    uint32_t cell = k;
    if (r3.w > F_(0.0)) cell = min(f2u(gx::next_u(&rs) * b.z * b.w * (float)samples), __float_as_uint(r3.z));
    uint32_t pixel = cell, sub_i = 0u;
    if (side > 1u) {
        pixel = side == 2u ? cell >> 2 : side == 4u ? cell >> 4 : cell / 9u;
        sub_i = cell - pixel * samples;
    }
    uint32_t row = __umulhi(pixel, __float_as_uint(r3.x)), col = pixel - row * bz;
    if (col >= bz) {
        col -= bz;
        ++row;
    }
    const uint32_t xx = __float_as_uint(b.x) + col, yy = __float_as_uint(b.y) + row;
    const float n1 = gx::next_u(&rs);
    const float n2 = gx::next_u(&rs);
    float uvx = n1, uvy = n2;
    if (side > 1u) {
        const uint32_t sy = side == 2u ? sub_i >> 1 : side == 4u ? sub_i >> 2 : sub_i / 3u;
        uvx = (float)(sub_i - sy * side) + n1;
        uvy = (float)sy + n2;
        if (side == 3u) {
            uvx = div_(uvx, F_(3.0));
            uvy = div_(uvy, F_(3.0));
        } else {  // a division by a power of two is exact
            const float h = side == 2u ? F_(0.5) : F_(0.25);
            uvx = uvx * h;
            uvy = uvy * h;
        }
    }
    const float dx = (float)xx + uvx - r0.x, dy = (float)yy + uvy - r0.y;
    SoCell c;
    c.r2 = fmax_(inv.x * dx * dx + inv.y * dx * dy + inv.z * dy * dy, F_(0.0));  // inv.y is doubled (exact)
    c.cell = (yy * f.W + xx) * samples + sub_i;
    return c;
}
// whether the particle is a hit, u its acceptance draw (gps_splat.wgsl:700-706)
__device__ __forceinline__ bool so_hit(const FrameConst& f, const FTabs& T, const float4* R, float r2, float u) {
    const float alpha = fmin_(R[0].w * gx::exp_t(-F_(0.5) * r2, T.ex), gxc::kOneMinus1e6);
    const float l = gx::log_t(F_(1.0) - alpha, T.lg);
    const float coverage = R[3].w > F_(0.0) ? div_(-l, R[2].w) : F_(1.0) - gx::exp_t(f.density * l, T.ex);
    return !(u >= coverage);
}
// ScreenOccupancy branch of particle_pass (gps_splat.wgsl:686-708); returns 1 on a hit
__device__ __forceinline__ uint32_t emit_so(const FrameConst& f, const FTabs& T, uint32_t i, uint32_t k, uint32_t& rs,
                                            const float4* R, ull* sub) {
    const SoCell c = so_cell(f, k, rs, R);
    if (!so_hit(f, T, R, c.r2, gx::next_u(&rs))) return 0u;
    splat_write(sub, c.cell, R[0].z, i);
    return 1u;
}

// ---------------------------------------------------------------- fast decisions (ScreenOccupancy, GPS)
// Both methods write a depth that is constant per splat, so a particle's whole effect is the
// subpixel it hits: once approximate maths with an error bound settles that, the exact path is not
// needed at all. The answers are the exact path's: 0 not written, 1 written, 2 undecided.

// so_hit with the MUFU forms. r2 is exact here, so the only errors are those of exp and log:
// y = o exp(-r2/2) within y rel (approximation, the exact exp's 2 ulp, both products' roundings),
// v = 1 - min(y, 1 - 1e-6) within ev, log v within el (its argument's error ev / v, 1.07 for
// ev / v <= 1/16, the approximation's and the exact log's own errors). Sparse splats compare u tau
// with -log v (one division and one product rounding), dense ones u with 1 - exp(density log v).
__device__ __forceinline__ uint32_t so_fast(const FrameConst& f, const float4* R, float r2, float u) {
    const float y = R[0].w * mufu(r2 * (-F_(0.5) * kLog2e), 1);
    const float rel = __fmaf_rn(F_(0.5) * kExpB, r2, kExpA + F_(5.4e-7) + F_(2.0) * kU);
    const float ev = __fmaf_rn(y, rel, F_(2.0) * kU + F_(2.0) * kExpTiny);
    const float v = F_(1.0) - fmin_(y, gxc::kOneMinus1e6);
    const float rv = ev * mufu(v, 3);
    const float l2 = mufu(v, 0);  // log2 v <= 0
    const float nl = l2 * -kLn2;
    const float el = __fmaf_rn(kLogRel + F_(5e-7), nl, __fmaf_rn(F_(1.08), rv, (kLogAbs + F_(4e-7)) * F_(1.01)));
    float a, e;  // the draw against a, within e
    bool sure = rv <= F_(0.0625);
    if (R[3].w > F_(0.0)) {
        u = u * R[2].w;
        a = nl;
        e = __fmaf_rn(F_(8.0) * kU, u, el);
    } else {
        const float x2 = f.density * l2;  // density log v, in powers of two
        const float ea = f.density * el;  // of density log v
        const float q = mufu(x2, 1);
        a = F_(1.0) - q;
        e = __fmaf_rn(q, __fmaf_rn(kExpB + F_(2.0) * kU, -x2, __fmaf_rn(ea, F_(1.1), kExpA + F_(5.4e-7))), F_(4.0) * kU + F_(2.0) * kExpTiny);
        sure = sure && ea >= F_(0.0) && ea <= F_(0.0625);
    }
    e = e * kSafe;
    const bool miss = u >= a + e, hit = u < a - e;
    return !sure ? 2u : miss ? 0u : hit ? 1u : 2u;
}

// A GPS particle's subpixel (bounds: gps_limits). At a node of the radius table either neighbouring
// cell gives the same value, so the cell may come from rounding w - 1/2.
__device__ __forceinline__ uint32_t gps_fast(const FrameConst& f, const float* lut, uint32_t rs, float4 r0, float4 r1,
                                             uint32_t row, float2 lim, uint32_t& cell) {
    const float a = fmax_(F_(1.0) - gx::next_u(&rs), gxc::kUMin);
    rs = gx::pcg(rs);
    const float x = mufu(a, 0) * (-F_(2.0) * kLn2);
    const float w = (x * mufu(x, 2)) * (gxc::kLutFv * F_(0.70710678));  // < 126.7
    const float t = (float)(rs >> 8u) * (gxc::kTwoPi * (F_(1.0) / F_(16777216.0)));
    const float wb = (w - F_(0.5)) + kCellBias;
    const float b = w - (wb - kCellBias);
    const float* L = lut + row + (__float_as_uint(wb) & 0xFFu);
    const bool far = x >= kXMin;  // else the radius bound does not hold (and w may be NaN)
    float ra = F_(0.0);
    if (far) {
        const float q00 = L[0], q01 = L[1], q10 = L[129], q11 = L[130];
        const float p0 = __fmaf_rn(b, q01 - q00, q00), p1 = __fmaf_rn(b, q11 - q10, q10);
        ra = __fmaf_rn(r1.w, p1 - p0, p0);
    }
    const float wx = ra * mufu(t, 5), wy = ra * mufu(t, 4);
    const float px = __fmaf_rn(r1.x, wx, r0.x), py = __fmaf_rn(r1.z, wy, __fmaf_rn(r1.y, wx, r0.y));
    const float side = (float)f.side;
    const float hx = __fmaf_rn(px, side, -F_(0.5)), hy = __fmaf_rn(py, side, -F_(0.5));
    const float bx = hx + kCellBias, by = hy + kCellBias;
    const bool sure = far && fabsf(hx - (bx - kCellBias)) < lim.x && fabsf(hy - (by - kCellBias)) < lim.y;
    const uint32_t cx = __float_as_uint(bx) - 0x4B400000u, cy = __float_as_uint(by) - 0x4B400000u;
    const bool on = cx < f.W * f.side && cy < f.H * f.side;
    cell = cell_of(f, cx, cy);
    return sure ? (on ? 1u : 0u) : 2u;
}

constexpr int kPT = 256;               // threads per particle block
constexpr uint32_t kRing = 64;         // per-warp ring of undecided particles (uint2 entries)
static_assert(kTabFloats % 2 == 0, "the unit table after the maths tables needs 8-byte alignment");

// Largest j in [lo, hi) with off(j) <= v, by a 32-ary warp search (off(lo) <= v must hold).
__device__ __forceinline__ uint32_t warp_last_le(const uint2* L, uint32_t lo, uint32_t hi, uint64_t v, int lane) {
    while (hi - lo > 1u) {
        uint32_t n = hi - lo;
        uint32_t step = (n + 31u) / 32u;
        uint32_t idx = lo + (uint32_t)(lane + 1) * step;
        bool p = idx < hi && (uint64_t)__ldg(&L[idx].y) <= v;
        uint32_t c = __popc(__ballot_sync(0xffffffffu, p));
        uint32_t nlo = lo + c * step;
        uint32_t nhi = lo + (c + 1u) * step;
        lo = nlo;
        hi = nhi < hi ? nhi : hi;
    }
    return lo;
}

// Whether variant (MC, FM) keeps the maths tables in shared memory: the variants whose particles
// mostly run the exact path. The fast GPS and ScreenOccupancy variants reach it for well under one
// particle in a hundred and read the global tables, which leaves the space to more blocks.
template <int MC, int FM>
constexpr bool kStageTabs = MC == 1 || FM != 1;

// Persistent particle kernel. A unit of work is up to steps * 32 consecutive particles of one
// ensemble; every warp by itself takes the next unit from a device counter, finds its first list
// entry with a 32-ary search and steps through it 32 particles at a time, lane l on particle
// p + l. Units are long (128 steps by default: near view 45.8 ms for 4 ensembles, 52.0 with 16)
// because each one pays for its search and for its last, partly filled run of undecided particles. Each particle is mapped to (splat i, k) through the compact list, regenerated from its own
// stream particle_seed(i, k + 1, seed) and written with one 64-bit atomicMin of (depth key << 32 | i),
// which equals the reference's depth pass followed by the colour pass (gps_splat.wgsl:276-281).
// Ensembles flagged skipped get no work.
//
// Bound: instruction issue (PBVR, ScreenOccupancy) or the scattered reads of the subpixel words
// (GPS). Consecutive lanes hold consecutive particles, so a step of a splat with 32 or more particles
// left is one warp-uniform comparison, and where splats change within a step the lanes share the
// records they load: the list entries of the step are one coalesced 256-byte read, the boundaries
// within it a __reduce_or_sync of one bit each. No list staging in shared memory, no block barrier.
// Measured against tiles of 4096 particles per block, 16 consecutive ones per thread, staged lists
// and the exact path for GPS and ScreenOccupancy (B200): a whole GPS frame, 560k splats, 1280x720, 2x2
// subpixels, 4 ensembles (773M particles) 10.9 -> 5.8 ms; ScreenOccupancy, 2M splats, 1920x1080, two
// cameras of 2 ensembles (9.8G particles) 114.6 -> 57.4 ms.
//
// MC: 0 GPS, 1 PBVR, 2 ScreenOccupancy; FM: fast decisions (0 off, 1 on, 2 validate: exact always,
// disagreements counted), template parameters so each variant gets its own register allocation.
// FL: the PBVR flags known at compile time, or -1: read from f; kViewConditioned: that method's flags (with fast
// decisions only; the others never are), kViewConditionedAny: the same, read from f.
constexpr int kViewConditioned = 8, kViewConditionedAny = -2;
template <int MC, int FM, int FL = -1>
__global__ void __launch_bounds__(kPT, MC == 1 && FM == 1 ? GPSB_FAST_MIN_BLOCKS : GPSB_PARTICLE_MIN_BLOCKS)
    k_particles(FrameConst f, const float4* __restrict__ rec, const float* __restrict__ lut, const uint2* clist,
                const EnsTotal* etot, uint32_t first_seed, uint32_t E, uint32_t max_steps, ull* sub,
                uint32_t* unit_counter, ull* stats) {
    // dynamic shared memory: [maths tables (kTabFloats)] [first unit of each ensemble (E + 1, 64-bit)]
    // [rings (FM == 1)] [radius table (GPS)]
    extern __shared__ __align__(16) uint32_t s_dyn[];
    constexpr bool kTabs = kStageTabs<MC, FM>;
    uint64_t* s_ubase = reinterpret_cast<uint64_t*>(s_dyn + (kTabs ? kTabFloats : 0));
    uint2* s_ring = reinterpret_cast<uint2*>(s_ubase + (E + 1));
    float* s_lut = reinterpret_cast<float*>(s_ring + (FM == 1 ? (kPT / 32) * kRing : 0));
    __shared__ uint32_t s_steps;
    const int tid = threadIdx.x, lane = tid & 31;
    grid_dependency_wait();
    launch_dependents();
    // particles per unit: max_steps * 32, fewer when warps would get less than four units each
    // (560k splats, far view, 4 ensembles: 0.775 ms; with one unit each 0.847), but at least two steps, as every
    // block that has a unit stages its tables (10k splats: 10.2 us; one step 12.9, four 11.6)
    if (tid < 32) {
        uint64_t total = 0;
        for (uint32_t e = lane; e < E; e += 32) {
            const EnsTotal t = etot[e];
            total += t.flags == 0u ? t.particles : 0ull;
        }
        for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        const uint64_t want = total / ((uint64_t)gridDim.x * kPT * 4u);
        const uint32_t steps = want >= max_steps ? max_steps : want < 2u ? 2u : (uint32_t)want;
        uint64_t acc = 0;
        for (uint32_t e0 = 0; e0 < E; e0 += 32) {
            const uint32_t e = e0 + lane;
            uint64_t n = 0;
            if (e < E) {
                const EnsTotal t = etot[e];
                n = t.flags == 0u ? (t.particles + steps * 32u - 1u) / (steps * 32u) : 0ull;
            }
            uint64_t incl = n;
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (e < E) s_ubase[e] = acc + incl - n;
            acc += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
            s_ubase[E] = acc;
            s_steps = steps;
        }
    }
    __syncthreads();
    const uint64_t total_units = s_ubase[E];
    // a block whose warps could not get a unit each leaves before it stages anything
    if ((uint64_t)blockIdx.x * (kPT / 32) >= total_units) return;
    FTabs T{gx::tab_log(), gx::tab_exp(), gx::tab_sc()};
    if (kTabs) T = stage_tabs(reinterpret_cast<float*>(s_dyn));
    if (MC == 0 && !f.exact_radius)
        for (int k = tid; k < kLutN; k += kPT) s_lut[k] = __ldg(&lut[k]);
    __syncthreads();
    const uint32_t unit = s_steps * 32u;
    const uint64_t PS = (uint64_t)f.W * f.H * f.S;
    const uint32_t upto = 0xFFFFFFFFu >> (31 - lane);  // lanes up to this one
    uint2* ring = s_ring + (size_t)(tid >> 5) * kRing;
    const uint32_t flags = FL >= 0 ? (uint32_t)(FL & ~kViewConditioned) : f.flags;
    const bool vc = FM == 2 ? f.method == 3u : FL == kViewConditionedAny || (FL >= 0 && (FL & kViewConditioned));  // of the decisions
    uint32_t points = 0, writes = 0, exact_runs = 0, mismatch = 0;
    // the first unit is the warp's own number, the next ones come from the counter (a call with no more units
    // than warps asks it nothing: thousands of warps queue up on one word)
    const uint32_t warps = gridDim.x * (kPT / 32);
    uint32_t next = blockIdx.x * (kPT / 32) + (tid >> 5);
    for (;;) {
        const uint32_t un = __shfl_sync(0xffffffffu, next, 0);
        if ((uint64_t)un >= total_units) break;
        next = 0xFFFFFFFFu;
        if (total_units > warps && lane == 0) next = warps + atomicAdd(unit_counter, 1u);  // its latency is covered by this unit
        // ensemble of the unit: largest e with s_ubase[e] <= un
        uint32_t e = 0, eh = E;
        while (eh - e > 1u) {
            const uint32_t mid = (e + eh) >> 1;
            if (s_ubase[mid] <= un) e = mid; else eh = mid;
        }
        const uint32_t n_part = (uint32_t)etot[e].particles;  // below 2^32: the ensemble is not skipped
        const uint32_t nz = etot[e].nonzero;
        const uint32_t p0 = (uint32_t)((uint64_t)un - s_ubase[e]) * unit;
        const uint32_t left = n_part - p0 < unit ? n_part - p0 : unit;  // particles of the unit
        const uint2* L = clist + (size_t)e * f.N;
        const uint32_t seed = first_seed + e;
        ull* S = sub + (size_t)e * PS;
        // the entry of the step's first particle: index ej, splat ci, offset co; nx the next offset
        uint32_t ej = warp_last_le(L, 0u, nz, p0, lane);
        uint32_t ci, co, nx;
        {
            const uint2 en = __ldg(&L[ej]);
            ci = en.x;
            co = en.y;
            nx = ej + 1u < nz ? __ldg(&L[ej + 1u].y) : n_part;
        }
        uint32_t cur = 0xFFFFFFFFu;
        float4 R[6];
        constexpr int kRec = MC == 1 ? 6 : FM == 1 || MC == 2 ? 4 : 3;
        auto load_rec = [&](uint32_t i) {
            const float4* Rg = rec + (size_t)i * kRecF4;
#pragma unroll
            for (int c = 0; c < kRec; ++c) R[c] = __ldg(&Rg[c]);
            cur = i;
        };
        float q[24];  // PBVR: the fast record of splat curq
        float keep = F_(0.0);
        uint32_t curq = 0xFFFFFFFFu;
        auto load_fast = [&](uint32_t i) {
            const float4* Rg = rec + (size_t)i * kRecF4 + 6;
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                const float4 v = __ldg(&Rg[c]);
                q[4 * c] = v.x;
                q[4 * c + 1] = v.y;
                q[4 * c + 2] = v.z;
                q[4 * c + 3] = v.w;
            }
            if (vc) keep = __ldg(&rec[(size_t)i * kRecF4 + 1].x);
            curq = i;
        };
        auto exact = [&](uint32_t i, uint32_t k, const float4* X) {
            uint32_t rs = gx::particle_seed(i, k + 1u, seed);
            if (MC == 0) {
                writes += emit_gps<FM == 0>(f, T, s_lut, i, rs, X[0], X[1], X[2], S);
            } else {
                const uint32_t r = MC == 1 ? emit_pbvr(f, T, i, rs, X, S) : emit_so(f, T, i, k, rs, X, S);
                points += r & 1u;
                writes += MC == 1 ? r >> 1 : r;
            }
        };
        auto run_exact = [&](uint32_t i, uint32_t k) {
            if (FM == 1) {  // the lanes' splats differ; the registers of the fast record stay
                const float4* Rg = rec + (size_t)i * kRecF4;
                float4 X[kRec];
#pragma unroll
                for (int c = 0; c < kRec; ++c) X[c] = __ldg(&Rg[c]);
                exact(i, k, X);
            } else {
                if (i != cur) load_rec(i);
                exact(i, k, R);
            }
        };
        uint32_t head = 0u, count = 0u;
        for (uint32_t d0 = 0; d0 < left; d0 += 32u) {
            const uint32_t pp0 = p0 + d0;  // first particle of the step
            const bool act = d0 + (uint32_t)lane < left;
            uint32_t i = ci, k = pp0 + (uint32_t)lane - co;
            const uint32_t room = nx - pp0;  // particles of the current entry from pp0 on
            if (room <= 32u) {
                // entries that begin within the step, in list order, one per lane; offsets are distinct
                const uint32_t j = ej + 1u + (uint32_t)lane;
                const uint2 en = j < nz ? __ldg(&L[j]) : make_uint2(0u, 0u);
                const uint32_t d = j < nz ? en.y - pp0 : 64u;
                const uint32_t starts = __reduce_or_sync(0xffffffffu, d < 32u ? 1u << d : 0u);
                const uint32_t c = (uint32_t)__popc(starts & upto);  // entries begun by this lane
                const uint32_t src = c - 1u;
                const uint32_t wi = __shfl_sync(0xffffffffu, en.x, src & 31u), wo = __shfl_sync(0xffffffffu, en.y, src & 31u);
                if (c) {
                    i = wi;
                    k = pp0 + (uint32_t)lane - wo;
                }
                // the entry of the next step's first particle
                const uint32_t adv = (uint32_t)__popc(__ballot_sync(0xffffffffu, d <= 32u));
                if (adv) {
                    ej += adv;
                    ci = __shfl_sync(0xffffffffu, en.x, adv - 1u);
                    co = __shfl_sync(0xffffffffu, en.y, adv - 1u);
                    nx = ej + 1u < nz ? (adv < 32u ? __shfl_sync(0xffffffffu, en.y, adv & 31u) : __ldg(&L[ej + 1u].y)) : n_part;
                }
            }
            if (FM == 1) {
                // converged fast step: every lane evaluates a particle (a lane past the unit one it does
                // not own, whose answer is ignored); where any lane's splat changed all lanes reload
                if (MC == 1) {
                    if (__any_sync(0xffffffffu, i != curq)) load_fast(i);
                } else if (__any_sync(0xffffffffu, i != cur)) {
                    load_rec(i);
                }
                uint32_t rs = gx::particle_seed(i, k + 1u, seed);
                uint32_t a;  // the answer
                if (MC == 0) {
                    uint32_t cell;
                    a = gps_fast(f, s_lut, rs, R[0], R[1], __float_as_uint(R[2].x) * 129u, make_float2(R[3].x, R[3].y), cell);
                    if (act && a == 1u) {
                        splat_write(S, cell, R[0].z, i);
                        ++writes;
                    }
                } else if (MC == 1) {
                    MufuWarp ap;
                    gxf::Point P;
                    a = gxf::decide(ap, f.ff, flags, vc, keep, rs, q, P);
                    if (act && a == 3u) {
                        // on screen: with the subpixel settled and the depth surely behind the subpixel's
                        // word (which only ever decreases) the write has no effect but its count
                        uint32_t cx, cy;
                        bool on;
                        a = 2u;
                        if (gxf::settle(f.ff, f.side, f.W, f.H, P, cx, cy, on)) {
                            a = 1u;
                            if (on) {
                                const uint32_t cell = cell_of(f, cx, cy);
                                if (flags & FLAG_CENTRE) {
                                    splat_write(S, cell, __ldg(&rec[(size_t)i * kRecF4].z), i);
                                    ++writes;
                                } else {
                                    const uint32_t front = f2b(P.z - q[21]) | 0x80000000u;
                                    const bool behind = front > __ldcg(reinterpret_cast<const uint32_t*>(S + cell) + 1);
                                    a = behind ? 1u : 2u;
                                    writes += behind ? 1u : 0u;
                                }
                            }
                        }
                    }
                    points += act ? a & 1u : 0u;
                } else {
                    const SoCell c = so_cell(f, k, rs, R);
                    a = so_fast(f, R, c.r2, gx::next_u(&rs));
                    if (act && a == 1u) {
                        splat_write(S, c.cell, R[0].z, i);
                        ++writes;
                        ++points;
                    }
                }
                // undecided particles wait in the warp's ring and run the exact path 32 at a time
                const bool need = act && a == 2u;
                const uint32_t bal = __ballot_sync(0xffffffffu, need);
                if (bal == 0u) continue;
                const uint32_t n = (uint32_t)__popc(bal);
                if (need) ring[(head + count + (uint32_t)__popc(bal & upto) - 1u) & (kRing - 1u)] = make_uint2(i, k);
                count += n;
                exact_runs += need ? 1u : 0u;
                if (count >= 32u) {
                    __syncwarp();
                    const uint2 en = ring[(head + (uint32_t)lane) & (kRing - 1u)];
                    __syncwarp();
                    head += 32u;
                    count -= 32u;
                    run_exact(en.x, en.y);
                }
            } else if (act) {
                if (FM == 2) {  // validation: the fast answer against the exact path, which alone writes
                    if (i != cur) load_rec(i);
                    uint32_t rs = gx::particle_seed(i, k + 1u, seed), rx = rs;
                    uint32_t a, x;
                    if (MC == 0) {
                        uint32_t cell;
                        a = gps_fast(f, s_lut, rs, R[0], R[1], __float_as_uint(R[2].x) * 129u, gps_limits(f, R[0].x, R[0].y, R[1].x, R[1].y, R[1].z), cell);
                        const uint32_t xc = subpixel_of(f, gps_position<false>(f, T, s_lut, rx, R[0], R[1], R[2]));
                        x = xc == kNoCell ? 0u : 1u;
                        if (a == 1u && xc != cell) x = 3u;
                    } else if (MC == 1) {
                        if (i != curq) load_fast(i);
                        Mufu ap;
                        gxf::Point P;
                        a = gxf::decide(ap, f.ff, f.flags, vc, keep, rs, q, P);
                        uint32_t xc;
                        float z;
                        x = pbvr_eval(f, T, rx, R, xc, z);
                        if (a == 3u) {
                            uint32_t cx, cy;
                            bool on, ok = (x & 1u) != 0u;
                            if (gxf::settle(f.ff, f.side, f.W, f.H, P, cx, cy, on)) {
                                ok = x == (on ? 3u : 1u);
                                if (ok && on)
                                    ok = xc == cell_of(f, cx, cy) && ((f.flags & FLAG_CENTRE) || fabsf(P.z - z) <= q[21]);
                            }
                            mismatch += ok ? 0u : 1u;
                            a = 2u;
                        }
                    } else {
                        const SoCell c = so_cell(f, k, rs, R);
                        const float u = gx::next_u(&rs);
                        a = so_fast(f, R, c.r2, u);
                        x = so_hit(f, T, R, c.r2, u) ? 1u : 0u;
                    }
                    mismatch += (a != 2u && a != x) ? 1u : 0u;
                    exact_runs += a == 2u ? 1u : 0u;
                    run_exact(i, k);
                } else {
                    run_exact(i, k);
                }
            }
        }
        if (FM == 1) {
            __syncwarp();
            if ((uint32_t)lane < count) {
                const uint2 q = ring[(head + (uint32_t)lane) & (kRing - 1u)];
                run_exact(q.x, q.y);
            }
            __syncwarp();  // the ring is free again
        }
    }
    ull v = points, wv = writes, xv = exact_runs, mv = mismatch;
    for (int o = 16; o; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
        wv += __shfl_xor_sync(0xffffffffu, wv, o);
        xv += __shfl_xor_sync(0xffffffffu, xv, o);
        mv += __shfl_xor_sync(0xffffffffu, mv, o);
    }
    if (lane == 0 && v && MC != 0) atomicAdd(&stats[ST_POINTS], v);
    if (lane == 0 && wv) atomicAdd(&stats[ST_WRITES], wv);
    if (lane == 0 && xv) atomicAdd(&stats[ST_FAST_EXACT], xv);
    if (lane == 0 && mv) atomicAdd(&stats[ST_FAST_MISMATCH], mv);
}

template <int MC, int FM, int FL = -1>
static void launch_particles_t(const FrameConst& fc, const float4* rec, const float* lut, const uint2* clist,
                               const EnsTotal* etot, uint32_t first_seed, uint32_t E, unsigned long long* sub,
                               uint32_t* unit_counter, unsigned long long* stats, int grid, int steps, cudaStream_t st) {
    size_t smem = ((kStageTabs<MC, FM> ? kTabFloats : 0) + 2 * ((size_t)E + 1)) * sizeof(uint32_t);
    if (FM == 1) smem += (size_t)(kPT / 32) * kRing * sizeof(uint2);
    if (MC == 0 && !fc.exact_radius) smem += kLutN * sizeof(float);
    // the attribute belongs to each device's context: remember the size set per device ordinal
    static size_t attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const bool known = dev >= 0 && dev < 64;
    if (smem > 48 * 1024 && (!known || smem > attr[dev])) {
        cudaFuncSetAttribute(k_particles<MC, FM, FL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (known) attr[dev] = smem;
    }
    launch_pdl(k_particles<MC, FM, FL>, dim3(grid), dim3(kPT), smem, st, fc, rec, lut, clist, etot, first_seed, E,
               (uint32_t)steps, sub, unit_counter, stats);
}

void launch_particles(const FrameConst& fc, const float4* rec, const float* lut, const uint2* clist,
                      const EnsTotal* etot, uint32_t first_seed, uint32_t E, unsigned long long* sub,
                      uint32_t* unit_counter, unsigned long long* stats, int grid, int items, cudaStream_t st) {
    if (fc.N == 0 || E == 0) return;
    // the fast GPS decisions cover single subpixels and the radius table; footprint blocks and the
    // iterated radius run the exact path
    uint32_t fm = fc.fast_mode;
    if (fc.method == 0u && (fc.exact_radius || fc.fp_fixed > 1u || fc.fp_kappa > 0.0f)) fm = 0u;
    auto go = [&](auto mc, auto mode) {
        launch_particles_t<decltype(mc)::value, decltype(mode)::value>(fc, rec, lut, clist, etot, first_seed, E, sub,
                                                                       unit_counter, stats, grid, items, st);
    };
    auto method = [&](auto mc) {
        if (fm == 1u) go(mc, std::integral_constant<int, 1>());
        else if (fm == 2u) go(mc, std::integral_constant<int, 2>());
        else go(mc, std::integral_constant<int, 0>());
    };
    // the two common flag sets of the fast PBVR decisions, compiled with the flags known (ViewConditioned, 560k
    // splats, 1280x720, 4 ensembles, jitter and radial, read / known: distance 2.5 10.71 / 10.57 ms, 20 9.64 / 9.50)
    constexpr int kJR = (int)(FLAG_JITTER | FLAG_RADIAL), kJ = (int)FLAG_JITTER;
    auto known = [&](auto fl) {
        launch_particles_t<1, 1, decltype(fl)::value>(fc, rec, lut, clist, etot, first_seed, E, sub, unit_counter, stats, grid,
                                                      items, st);
    };
    const bool pbvr = fc.method == 1u || fc.method == 2u, vc = fc.method == 3u;
    if (pbvr && fm == 1u && fc.flags == (uint32_t)kJR) known(std::integral_constant<int, kJR>());
    else if (pbvr && fm == 1u && fc.flags == (uint32_t)kJ) known(std::integral_constant<int, kJ>());
    else if (vc && fm == 1u && fc.flags == (uint32_t)kJR) known(std::integral_constant<int, kViewConditioned | kJR>());
    else if (vc && fm == 1u && fc.flags == (uint32_t)kJ) known(std::integral_constant<int, kViewConditioned | kJ>());
    else if (vc && fm == 1u) known(std::integral_constant<int, kViewConditionedAny>());
    else if (fc.method == 0u) method(std::integral_constant<int, 0>());
    else if (fc.method == 4u) method(std::integral_constant<int, 2>());
    else method(std::integral_constant<int, 1>());
}

// ============================================================================ primitive path
// splat_pass (gps_splat.wgsl:304-333): one thread per splat and ensemble generates all particles
// of the splat from one sequential stream. Validation path of GPS only (RenderPath::Primitive).
__global__ void __launch_bounds__(128) k_primitive(FrameConst f, const float4* __restrict__ rec,
                                                   const uint2* __restrict__ cdesc, const float* __restrict__ lut,
                                                   uint32_t first_seed, uint32_t E, ull* sub, ull* stats) {
    uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t i = gi % f.N, e = gi / f.N;
    if (e >= E) return;
    uint2 cd = __ldg(&cdesc[i]);
    if ((cd.y & 3u) != CD_POISSON_CAP) return;
    uint32_t rs = gx::particle_seed(i, 0u, first_seed + e);
    uint32_t n = poisson(__uint_as_float(cd.x), &rs);
    atomicAdd(&stats[ST_POINTS], (ull)n);
    atomicAdd(&stats[ST_VISIBLE], 1ull);
    if (n > f.cap) {
        atomicAdd(&stats[ST_TRUNCATED], 1ull);
        atomicAdd(&stats[ST_DROPPED], (ull)(n - f.cap));
        n = f.cap;
    }
    const float4* Rg = rec + (size_t)i * kRecF4;
    float4 r0 = Rg[0], r1 = Rg[1], r2 = Rg[2];
    ull* S = sub + (size_t)e * ((uint64_t)f.W * f.H * f.S);
    ull writes = 0;
    const FTabs T{gx::tab_log(), gx::tab_exp(), gx::tab_sc()};
    for (uint32_t q = 0; q < n; ++q) writes += emit_gps(f, T, lut, i, rs, r0, r1, r2, S);
    if (writes) atomicAdd(&stats[ST_WRITES], writes);
}

void launch_primitive(const FrameConst& fc, const float4* rec, const uint2* cdesc, const float* lut,
                      uint32_t first_seed, uint32_t E, unsigned long long* sub, EnsTotal* etot,
                      unsigned long long* stats, cudaStream_t st) {
    cudaMemsetAsync(etot, 0, (size_t)E * sizeof(EnsTotal), st);
    if (fc.N == 0 || E == 0) return;
    uint64_t n = (uint64_t)fc.N * E;
    k_primitive<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(fc, rec, cdesc, lut, first_seed, E, sub, stats);
}

// ============================================================================ resolve
// resolve (gps_splat.wgsl:362-386) for every ensemble of the batch, in ensemble order, so the
// f32 accumulation sequence equals the reference's one resolve per ensemble.
__global__ void __launch_bounds__(256) k_resolve(FrameConst f, const ull* sub,
                                                  const EnsTotal* __restrict__ etot, const float4* __restrict__ colour,
                                                  uint32_t E, float4* accum, ull* stats) {
    grid_dependency_wait();
    launch_dependents();
    uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t P = f.W * f.H;
    if (pix >= P) return;
    const uint32_t S = f.S;
    const uint64_t PS = (uint64_t)P * S;
    float4 acc = accum[pix];
    const float inv_bg0 = f.bg[0], inv_bg1 = f.bg[1], inv_bg2 = f.bg[2];
    uint32_t orphans = 0;
    for (uint32_t e = 0; e < E; ++e) {
        if (__ldg(&etot[e].flags) != 0u) continue;
        const ull* s = sub + (size_t)e * PS + (size_t)pix * S;
        float sx = F_(0.0), sy = F_(0.0), sz = F_(0.0);
        for (uint32_t k = 0; k < S; ++k) {
            ull v = __ldcs(s + k);
            uint32_t key = (uint32_t)(v >> 32), id = (uint32_t)v;
            if (key == gxc::kEmpty) {
                sx = sx + inv_bg0; sy = sy + inv_bg1; sz = sz + inv_bg2;
            } else if (id == gxc::kEmpty) {
                ++orphans;
                sx = sx + inv_bg0; sy = sy + inv_bg1; sz = sz + inv_bg2;
            } else {
                float4 c = __ldg(&colour[id]);
                sx = sx + c.x; sy = sy + c.y; sz = sz + c.z;
            }
        }
        const float Sf = (float)S;
        acc.x = acc.x + div_(sx, Sf);
        acc.y = acc.y + div_(sy, Sf);
        acc.z = acc.z + div_(sz, Sf);
        acc.w = acc.w + F_(1.0);
    }
    accum[pix] = acc;
    if (orphans) atomicAdd(&stats[ST_ORPHAN], (ull)orphans);
}

void launch_resolve(const FrameConst& fc, const unsigned long long* sub, const EnsTotal* etot, const float4* colour,
                    uint32_t E, float4* accum, unsigned long long* stats, cudaStream_t st) {
    uint32_t P = fc.W * fc.H;
    if (P == 0 || E == 0) return;
    launch_pdl(k_resolve, dim3((P + 255) / 256), dim3(256), 0, st, fc, sub, etot, colour, E, accum, stats);
}

// Denoiser features of the batch's ensembles (no counterpart in the reference, which has no
// denoiser): per pixel and ensemble the resolved colour c (as k_resolve computes it), the covered
// fraction alpha of its subpixels and the covered subpixels' depth sum / S; adds (c.r^2, c.g^2,
// c.b^2, alpha, depth) to feat[pix * 8 + 0..4]. Skipped ensembles add nothing.
__global__ void __launch_bounds__(256) k_features(FrameConst f, const ull* __restrict__ sub,
                                                   const EnsTotal* __restrict__ etot, const float4* __restrict__ colour,
                                                   uint32_t E, float* feat) {
    grid_dependency_wait();
    launch_dependents();
    uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t P = f.W * f.H;
    if (pix >= P) return;
    const uint32_t S = f.S;
    const uint64_t PS = (uint64_t)P * S;
    float q[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t e = 0; e < E; ++e) {
        if (__ldg(&etot[e].flags) != 0u) continue;
        const ull* s = sub + (size_t)e * PS + (size_t)pix * S;
        float sx = F_(0.0), sy = F_(0.0), sz = F_(0.0), cov = 0.0f, dep = 0.0f;
        for (uint32_t k = 0; k < S; ++k) {
            ull v = __ldcs(s + k);
            uint32_t key = (uint32_t)(v >> 32), id = (uint32_t)v;
            if (key == gxc::kEmpty || id == gxc::kEmpty) {
                sx = sx + f.bg[0]; sy = sy + f.bg[1]; sz = sz + f.bg[2];
            } else {
                float4 c = __ldg(&colour[id]);
                sx = sx + c.x; sy = sy + c.y; sz = sz + c.z;
                cov += 1.0f;
                dep += __uint_as_float(key & 0x7FFFFFFFu);
            }
        }
        const float Sf = (float)S;
        const float cr = div_(sx, Sf), cg = div_(sy, Sf), cb = div_(sz, Sf);
        q[0] += cr * cr;
        q[1] += cg * cg;
        q[2] += cb * cb;
        q[3] += cov / Sf;
        q[4] += dep / Sf;
    }
    float* o = feat + (size_t)pix * 8;
#pragma unroll
    for (int j = 0; j < 5; ++j) o[j] += q[j];
}

void launch_features(const FrameConst& fc, const unsigned long long* sub, const EnsTotal* etot, const float4* colour,
                     uint32_t E, float* feat, cudaStream_t st) {
    const uint32_t P = fc.W * fc.H;
    if (P == 0 || E == 0) return;
    launch_pdl(k_features, dim3((P + 255) / 256), dim3(256), 0, st, fc, sub, etot, colour, E, feat);
}

// A new accumulation window: the accumulator and the window's counter to zero.
__global__ void __launch_bounds__(256) k_clear_accum(float4* __restrict__ accum, uint64_t P, ull* counter) {
    grid_dependency_wait();
    launch_dependents();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t k = i; k < P; k += gridDim.x * blockDim.x) accum[k] = make_float4(F_(0.0), F_(0.0), F_(0.0), F_(0.0));
    if (i == 0) *counter = 0ull;
}
void launch_clear_accum(float4* accum, uint64_t P, unsigned long long* counter, cudaStream_t st) {
    launch_pdl(k_clear_accum, dim3((uint32_t)std::min<uint64_t>((P + 255u) / 256u, 148u * 16u)), dim3(256), 0, st, accum, P, counter);
}

__global__ void k_add_stat(ull* stats, int word, ull v) { stats[word] += v; }
void launch_add_stat(unsigned long long* stats, int word, unsigned long long v, cudaStream_t st) {
    k_add_stat<<<1, 1, 0, st>>>(stats, word, v);
}

// ----------------------------------------------------------------------------- debug probes
// The shared maths evaluated on the device, as the kernels evaluate it: which 0 exp, 1 log, 2 sin,
// 3 cos, 4 log for positive normal arguments, with the tables staged in shared memory (the
// particle kernel's form); which | 8: the same functions reading the global tables (the form of
// the other kernels).
__global__ void __launch_bounds__(256) k_debug_fmath(uint32_t which, const float* __restrict__ in,
                                                     float* __restrict__ out, uint64_t n) {
    __shared__ __align__(16) float s_tab[kTabFloats];
    const FTabs T = stage_tabs(s_tab);
    __syncthreads();
    const bool global = (which & 8u) != 0u;
    const uint32_t op = which & 7u;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float x = in[i];
        float y, sn, cs;
        if (op == 0u) {
            y = global ? gx::exp(x) : gx::exp_t(x, T.ex);
        } else if (op == 1u) {
            y = global ? gx::log(x) : gx::log_t(x, T.lg);
        } else if (op == 4u) {
            y = gx::log_t_pos(x, global ? gx::tab_log() : T.lg);
        } else {
            if (global) gx::sincos(x, &sn, &cs); else gx::sincos_t(x, T.sc, &sn, &cs);
            y = op == 2u ? sn : cs;
        }
        out[i] = y;
    }
}

void launch_debug_fmath(uint32_t which, const float* in, float* out, uint64_t n, cudaStream_t st) {
    if (n == 0) return;
    const uint64_t blocks = (n + 255) / 256;
    k_debug_fmath<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, st>>>(which, in, out, n);
}

// For each particle p in [p0, p0 + n) of one ensemble's compact (splat id, offset) list: its splat
// i (the last entry with offset <= p, found with the particle kernel's 32-ary warp search), its
// index k within the splat and its stream seed particle_seed(i, k + 1, seed). out: 3 words per
// particle. One warp per 32 consecutive particles; the host checks p0 + n <= the list's total.
__global__ void __launch_bounds__(128) k_debug_seeds(const uint2* __restrict__ L, uint32_t nonzero, uint64_t p0,
                                                     uint32_t n, uint32_t seed, uint32_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u;
    if (base >= n) return;  // warp-uniform
    const uint32_t m = n - base < 32u ? n - base : 32u;
    for (uint32_t q = 0; q < m; ++q) {
        const uint64_t p = p0 + base + q;
        const uint32_t j = warp_last_le(L, 0u, nonzero, p, lane);
        if (lane == 0) {
            const uint2 e = L[j];
            const uint32_t k = (uint32_t)(p - e.y);
            out[3u * (base + q)] = e.x;
            out[3u * (base + q) + 1u] = k;
            out[3u * (base + q) + 2u] = gx::particle_seed(e.x, k + 1u, seed);
        }
    }
}

void launch_debug_seeds(const uint2* list, uint32_t nonzero, uint64_t p0, uint32_t n, uint32_t seed, uint32_t* out,
                        cudaStream_t st) {
    if (n == 0 || nonzero == 0) return;
    const uint32_t warps = (n + 31u) / 32u;
    k_debug_seeds<<<(warps + 3u) / 4u, 128, 0, st>>>(list, nonzero, p0, n, seed, out);
}

int device_sm_count(int device) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
    return n;
}

}  // namespace gpsb
