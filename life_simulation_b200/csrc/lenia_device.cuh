// life_simulation_b200/csrc/lenia_device.cuh -- device helpers shared by
// every Lenia kernel: the PCG hash (bit-exact with the reference), and the
// growth map + Euler step + noise + blob injection + clip epilogue.
#pragma once
#include <cstdint>

#include "lenia_types.h"

namespace lenia {

// pcg_hash, Shaders/Common/Random.metal:5-9 (integer, bit-exact).
__host__ __device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {
    uint32_t state = v * 747796405u + 2891336453u;
    uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
    return (word >> 22u) ^ word;
}

// rand01, Shaders/Common/Random.metal:16-19: top 24 bits / 2^24, exact in f32.
__host__ __device__ __forceinline__ float rand01(uint32_t px, uint32_t py, uint32_t tag,
                                                 uint32_t seed) {
    uint32_t h = pcg_hash(px ^ pcg_hash(py ^ pcg_hash(tag ^ seed)));
    return float(h >> 8) * (1.0f / 16777216.0f);
}

// rand01 with its two inner hashes taken out: `row` is rand_row(py, base),
// `base` = pcg_hash(tag ^ seed) (the same value, one hash per pixel).
__device__ __forceinline__ uint32_t rand_row(uint32_t py, uint32_t base) { return pcg_hash(py ^ base); }
__device__ __forceinline__ float rand01_row(uint32_t px, uint32_t row) {
    return float(pcg_hash(px ^ row) >> 8) * (1.0f / 16777216.0f);
}

// The values of a substep that every pixel's noise, mu jitter and injection
// share, computed once per CTA (in shared memory): the blob centres (six
// hashes a blob, which the per-pixel form of the shader repeats for every
// pixel), the field's aspect and the blobs' squared radius, and the seeds'
// hashes.
constexpr int kBlobs = 32;  // blobs kept; further ones are hashed per pixel
struct GrowthExtras {
    float cx[kBlobs], cy[kBlobs];
    float aspect, blob_k, far2;  // blob_k: -1 / (2 blob radius^2)
    uint32_t noise_base, jitter_base;
};
// Filled by the CTA's first threads (blockDim.x >= kBlobs); the caller puts a
// block barrier between this and the first use.
__device__ __forceinline__ void growth_extras_init(GrowthExtras& ex, const StepParams& p) {
    const uint32_t i = threadIdx.x;
    if (i == 0) {
        const float blobR = float(p.radius) * 0.9f / float(p.height);
        ex.aspect = float(p.width) / float(p.height);
        ex.blob_k = -0.5f / (blobR * blobR);
        ex.far2 = 210.0f * (blobR * blobR);
        ex.noise_base = pcg_hash(503u ^ p.seed);
        ex.jitter_base = pcg_hash((401u + p.audio_frame % 613u) ^ p.seed);
    }
    if (p.inject_amount > 0.0f && i < uint32_t(kBlobs) && i < p.inject_count) {
        const uint32_t cycle = p.frame_index / 12u;
        ex.cx[i] = rand01(i, cycle, 811u, p.seed);
        ex.cy[i] = rand01(cycle, i, 823u, p.seed);
    }
}

// The per-pixel mu shift of muJitter (Lenia.metal:89-93 and :176-180);
// `row` = rand_row(gy, ex.jitter_base).
__device__ __forceinline__ float mu_jitter_shift(const StepParams& p, uint32_t gx, uint32_t row) {
    return (rand01_row(gx, row) - 0.5f) * p.mu_jitter * 0.05f;
}

// bell(u; mu, sigma) = exp(-0.5 t^2), t = (u - mu) / sigma (Lenia.metal:156-159).
__device__ __forceinline__ float bell(float u, float mu, float sigma) {
    const float t = (u - mu) / sigma;
    return expf(-0.5f * t * t);
}
// A pixel's growth sum with one more kernel's term, in the reference's order
// (Lenia.metal:188-195): sum_k h_k bell_k (asymptotic) or sum_k h_k (2 bell_k - 1).
__device__ __forceinline__ float growth_add(float sum, float h, float b, bool asym) {
    return fmaf(h, asym ? b : 2.0f * b - 1.0f, sum);
}

// 2^x by the SFU's approximate base-2 exponential (relative error < 2^-22,
// subnormal results flushed to zero).
__device__ __forceinline__ float ex2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One kernel's growth terms at a pixel pair of the spectral row passes, where
// the map is a large share: a precomputed 1/sigma and one hardware base-2
// exponential (relative error below 2^-22) for the division and the full-range
// expf of `bell`, under the transforms' own rounding.
// bell(u) = exp(-(u - mu)^2 / (2 sigma^2)) = 2^-((u*sc - mu*sc)^2) with
// sc = sqrt(log2(e) / 2) / sigma, and the term h * (2 bell - 1) (growth mode
// 0) or h * bell (mode 1) as g1 * bell + g0 -- in packed FP32x2 pairs (one
// FFMA2, one FMUL2, two SFU exponentials, one FFMA2 per pair). With mu
// jitter the pair's centres come per pixel (mu + shift).
struct GrowthPair {
    float mu, sc;
    float2 SC, MSC, G1, G0;
    __device__ __forceinline__ GrowthPair(float mu_, float inv_sigma, float h, bool asym) : mu(mu_) {
        sc = inv_sigma * 0.84932180028801904272f;
        SC = make_float2(sc, sc);
        MSC = make_float2(-mu * sc, -mu * sc);
        const float g1 = asym ? h : 2.0f * h, g0 = asym ? 0.0f : -h;
        G1 = make_float2(g1, g1);
        G0 = make_float2(g0, g0);
    }
    // u: the potentials of the pixel pair.
    __device__ __forceinline__ float2 term(float2 u) const { return bells(__ffma2_rn(u, SC, MSC)); }
    // The same with the pair's mu shifts.
    __device__ __forceinline__ float2 term(float2 u, float2 shift) const {
        return bells(make_float2((u.x - (mu + shift.x)) * sc, (u.y - (mu + shift.y)) * sc));
    }
    // The difference u - mu taken first, which is exact near mu: u * sc - mu * sc
    // adds the rounding of mu * sc, and with it the map's error shows beside the
    // transforms' (RMS of a step against 64 bits at 810 x 486: 2.41e-8 with
    // `term`, 2.34e-8 with this and with `bell` alike; a 1280 x 720 substep alone
    // 23.2, 23.9 and 27.5 us).
    __device__ __forceinline__ float2 term_near(float2 u, float2 shift) const {
        return bells(__fmul2_rn(__fadd2_rn(u, make_float2(-(mu + shift.x), -(mu + shift.y))), SC));
    }
    // d: (u - mu) * sc for both pixels.
    __device__ __forceinline__ float2 bells(float2 d) const {
        const float2 q = __fmul2_rn(d, d);
        const float2 b = make_float2(ex2_fast(-q.x), ex2_fast(-q.y));
        return __ffma2_rn(b, G1, G0);
    }
};

__device__ __forceinline__ float bell_fast(float u, float mu, float inv_sigma) {
    const float t = (u - mu) * inv_sigma;
    return ex2_fast(-0.72134752044448170368f * t * t);
}

// Euler step (Lenia.metal:197-209, identical to leniaStep's for one kernel of
// weight 1); s: the mode's growth sum, sum_k h_k * bell_k (asymptotic) or
// sum_k h_k * (2 bell_k - 1), in kernel order (Lenia.metal:188-195).
struct EulerStep {
    float dt, sum_weights;
    bool asym, weighted, divides;
    __device__ __forceinline__ explicit EulerStep(const StepParams& p)
        : dt(p.dt), sum_weights(p.sum_weights), asym(p.growth_mode == 1u), weighted(p.sum_weights > 1e-6f),
          divides(asym && weighted && p.sum_weights != 1.0f) {}
    // The sums divided by the weights' sum, where that is not one: in a branch
    // around all of a thread's sums, since the compiler divides first and selects
    // then where each has its own (1920 x 1080 spectral, three kernels of weight sum
    // one, four substeps 154 -> 149 us; byte form with blobs 35.4 -> 33.7 us).
    template <int N>
    __device__ __forceinline__ void divide(float (&s)[N]) const {
        if (divides) {
#pragma unroll
            for (int i = 0; i < N; ++i) s[i] = s[i] / sum_weights;
        }
    }
    // dA / dt from a divided sum.
    __device__ __forceinline__ float rate(float A, float s) const { return asym ? (weighted ? s : A) - A : s; }
    __device__ __forceinline__ float operator()(float A, float s) const { return fmaf(dt, rate(A, s), A); }
    // With its product rounded before the sum: how a batch's direct worlds have always
    // stepped, and over a sweep's thousands of substeps a field amplifies a last place.
    __device__ __forceinline__ float rounded(float A, float s) const { return __fadd_rn(A, __fmul_rn(dt, rate(A, s))); }
};

// Noise stir, blob injection and clip (Lenia.metal:210-231) of the N pixels
// (gx, gy) .. (gx + N - 1, gy).
//
// Bound by instructions, so what the pixels share is done once: the blob
// centres once per CTA (GrowthExtras), a blob's dy once for the N pixels.
// A bump exp(-r2 / 2) is exactly zero in FP32 beyond r2 = 208 and the
// injection then leaves a finite A as it is: those pixels (a blob reaches
// 14.4 blob radii, 170 pixels at R = 13) skip the exponential, all N at once
// where the row is that far away; far2 = 210 radii^2 keeps the test on the
// safe side of its rounding.
// Back-to-back frames before (every pixel hashing every centre, a division
// and an exponential per blob) and after: 1920x1080 direct R = 13 with four
// blobs 94.9 -> 66.9 us, 1001x703 R = 9 with noise, jitter and blobs (two
// substeps) 50.4 -> 41.1 us, 1024x512 spectral with three kernels and blobs
// 18.9 -> 15.0 us.
// Within reach all N take the exponential, without a branch per pixel between
// them (a far pixel's bump is the exact zero): 1920x1080 on the byte form, two
// substeps with four blobs, noise and jitter 65.4 -> 61.9 us.
template <int N>
__device__ __forceinline__ void noise_inject_clip(const StepParams& p, const GrowthExtras& ex, float (&A2)[N],
                                                  uint32_t gx, uint32_t gy) {
    if (p.noise_amount > 0.0f) {
        const uint32_t row = rand_row(gy, ex.noise_base);
#pragma unroll
        for (int i = 0; i < N; ++i) A2[i] += (rand01_row(gx + uint32_t(i), row) - 0.5f) * p.noise_amount * 0.03f;
    }
    if (p.inject_amount > 0.0f) {
        const float uvy = (float(gy) + 0.5f) / float(p.height);
        float uvx[N];
        bool finite = true;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            uvx[i] = (float(gx + uint32_t(i)) + 0.5f) / float(p.width);
            finite = finite && fabsf(A2[i]) <= 3.4028234663852886e38f;
        }
        const float far2 = finite ? ex.far2 : __int_as_float(0x7f800000);
        for (uint32_t b = 0; b < p.inject_count; ++b) {
            const bool kept = b < uint32_t(kBlobs);
            const uint32_t cycle = p.frame_index / 12u;
            float dy = uvy - (kept ? ex.cy[b] : rand01(cycle, b, 823u, p.seed));
            dy = dy - roundf(dy);
            if (dy * dy > far2) continue;
            const float cx = kept ? ex.cx[b] : rand01(b, cycle, 811u, p.seed);
            float d2[N];
            bool near = false;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                float dx = uvx[i] - cx;
                dx = dx - roundf(dx);
                dx *= ex.aspect;
                d2[i] = dx * dx + dy * dy;
                near = near || !(d2[i] > far2);
            }
            if (!near) continue;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const float bump = expf(d2[i] * ex.blob_k);
                const float a = fminf(fmaxf(bump * p.inject_amount, 0.0f), 1.0f);
                A2[i] = A2[i] + (0.6f - A2[i]) * a;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) A2[i] = fminf(fmaxf(A2[i], 0.0f), 1.0f);
}

// Out-of-line copies for kernels whose code size matters (the spectral row
// passes): noise, injection and mu jitter are rare, and inlining them grows
// the kernel past the instruction cache. The pixel pair (gx, gy), (gx + 1,
// gy); s: the mode's growth sums.
static __device__ __noinline__ float2 growth_finish_pair(const StepParams& p, const GrowthExtras& ex, float2 A,
                                                         float2 s, uint32_t gx, uint32_t gy) {
    const EulerStep euler(p);
    float v[2] = {s.x, s.y};
    euler.divide(v);
    v[0] = euler(A.x, v[0]);
    v[1] = euler(A.y, v[1]);
    noise_inject_clip(p, ex, v, gx, gy);
    return make_float2(v[0], v[1]);
}
static __device__ __noinline__ float2 mu_jitter_pair(const StepParams& p, const GrowthExtras& ex, uint32_t gx,
                                                     uint32_t gy) {
    const uint32_t row = rand_row(gy, ex.jitter_base);
    return make_float2(mu_jitter_shift(p, gx, row), mu_jitter_shift(p, gx + 1u, row));
}

}  // namespace lenia
