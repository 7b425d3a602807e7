// simulate.cu -- (d) the Simulator's emitter-phase intensity sum, photon
// statistics and device-side photonisation, batched over frames.
//
// Replaces Simulator::SimulatePart (IAC/Simulator.cpp:662-944) with its kernel
// SimulateCrystal (IAC/kernel.cl:768-859), Crystal::GetEmitters
// (IAC/Crystal.cpp:29-184), ArrayOperators::ScalarPoissonSampling
// (IAC/ArrayOperators.h:25-55) and Detector::CreateSparseHitList
// (IAC/Detector.cpp:926-977), so that simulated frames reach the pair
// correlator without leaving the GPU.
//
//  crystal_emitters_kernel   one CTA per (frame, mode): the frame's random
//                            orientation (axis uniform in the unit ball scaled
//                            by the isotropy, angle uniform), the rotated atom
//                            positions, per-mode fluorescence roll and phases;
//                            the event matrix is the inverse rotation.
//  simulate_kernel           two pixels per thread, grid over (pixels, frames):
//                            per mode and sub-pixel, Psi = sum_j exp(i(k.r_j +
//                            phi_j)) with the phase argument formed in FP32 in
//                            the reference's order, then |Psi| (reference) or
//                            |Psi|^2 summed over modes as the host does.
//  frame_sum_kernel          per-frame integrated intensity (double).
//  photon_kernel             rescale to the expected photon number, Poisson
//                            draw (inversion below 25, clipped Box-Muller above),
//                            optional ADU noise, value per photon.
//  sparsify_*                stream compaction of photon frames into the
//                            (k, count) photon lists of the pair correlator,
//                            pixel order kept.
//
// Sine and cosine: the phase argument (|arg| up to ~10^2 rad) is reduced to
// [-pi, pi] explicitly with a two-word Cody-Waite split of 2*pi (the split is
// computed from pi in double below) and evaluated with the SFU's __sincosf, or
// (accurate mode) with sincosf.  Accuracy against an FP64 evaluation is
// measured by the tests.
#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

#include "iac_internal.cuh"
#include "rng.cuh"

namespace iac {

namespace cg = cooperative_groups;

constexpr double TWO_PI_D = 6.283185307179586476925286766559;
constexpr float TWO_PI_HI = (float)TWO_PI_D;
constexpr float TWO_PI_LO = (float)(TWO_PI_D - (double)TWO_PI_HI);
constexpr float INV_TWO_PI = (float)(1.0 / TWO_PI_D);

// The whole number of turns in a phase, rintf(arg / 2 pi) with ties to even, is
// formed by two FP32 adds on the FMA pipe: x + 1.5 * 2^23 rounds x to an integer in
// the float's last place for |x| < 2^22 (phases below 2.6e7 rad; past that an FP32
// phase has lost every fraction of a turn anyway).  rintf is a conversion-unit
// instruction, and that unit also runs the two MUFU operations of every term,
// which bound the simulator.

struct CrystalArgs {
    const double *__restrict__ atoms;  // 3 doubles per atom
    uint32_t natoms, nframes, nmodes;
    uint64_t seed;
    float yield;
    float isotropy;
    int rand_orientation;
    int incoherent;
    float4 *__restrict__ em;        // [frame][mode][atom] (x, y, z, phase)
    uint32_t *__restrict__ em_count;  // [frame][mode]
    float *__restrict__ rot_event;  // 9 per frame (inverse of the crystal rotation)
    float *__restrict__ rot_crystal;  // 9 per frame (may be null)
};

// Crystal::RotateVectors matrix (IAC/Crystal.cpp:125-157) in double.
__device__ void axis_angle(double alpha, double ax0, double ax1, double ax2, double m[9])
{
    const double N = sqrt(ax0 * ax0 + ax1 * ax1 + ax2 * ax2);
    ax0 /= N;
    ax1 /= N;
    ax2 /= N;
    const double c = cos(alpha), s = sin(alpha);
    m[0] = ax0 * ax0 * (1 - c) + c;
    m[1] = ax1 * ax0 * (1 - c) - ax2 * s;
    m[2] = ax2 * ax0 * (1 - c) + ax1 * s;
    m[3] = ax0 * ax1 * (1 - c) + ax2 * s;
    m[4] = ax1 * ax1 * (1 - c) + c;
    m[5] = ax2 * ax1 * (1 - c) - ax0 * s;
    m[6] = ax0 * ax2 * (1 - c) - ax1 * s;
    m[7] = ax1 * ax2 * (1 - c) + ax0 * s;
    m[8] = ax2 * ax2 * (1 - c) + c;
}

__global__ void crystal_emitters_kernel(const CrystalArgs a)
{
    const uint32_t f = blockIdx.x / a.nmodes, mode = blockIdx.x % a.nmodes;
    __shared__ double s_m[9];
    __shared__ uint32_t s_count;
    if (threadIdx.x == 0) {
        double m[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        if (a.rand_orientation) {
            // IAC/Crystal.cpp:53-69: axis uniform in the unit ball (rejection,
            // bounded; the acceptance rate is pi/6), angle uniform in [0, 2 pi)
            double v0 = 0, v1 = 0, v2 = 1;
            for (uint32_t t = 0; t < 256; t++) {
                double u0, u1, u2, u3;
                uniform2(a.seed, RNG_ROTATION | f, 2 * (uint64_t)t, u0, u1);
                uniform2(a.seed, RNG_ROTATION | f, 2 * (uint64_t)t + 1, u2, u3);
                v0 = u0 * 2. - 1.;
                v1 = (u1 * 2. - 1.) * a.isotropy;
                v2 = (u2 * 2. - 1.) * a.isotropy;
                if (!(v0 * v0 + v1 * v1 + v2 * v2 > 1) && (v0 != 0 || v1 != 0 || v2 != 0)) break;
            }
            double ua, ub;
            uniform2(a.seed, RNG_ROTATION | f, 1u << 20, ua, ub);
            axis_angle(ua * 2 * 3.14159265358979323846, v0, v1, v2, m);
        }
        // the crystal matrix is kept in float, as the reference's array<float,9>
        float R[9];
        for (int k = 0; k < 9; k++) R[k] = (float)m[k];
        for (int k = 0; k < 9; k++) s_m[k] = m[k];
        if (mode == 0) {
            // event matrix = inverse of the float crystal matrix, in double
            const double A = R[0], B = R[1], C = R[2], D = R[3], E = R[4], F = R[5], G = R[6],
                         H = R[7], I = R[8];
            const double c0 = E * I - F * H, c1 = -(D * I - F * G), c2 = D * H - E * G;
            const double det = A * c0 + B * c1 + C * c2;
            float *o = a.rot_event + 9 * (size_t)f;
            o[0] = (float)(c0 / det);
            o[1] = (float)(-(B * I - C * H) / det);
            o[2] = (float)((B * F - C * E) / det);
            o[3] = (float)(c1 / det);
            o[4] = (float)((A * I - C * G) / det);
            o[5] = (float)(-(A * F - C * D) / det);
            o[6] = (float)(c2 / det);
            o[7] = (float)(-(A * H - B * G) / det);
            o[8] = (float)((A * E - B * D) / det);
            if (a.rot_crystal)
                for (int k = 0; k < 9; k++) a.rot_crystal[9 * (size_t)f + k] = R[k];
        }
        s_count = 0;
    }
    __syncthreads();
    const size_t base = ((size_t)f * a.nmodes + mode) * a.natoms;
    // atoms kept with probability FlYield (IAC/Crystal.cpp:35-43), in order
    for (uint32_t i0 = 0; i0 < a.natoms; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        bool keep = false;
        double phase = 0.0;
        if (i < a.natoms) {
            keep = true;
            if (a.yield < 1.0f) {
                double y0, y1;
                uniform2(a.seed, RNG_YIELD | ((uint64_t)mode << 32) | f, i, y0, y1);
                keep = y0 <= (double)a.yield;
            }
            if (a.incoherent) {
                double p0, p1;
                uniform2(a.seed, RNG_PHASE | ((uint64_t)mode << 32) | f, i, p0, p1);
                phase = p0 * 2.0 * 3.14159265358979323846;
            }
        }
        // order-preserving compaction within the chunk
        const unsigned ball = __ballot_sync(0xffffffffu, keep);
        __shared__ uint32_t s_w[32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) s_w[w] = __popc(ball);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t t = s_count;
            for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
                const uint32_t c = s_w[k];
                s_w[k] = t;
                t += c;
            }
            s_count = t;
        }
        __syncthreads();
        if (keep) {
            const double *p = a.atoms + 3 * (size_t)i;
            const double x = s_m[0] * p[0] + s_m[1] * p[1] + s_m[2] * p[2];
            const double y = s_m[3] * p[0] + s_m[4] * p[1] + s_m[5] * p[2];
            const double z = s_m[6] * p[0] + s_m[7] * p[1] + s_m[8] * p[2];
            a.em[base + s_w[w] + __popc(ball & ((1u << lane) - 1))] =
                make_float4((float)x, (float)y, (float)z, (float)phase);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) a.em_count[(size_t)f * a.nmodes + mode] = s_count;
}

struct SimArgs {
    const float *__restrict__ pm;  // pixel map, 3 floats per pixel
    const float4 *__restrict__ em;
    const uint32_t *__restrict__ em_count;
    uint64_t npix;
    uint32_t natoms, nmodes, nframes;
    int susa;
    float us[3], vs[3];
    float wavelength;
    int amplitude_sq;  // 0: |Psi| as the reference, 1: |Psi|^2
    int accurate;      // 1: sincosf instead of explicit reduction + SFU
    float neg_zero;    // -0.0f: fma(x, y, -0) is x * y rounded once, and never merges with an add
    float *__restrict__ out;  // [frame][pixel]
};

constexpr int SIM_THREADS = 128;
constexpr int SIM_MAX_EM = 1024;  // emitters staged in shared memory at a time

// Two pixels per thread, p and p + SIM_THREADS: every FP32 operation of a term is
// one f32x2 instruction for both (same roundings as two scalar ones), with the
// emitter staged as pairs (x, x, y, y), (z, z, phase, phase).  Bound by the two
// MUFU operations of a term: 5 x 5 x 8 emitters, 4 modes, 100 frames of 512^2
// 10.8 ms = 0.83 of the SFU rate; with scalar FP32, whose issue slots ran
// out beside the MUFU's, 11.7 ms (0.77).  An emitter list is staged once per mode;
// one longer than SIM_MAX_EM streams through the stage in chunks, in order, for
// every sub-pixel, so each pixel's sums always add the same terms in the same order.
template <bool ACCURATE>
__global__ void __launch_bounds__(SIM_THREADS) simulate_kernel(const SimArgs a)
{
    extern __shared__ float4 s_em[];  // two per emitter
    const uint32_t f = blockIdx.y;
    const uint64_t p0 = blockIdx.x * (uint64_t)(2 * SIM_THREADS) + threadIdx.x, p1 = p0 + SIM_THREADS;
    // a pixel past the end repeats the first, unwritten
    const float *pc0 = a.pm + 3 * (p0 < a.npix ? p0 : 0), *pc1 = a.pm + 3 * (p1 < a.npix ? p1 : 0);
    const float2 c0 = make_float2(pc0[0], pc1[0]), c1 = make_float2(pc0[1], pc1[1]), c2 = make_float2(pc0[2], pc1[2]);
    const float2 nz = make_float2(a.neg_zero, a.neg_zero);
    auto mul = [&](float2 x, float2 y) { return f2fma(x, y, nz); };
    auto dup = [](float x) { return make_float2(x, x); };
    const float nsub = (float)((2 * a.susa + 1) * (2 * a.susa + 1));
    float total0 = 0.0f, total1 = 0.0f;
    for (uint32_t m = 0; m < a.nmodes; m++) {
        const uint32_t n = min(a.em_count[(size_t)f * a.nmodes + m], a.natoms);
        const float4 *src = a.em + ((size_t)f * a.nmodes + m) * a.natoms;
        float acc0 = 0.0f, acc1 = 0.0f;
        bool staged = false;
        for (int v = -a.susa; v <= a.susa; v++)
            for (int u = -a.susa; u <= a.susa; u++) {
                // IAC/kernel.cl:823-832
                auto wave = [&](float x, float y, float z, float k[3]) {
                    x = fadd(fadd(x, fmul((float)v, a.vs[0])), fmul((float)u, a.us[0]));
                    y = fadd(fadd(y, fmul((float)v, a.vs[1])), fmul((float)u, a.us[1]));
                    z = fadd(fadd(z, fmul((float)v, a.vs[2])), fmul((float)u, a.us[2]));
                    float nk = (float)(1.0 / (double)norm3(x, y, z));
                    nk = (float)((double)nk * ((2.0 * 3.1415926535897932) / (double)a.wavelength));
                    k[0] = fmul(x, nk);
                    k[1] = fmul(y, nk);
                    k[2] = fmul(z, nk);
                };
                float ka[3], kb[3];
                wave(c0.x, c1.x, c2.x, ka);
                wave(c0.y, c1.y, c2.y, kb);
                const float2 k0 = make_float2(ka[0], kb[0]), k1 = make_float2(ka[1], kb[1]), k2 = make_float2(ka[2], kb[2]);
                float2 re = make_float2(0.0f, 0.0f), im = re;
                for (uint32_t c = 0; c < n; c += SIM_MAX_EM) {
                    const uint32_t cn = min(n - c, (uint32_t)SIM_MAX_EM);
                    if (!staged) {
                        __syncthreads();  // the last stage is read
                        for (uint32_t i = threadIdx.x; i < cn; i += SIM_THREADS) {
                            const float4 e = src[c + i];
                            s_em[2 * i] = make_float4(e.x, e.x, e.y, e.y);
                            s_em[2 * i + 1] = make_float4(e.z, e.z, e.w, e.w);
                        }
                        __syncthreads();
                        staged = n <= (uint32_t)SIM_MAX_EM;
                    }
#pragma unroll 4
                    for (uint32_t i = 0; i < cn; i++) {
                        const float4 ea = s_em[2 * i], eb = s_em[2 * i + 1];
                        float2 arg = mul(k0, make_float2(ea.x, ea.y));
                        arg = f2add(arg, mul(k1, make_float2(ea.z, ea.w)));
                        arg = f2add(arg, mul(k2, make_float2(eb.x, eb.y)));
                        arg = f2add(arg, make_float2(eb.z, eb.w));
                        float2 sn, cs;
                        if (ACCURATE) {
                            sincosf(arg.x, &sn.x, &cs.x);
                            sincosf(arg.y, &sn.y, &cs.y);
                        } else {
                            // the whole turns of the phase by two adds
                            const float2 t = f2sub(f2add(mul(arg, dup(INV_TWO_PI)), dup(ROUND_MAGIC)), dup(ROUND_MAGIC));
                            const float2 nt = make_float2(-t.x, -t.y);
                            const float2 r = f2fma(nt, dup(TWO_PI_LO), f2fma(nt, dup(TWO_PI_HI), arg));
                            __sincosf(r.x, &sn.x, &cs.x);
                            __sincosf(r.y, &sn.y, &cs.y);
                        }
                        re = f2add(re, cs);
                        im = f2add(im, sn);
                    }
                }
                const float q0 = fadd(fmul(re.x, re.x), fmul(im.x, im.x)), q1 = fadd(fmul(re.y, re.y), fmul(im.y, im.y));
                acc0 = fadd(acc0, a.amplitude_sq ? q0 : __fsqrt_rn(q0));
                acc1 = fadd(acc1, a.amplitude_sq ? q1 : __fsqrt_rn(q1));
            }
        total0 = fadd(total0, __fdiv_rn(acc0, nsub));  // as ParAdd sums modes
        total1 = fadd(total1, __fdiv_rn(acc1, nsub));
    }
    if (p0 < a.npix) a.out[(size_t)f * a.npix + p0] = total0;
    if (p1 < a.npix) a.out[(size_t)f * a.npix + p1] = total1;
}

// per-frame double sum, one CTA per frame: SUM_THREADS chains of adds, each over
// every SUM_THREADS-th pixel, SUM_AHEAD loads ahead of them (100 frames of 512^2 in
// 58 us, 488 with the loads in the chain)
constexpr int SUM_THREADS = 256, SUM_AHEAD = 32;
__global__ void __launch_bounds__(SUM_THREADS) frame_sum_kernel(const float *__restrict__ I, uint64_t npix,
                                                                double *__restrict__ sums)
{
    const uint32_t f = blockIdx.x;
    const float *x = I + (size_t)f * npix + threadIdx.x;
    double s = 0;
    const uint64_t n = npix > threadIdx.x ? (npix - threadIdx.x + SUM_THREADS - 1) / SUM_THREADS : 0;  // of this thread
    uint64_t i = 0;
    for (; i + SUM_AHEAD <= n; i += SUM_AHEAD) {
        float v[SUM_AHEAD];
#pragma unroll
        for (int k = 0; k < SUM_AHEAD; k++) v[k] = x[(i + k) * SUM_THREADS];
#pragma unroll
        for (int k = 0; k < SUM_AHEAD; k++) s += (double)v[k];
    }
    for (; i < n; i++) s += (double)x[i * SUM_THREADS];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ double sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; w++) t += sh[w];
        sums[f] = t;
    }
}

// ScalarPoissonSampling, IAC/ArrayOperators.h:25-55; the sequential search
// stops once the term underflows to zero (a draw the rounded cumulative sum
// never reaches would otherwise not end).
__device__ __forceinline__ uint32_t poisson_draw(double mean, uint64_t seed, uint64_t stream, uint64_t idx)
{
    double u0, u1;
    uniform2(seed, stream, idx, u0, u1);
    double ret;
    if (mean < 25) {
        int i = 0;
        double r = exp(-mean);
        double pcum = r;
        while (pcum < u0 && r > 0) {
            i++;
            r *= mean / i;
            pcum += r;
        }
        ret = i;
    } else {
        const double u = 1 - u0, v = 1 - u1;
        ret = (mean + sqrt(mean) * sqrt(-2. * log(u)) * cos(2. * 3.14159265358979323846 * v));
        if (ret < 0) ret = 0;
    }
    return (uint32_t)ret;
}

struct PhotonArgs {
    float *__restrict__ I;  // in: intensity, out: photon image
    const double *__restrict__ sums;
    uint64_t npix;
    uint32_t nframes;
    uint64_t frame0;        // global index of the first frame (random streams)
    double expected;        // AveragePhotonesPerEmitterOnDetector * FlYield * atoms
    int poisson;
    float adu_noise;
    float value_per_photon;
    uint64_t seed;
};

// the photon image's value of one pixel from its rescaled intensity
__device__ __forceinline__ float photon_finish(const PhotonArgs &a, float v, uint64_t gf, uint64_t p)
{
    if (a.adu_noise != 0.0f) {
        double n0, n1;
        uniform2(a.seed, RNG_NOISE | gf, p, n0, n1);
        v = fadd(v, (float)((2 * n0 - 1) * a.adu_noise));
    }
    return fmul(v, a.value_per_photon);
}

// A block takes PHOTON_PIX pixels of a frame.  At the few hundredths of a photon
// per pixel of these images nearly every draw is 0, and that needs no exponential:
// u0 < 1 - mean implies u0 < exp(-mean), where the search ends at 0.  The test is
// made on the top 32 bits of u0's integer, with a margin of 2^-16 for the FP32
// arithmetic on the right.  The pixels that fail it
// are collected in shared memory and drawn in full, a thread each, so that whole
// warps run the FP64 search instead of the few lanes of every warp that need it.
// 100 images of 512^2 at 0.02 photons: 146 us, 254 with a search per pixel.
constexpr int PHOTON_THREADS = 256, PHOTON_PER = 8, PHOTON_PIX = PHOTON_THREADS * PHOTON_PER;

__global__ void __launch_bounds__(PHOTON_THREADS) photon_kernel(const PhotonArgs a)
{
    __shared__ uint16_t s_list[PHOTON_PIX];
    __shared__ float s_mean[PHOTON_PIX];
    __shared__ uint32_t s_n;
    const uint32_t f = blockIdx.y;
    const uint64_t gf = a.frame0 + f, p0 = blockIdx.x * (uint64_t)PHOTON_PIX;
    float *row = a.I + (size_t)f * a.npix;
    // IAC/Simulator.cpp:871-894: factor in double, applied as float
    const float factor = (float)(a.expected / a.sums[f]);
    if (threadIdx.x == 0) s_n = 0u;
    __syncthreads();
    float x[PHOTON_PER];
#pragma unroll
    for (int k = 0; k < PHOTON_PER; k++) {
        const uint64_t p = p0 + k * PHOTON_THREADS + threadIdx.x;
        x[k] = p < a.npix ? row[p] : 0.0f;
    }
#pragma unroll 2
    for (int k = 0; k < PHOTON_PER; k++) {
        const uint32_t at = k * PHOTON_THREADS + threadIdx.x;
        const uint64_t p = p0 + at;
        if (p >= a.npix) break;
        const float v = fmul(x[k], factor);
        if (!a.poisson) {
            row[p] = photon_finish(a, v, gf, p);
            continue;
        }
        // (1 - v - 2^-16) 2^32; a v outside [0, 1) or NaN is drawn in full
        const float room = (1.0f - v) * 4294967296.0f - 65536.0f;
        bool zero = false;
        if (v >= 0.0f && room > 0.0f) {
            uint32_t c[4] = {(uint32_t)p, (uint32_t)(p >> 32), (uint32_t)(RNG_POISSON | gf),
                             (uint32_t)((RNG_POISSON | gf) >> 32)};
            philox4x32_10(c, (uint32_t)a.seed, (uint32_t)(a.seed >> 32));
            zero = c[0] < __float2uint_rz(room);
        }
        if (zero) {
            row[p] = photon_finish(a, 0.0f, gf, p);
        } else {
            const uint32_t o = atomicAdd(&s_n, 1u);
            s_list[o] = (uint16_t)at;
            s_mean[o] = v;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < s_n; i += PHOTON_THREADS) {
        const uint64_t p = p0 + s_list[i];
        row[p] = photon_finish(a, (float)poisson_draw((double)s_mean[i], a.seed, RNG_POISSON | gf, p), gf, p);
    }
}

// ---------------------------------------------------------------------------
// CreateSparseHitList on the device: photons = pixels with I >= Threshold and
// I > 0 (after the pixel mask), value photonised as ceil((I - T) / Step).
// Pass 1 reads the frames, counts the photons of every tile of SPARSE_PIX pixels
// and keeps a bit per pixel; the counts are scanned; pass 2 ranks the bits and
// reads only the pixels that have one, in pixel order.  Bound by reading the
// frames once (pass 1): 200 frames of 1024 x 512 with 1 % hits in 138 us,
// 68 at the copy rate; reading them twice with a block-wide rank per 256 pixels
// took 506.  One pass whose tiles look back at their predecessors' counts took
// 316: with a thousand tiles in flight the looking back outlasts the reading.
// ---------------------------------------------------------------------------
constexpr int SPARSE_THREADS = 256;
constexpr int SPARSE_ROUNDS = 4;                                    // four pixels per thread and round
constexpr int SPARSE_PIX = 4 * SPARSE_THREADS * SPARSE_ROUNDS;      // pixels per tile
constexpr int SPARSE_WARPS = SPARSE_THREADS / 32;

// the value of pixel p of a frame
__device__ __forceinline__ float hit_value(const float *row, const int *mask, uint64_t p)
{
    const float v = row[p];
    return mask ? fmul(v, (float)__ldg(mask + p)) : v;
}
__device__ __forceinline__ bool is_hit(float v, float thr) { return v >= thr && v > 0.0f; }

// this thread's 16 pixels of a tile as bits, bit 4 r + e for pixel e of round r
template <bool VEC>  // rows of frames and mask are 16-byte aligned
__device__ __forceinline__ uint32_t hit_bits(const float *__restrict__ row, const int *__restrict__ mask, uint64_t npix,
                                             uint64_t p0, float thr)
{
    uint32_t bits = 0;
    if (VEC) {
        float4 x[SPARSE_ROUNDS];
#pragma unroll
        for (int r = 0; r < SPARSE_ROUNDS; r++) {
            const uint64_t p = p0 + 4 * (uint64_t)(r * SPARSE_THREADS + threadIdx.x);
            // npix % 4 == 0: four pixels are whole or absent
            x[r] = p < npix ? __ldcs(reinterpret_cast<const float4 *>(row + p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < SPARSE_ROUNDS; r++) {
            const uint64_t p = p0 + 4 * (uint64_t)(r * SPARSE_THREADS + threadIdx.x);
            if (mask && p < npix) {
                const int4 m = __ldg(reinterpret_cast<const int4 *>(mask + p));
                x[r] = make_float4(fmul(x[r].x, (float)m.x), fmul(x[r].y, (float)m.y), fmul(x[r].z, (float)m.z),
                                   fmul(x[r].w, (float)m.w));
            }
            bits |= ((is_hit(x[r].x, thr) ? 1u : 0u) | (is_hit(x[r].y, thr) ? 2u : 0u) | (is_hit(x[r].z, thr) ? 4u : 0u) |
                     (is_hit(x[r].w, thr) ? 8u : 0u))
                    << (4 * r);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4 * SPARSE_ROUNDS; k++) {
            const uint64_t p = p0 + 4 * (uint64_t)(k / 4 * SPARSE_THREADS + threadIdx.x) + k % 4;
            if (p < npix && is_hit(hit_value(row, mask, p), thr)) bits |= 1u << k;
        }
    }
    return bits;
}

template <bool VEC>
__global__ void __launch_bounds__(SPARSE_THREADS)
    sparsify_count_kernel(const float *__restrict__ I, const int *__restrict__ mask, uint64_t npix, float thr,
                          uint32_t *__restrict__ counts, uint16_t *__restrict__ bits_out)
{
    const uint64_t tile = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x;
    const uint32_t bits = hit_bits<VEC>(I + (size_t)blockIdx.y * npix, mask, npix, (uint64_t)blockIdx.x * SPARSE_PIX, thr);
    if (bits_out) bits_out[tile * SPARSE_THREADS + threadIdx.x] = (uint16_t)bits;
    __shared__ uint32_t s[SPARSE_WARPS];
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(bits));
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < SPARSE_WARPS; w++) t += s[w];
        counts[tile] = t;
    }
}

// exclusive scan of counts (n entries, 16-byte aligned) into offs (n + 1 entries):
// one cluster, every CTA a contiguous share, four entries per thread at a time
constexpr int SCAN_CTAS = 8;
__global__ void __cluster_dims__(SCAN_CTAS, 1, 1) __launch_bounds__(1024)
    scan_u32_kernel(const uint32_t *__restrict__ counts, uint64_t n, uint64_t *__restrict__ offs)
{
    __shared__ unsigned long long s_mine;
    __shared__ uint32_t ws[2][32];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t rank = cl.block_rank();
    const uint64_t quads = (n + 3) / 4, b0 = 4 * (quads * rank / SCAN_CTAS),
                   b1 = min(n, 4 * (quads * (rank + 1) / SCAN_CTAS));
    auto load = [&](uint64_t i) {
        uint4 c = make_uint4(0u, 0u, 0u, 0u);
        if (i + 3 < b1) {
            c = *reinterpret_cast<const uint4 *>(counts + i);
        } else {
            if (i < b1) c.x = counts[i];
            if (i + 1 < b1) c.y = counts[i + 1];
            if (i + 2 < b1) c.z = counts[i + 2];
        }
        return c;
    };
    if (tid == 0) s_mine = 0ull;
    __syncthreads();
    unsigned long long sum = 0;
    for (uint64_t i = b0 + 4 * tid; i < b1; i += 4096) {
        const uint4 c = load(i);
        sum += c.x + c.y + c.z + c.w;  // four tiles: 32 bits
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && sum) atomicAdd(&s_mine, sum);
    cl.sync();
    uint64_t run = 0, total = 0;
    for (uint32_t r = 0; r < SCAN_CTAS; r++) {
        const unsigned long long v = *cl.map_shared_rank(&s_mine, r);
        run += r < rank ? v : 0ull;
        total += v;
    }
    cl.sync();  // no CTA leaves while its sum is read
    for (uint64_t i0 = b0, k = 0; i0 < b1; i0 += 4096, k++) {  // at most 4096 * SPARSE_PIX photons a time: 32 bits
        const uint64_t i = i0 + 4 * tid;
        const uint4 c = load(i);
        const uint32_t mine = c.x + c.y + c.z + c.w;
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) ws[k & 1][w] = incl;
        __syncthreads();
        const uint32_t t = ws[k & 1][lane];
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? t : 0u),
                       all = __reduce_add_sync(0xffffffffu, t);
        uint64_t o = run + before + incl - mine;
        if (i < b1) offs[i] = o;
        if (i + 1 < b1) offs[i + 1] = o += c.x;
        if (i + 2 < b1) offs[i + 2] = o += c.y;
        if (i + 3 < b1) offs[i + 3] = o += c.z;
        run += all;
    }
    if (rank == 0 && tid == 0) offs[n] = total;
}

template <bool VEC>  // used without the bits of pass 1
__global__ void __launch_bounds__(SPARSE_THREADS)
    sparsify_write_kernel(const float *__restrict__ I, const int *__restrict__ mask, const float *__restrict__ kmap,
                          uint64_t npix, uint32_t nframes, float thr, float step, int photonize,
                          const uint16_t *__restrict__ bits_in, const uint64_t *__restrict__ tile_off,
                          float4 *__restrict__ out, uint64_t capacity, uint64_t *__restrict__ frame_off,
                          DeviceCounters *counters)
{
    __shared__ uint32_t s_count[SPARSE_ROUNDS * SPARSE_WARPS];  // photons of (round, warp)
    __shared__ uint16_t s_hit[SPARSE_PIX];
    const uint32_t f = blockIdx.y;
    const uint64_t tile = (uint64_t)f * gridDim.x + blockIdx.x, p0 = (uint64_t)blockIdx.x * SPARSE_PIX;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint64_t base = tile_off[tile];
    if (tid == 0) {
        // frame offsets, clamped to the capacity so that no consumer reads past the
        // photons actually written; a clamp is counted as an overflow
        if (blockIdx.x == 0) frame_off[f] = min(base, capacity);
        if (f == nframes - 1 && blockIdx.x == gridDim.x - 1) {
            const uint64_t all = tile_off[tile + 1];
            frame_off[nframes] = min(all, capacity);
            if (all > capacity) atomicAdd(&counters->photon_overflow, all - capacity);
        }
    }
    if (tile_off[tile + 1] == base) return;  // an empty tile
    const float *row = I + (size_t)f * npix;
    const uint32_t bits = bits_in ? bits_in[tile * SPARSE_THREADS + tid] : hit_bits<VEC>(row, mask, npix, p0, thr);
    // ranks: a scan over the warp of the rounds' counts, a byte each (128 at most), then over (round, warp)
    uint32_t counts = 0;
#pragma unroll
    for (int r = 0; r < SPARSE_ROUNDS; r++) counts |= (uint32_t)__popc((bits >> (4 * r)) & 15u) << (8 * r);
    uint32_t incl = counts;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31)
#pragma unroll
        for (int r = 0; r < SPARSE_ROUNDS; r++) s_count[r * SPARSE_WARPS + warp] = (incl >> (8 * r)) & 255u;
    __syncthreads();
    static_assert(SPARSE_ROUNDS * SPARSE_WARPS == 32, "one count per lane");
    const uint32_t of_lane = s_count[lane];
    // the tile's hits in order, then a thread per hit: few pixels are hits, and so
    // their loads run side by side and the list is written in whole rows
#pragma unroll
    for (int r = 0; r < SPARSE_ROUNDS; r++) {
        uint32_t o = __reduce_add_sync(0xffffffffu, lane < r * SPARSE_WARPS + warp ? of_lane : 0u) +
                     (((incl - counts) >> (8 * r)) & 255u);
        for (uint32_t b = (bits >> (4 * r)) & 15u; b; b &= b - 1)
            s_hit[o++] = (uint16_t)(4 * (r * SPARSE_THREADS + tid) + (__ffs(b) - 1));
    }
    __syncthreads();
    const uint32_t hits = (uint32_t)(tile_off[tile + 1] - base);
    for (uint32_t h = tid; h < hits && base + h < capacity; h += SPARSE_THREADS) {
        const uint64_t p = p0 + s_hit[h];
        const float v = hit_value(row, mask, p);
        // IAC/ArrayOperators.h:144: ceil((I - T) / Step) * (I >= T)
        const float val = photonize ? ceilf(__fdiv_rn(fsub(v, thr), step)) : v;
        out[base + h] = make_float4(kmap[3 * p], kmap[3 * p + 1], kmap[3 * p + 2], val);
    }
}

}  // namespace iac

using namespace iac;

extern "C" {

iac_status iac_crystal_emitters(iac_ctx *ctx, const double *d_atoms, uint32_t natoms,
                                uint32_t nframes, uint32_t nmodes, const iac_crystal_params *cp,
                                uint64_t seed, float *d_emitters, uint32_t *d_em_count,
                                float *d_rot_event, float *d_rot_crystal, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_atoms && cp && d_emitters && d_em_count && d_rot_event,
                "iac_crystal_emitters: NULL argument");
    IAC_REQUIRE(natoms > 0 && nmodes > 0, "iac_crystal_emitters: no atoms or modes");
    IAC_REQUIRE(cp->fluorescence_yield > 0 && cp->fluorescence_yield <= 1,
                "FluorescenceYield must be in (0, 1]");
    if (nframes == 0) return IAC_OK;
    DeviceGuard g(ctx->device);
    CrystalArgs a;
    a.atoms = d_atoms;
    a.natoms = natoms;
    a.nframes = nframes;
    a.nmodes = nmodes;
    a.seed = seed;
    a.yield = cp->fluorescence_yield;
    a.isotropy = cp->isotropy;
    a.rand_orientation = cp->random_orientation;
    a.incoherent = cp->incoherent;
    a.em = (float4 *)d_emitters;
    a.em_count = d_em_count;
    a.rot_event = d_rot_event;
    a.rot_crystal = d_rot_crystal;
    crystal_emitters_kernel<<<nframes * nmodes, 128, 0, as_stream(stream)>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

iac_status iac_simulate_intensity(iac_ctx *ctx, const float *d_pixel_map, uint64_t npix,
                                  const float *d_emitters, const uint32_t *d_em_count,
                                  uint32_t natoms, uint32_t nmodes, uint32_t nframes,
                                  const iac_sim_params *sp, float *d_intensity, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_pixel_map && d_emitters && d_em_count && sp && d_intensity,
                "iac_simulate_intensity: NULL argument");
    IAC_REQUIRE(npix > 0 && natoms > 0 && nmodes > 0, "iac_simulate_intensity: empty input");
    IAC_REQUIRE(sp->subsampling >= 0 && sp->subsampling <= 16, "SubSampling out of range");
    IAC_REQUIRE(sp->wavelength > 0, "wavelength must be positive");
    IAC_REQUIRE(nframes <= 65535, "at most 65535 frames per call");
    if (nframes == 0) return IAC_OK;
    DeviceGuard g(ctx->device);
    SimArgs a;
    a.pm = d_pixel_map;
    a.em = (const float4 *)d_emitters;
    a.em_count = d_em_count;
    a.npix = npix;
    a.natoms = natoms;
    a.nmodes = nmodes;
    a.nframes = nframes;
    a.susa = sp->subsampling;
    for (int d = 0; d < 3; d++) {
        a.us[d] = (float)sp->u_step[d];
        a.vs[d] = (float)sp->v_step[d];
    }
    a.wavelength = (float)sp->wavelength;
    a.amplitude_sq = sp->intensity_squared;
    a.accurate = sp->accurate_sincos;
    a.out = d_intensity;
    a.neg_zero = -0.0f;
    const dim3 grid((unsigned)((npix + 2 * SIM_THREADS - 1) / (2 * SIM_THREADS)), nframes);
    const size_t smem = 2 * sizeof(float4) * std::min<uint32_t>(natoms, SIM_MAX_EM);
    if (a.accurate)
        simulate_kernel<true><<<grid, SIM_THREADS, smem, as_stream(stream)>>>(a);
    else
        simulate_kernel<false><<<grid, SIM_THREADS, smem, as_stream(stream)>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

iac_status iac_simulate_photons(iac_ctx *ctx, float *d_intensity, uint64_t npix, uint32_t nframes,
                                uint64_t first_frame, const iac_photon_params *pp, uint64_t seed,
                                void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_intensity && pp, "iac_simulate_photons: NULL argument");
    IAC_REQUIRE(nframes <= 65535, "at most 65535 frames per call");
    if (nframes == 0 || npix == 0) return IAC_OK;
    DeviceGuard g(ctx->device);
    void *scr = nullptr;
    iac_status st = stream_scratch(ctx, stream, SLOT_AUX0, sizeof(double) * nframes, &scr);
    if (st != IAC_OK) return st;
    cudaStream_t s = as_stream(stream);
    frame_sum_kernel<<<nframes, SUM_THREADS, 0, s>>>(d_intensity, npix, (double *)scr);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    PhotonArgs a;
    a.I = d_intensity;
    a.sums = (const double *)scr;
    a.npix = npix;
    a.nframes = nframes;
    a.frame0 = first_frame;
    a.expected = pp->expected_photons;
    a.poisson = pp->poisson;
    a.adu_noise = pp->adu_noise;
    a.value_per_photon = pp->value_per_photon;
    a.seed = seed;
    dim3 grid((unsigned)((npix + PHOTON_PIX - 1) / PHOTON_PIX), nframes);
    photon_kernel<<<grid, PHOTON_THREADS, 0, s>>>(a);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    return IAC_OK;
}

iac_status iac_sparsify_frames(iac_ctx *ctx, const float *d_intensity, const int *d_mask,
                               const float *d_kmap, uint64_t npix, uint32_t nframes, float threshold,
                               float step, int photonize, float *d_photons, uint64_t capacity,
                               uint64_t *d_frame_offsets, uint64_t *h_total, void *stream)
{
    IAC_TRACE();
    IAC_REQUIRE(ctx && d_intensity && d_kmap && d_photons && d_frame_offsets,
                "iac_sparsify_frames: NULL argument");
    IAC_REQUIRE(!photonize || step > 0, "photon step must be positive");
    IAC_REQUIRE(nframes <= 65535, "at most 65535 frames per call");
    DeviceGuard g(ctx->device);
    cudaStream_t s = as_stream(stream);
    if (nframes == 0 || npix == 0) {
        IAC_CUDA(cudaMemsetAsync(d_frame_offsets, 0, sizeof(uint64_t) * (nframes + 1), s));
        if (h_total) *h_total = 0;
        return IAC_OK;
    }
    const uint32_t bpf = (uint32_t)((npix + SPARSE_PIX - 1) / SPARSE_PIX);
    const uint64_t nb = (uint64_t)bpf * nframes;
    void *scr = nullptr;
    // counts, offsets, and behind them a bit per pixel; where the context's scratch
    // has no room for the bits, pass 2 reads the frames again
    const size_t counts_bytes = ((sizeof(uint32_t) * nb + 15) / 16) * 16;
    const size_t offs_bytes = ((sizeof(uint64_t) * (nb + 2) + 15) / 16) * 16;
    const size_t bits_bytes = sizeof(uint16_t) * SPARSE_THREADS * nb;
    bool bits = true;
    iac_status st = stream_scratch(ctx, stream, SLOT_AUX1, counts_bytes + offs_bytes + bits_bytes, &scr);
    if (st == IAC_ERR_NO_MEMORY) {
        cudaGetLastError();
        bits = false;
        st = stream_scratch(ctx, stream, SLOT_AUX1, counts_bytes + sizeof(uint64_t) * (nb + 2), &scr);
    }
    if (st != IAC_OK) return st;
    uint32_t *counts = (uint32_t *)scr;
    uint64_t *toff = (uint64_t *)((char *)scr + counts_bytes);
    uint16_t *tbits = bits ? (uint16_t *)((char *)scr + counts_bytes + offs_bytes) : nullptr;
    const bool vec = npix % 4 == 0 && ((uintptr_t)d_intensity & 15) == 0 && ((uintptr_t)d_mask & 15) == 0;
    const dim3 grid(bpf, nframes);
    auto count = vec ? sparsify_count_kernel<true> : sparsify_count_kernel<false>;
    auto write = vec ? sparsify_write_kernel<true> : sparsify_write_kernel<false>;
    count<<<grid, SPARSE_THREADS, 0, s>>>(d_intensity, d_mask, npix, threshold, counts, tbits);
    IAC_LAUNCHED(ctx);
    scan_u32_kernel<<<SCAN_CTAS, 1024, 0, s>>>(counts, nb, toff);
    IAC_LAUNCHED(ctx);
    write<<<grid, SPARSE_THREADS, 0, s>>>(d_intensity, d_mask, d_kmap, npix, nframes, threshold, step, photonize, tbits,
                                          toff, (float4 *)d_photons, capacity, d_frame_offsets, ctx->d_counters);
    IAC_LAUNCHED(ctx);
    IAC_CUDA(cudaGetLastError());
    if (h_total) {
        IAC_CUDA(cudaMemcpyAsync(h_total, toff + nb, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        IAC_CUDA(cudaStreamSynchronize(s));
        if (*h_total > capacity) {
            set_error("photon lists need %llu entries, capacity is %llu",
                      (unsigned long long)*h_total, (unsigned long long)capacity);
            return IAC_ERR_INVALID_ARG;
        }
    }
    return IAC_OK;
}

}  // extern "C"
