// Shared device/host definitions of the legendre B200 library.
//
// Layout (the reference's `State`, src/core/state.rs:219-296): every field of
// every block owns one dense slab of (n_d + 2g) entries per dimension,
// dimension 0 fastest (src/geometry/cartesian.rs:8-11, linearize :189-204).
// On the device all slabs of one state live in a single arena, block-major:
// slab(b, f) starts at arena + (b * nfields + f) * slab_stride, with
// slab_stride the largest field's slab rounded up to 256 bytes, so each slab
// starts 256-byte aligned.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "lg_log_table.h"

#define LG_MAX_DIM 3

namespace lg {

// Per-grid topology as seen by kernels.  `nbr[(b * 3 + d) * 2 + side]` is the
// face neighbour of block b across dimension d (side 0 = low, 1 = high),
// already wrapped in periodic dimensions, or -1 at a physical (mirror)
// boundary -- CartesianGrid::face_neighbor (src/geometry/cartesian.rs:162-181).
struct CartTopo {
    int D;
    int n[LG_MAX_DIM];    // interior cells per block per dimension
    int nb[LG_MAX_DIM];   // blocks per dimension
    int nblocks;
    const int* nbr;       // device table, nblocks * 3 * 2 entries
};

// Slab addressing of one state arena.
struct SlabLayout {
    int nfields;
    int ghost;            // ghost width of the fields a kernel touches
    int64_t slab_stride;  // elements between consecutive slabs
    int64_t len;          // ghost-inclusive slab length of those fields
    int gdim[LG_MAX_DIM]; // n_d + 2g
};

// ------------------------------------------------------------------ rng ---
// Counter-based generator of the reference (src/util/rng.rs:13-49).
__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// mix_key(seed, [salt, stream, block]) -- the per-block key of the Wiener
// driver (src/core/driver.rs:139-158).
__host__ __device__ __forceinline__ uint64_t wiener_block_key(uint64_t seed, uint64_t salt, uint64_t stream,
                                                              uint64_t block) {
    uint64_t s = splitmix64(seed);
    s = splitmix64(s ^ salt);
    s = splitmix64(s ^ stream);
    return splitmix64(s ^ block);
}

__host__ __device__ __forceinline__ double unit_open(uint64_t bits) {
    return (double)((bits >> 11) + 1) * (1.0 / 9007199254740992.0);
}

constexpr double kTau = 6.283185307179586476925286766559;

// ln u for the Box-Muller radius, u = n 2^-53 with n = 1 .. 2^53 exact in a
// double, within 3.5e-16 relative of the exact logarithm (the Gaussian is
// held to 1e-12 of glibc's).  A table-driven reduction (the method of Tang,
// ACM TOMS 16, 1990, with the table holding the logarithm of its own rounded
// reciprocals): u = 2^e f with f in [sqrt(1/2), sqrt(2)) by the high word,
// F_j = 1 + j/128 the nearest centre (128 f - 128 rounded to an integer by
// one fma with 1.5 2^52), r = f RN(1/F_j) - 1 by one fma (|r| <= 0.0055), and
// ln u = e ln 2 + L_j + log1p(r) with L_j = -ln RN(1/F_j) from lg_log_table.h
// and log1p by its Taylor series to r^7 (truncation below 2e-17 relative).
// The centre F_0 = 1 makes r = f - 1 exact next to u = 1, where ln u is tiny;
// ln 2 is split so that e ln2_hi is exact.  u = 1 gives exactly +0.
__device__ __forceinline__ double log_unit_interval(double n) {
    const int hx = __double2hiint(n) + (0x3ff00000 - 0x3fe6a09e);
    const int e = (hx >> 20) - (0x3ff + 53);
    const double f = __hiloint2double((hx & 0x000fffff) + 0x3fe6a09e, __double2loint(n));
    const int j = __double2loint(fma(f, 128.0, 0x1.8p52 - 128.0));
    const double2 E = __ldg(&kLogTable[j - kLogTableMin]);
    const double r = fma(f, E.x, -1.0);
    double q = 1.0 / 7.0;
    q = fma(q, r, -1.0 / 6.0);
    q = fma(q, r, 1.0 / 5.0);
    q = fma(q, r, -0.25);
    q = fma(q, r, 1.0 / 3.0);
    q = fma(q, r, -0.5);
    const double p = fma(r * r, q, r);
    const double ln2_hi = 0x1.62e42fefa3800p-1, ln2_lo = 0x1.ef35793c76730p-45;
    return fma((double)e, ln2_hi, E.y) + fma((double)e, ln2_lo, p);
}

// cos x for the Box-Muller angle, x = fl(2 pi v) in (0, 2 pi] and `top` the
// first three bits of v, within 2.3e-16 relative, also next to the zeros of
// cos: x = k pi/2 + r, |r| <= pi/4, with pi/2 in two parts (the first
// subtraction is exact), then the sine r + r z S(z) or the cosine 1 + z C(z),
// z = r^2, and the quadrant's sign.  S and C minimise the relative error on
// that interval (Remez exchange; 3.6e-18 and 5.6e-20).  A warp's lanes draw all
// quadrants, so the coefficients are selected (two polynomials and a select of
// the results run 10080^2 1.6 % and blocks of 196 x 146 3 % slower, by spills).
// One polynomial over |r| <= pi/2 takes fewer instructions (10080^2 4 % faster
// with a root within an ulp), but its rounding errors are larger: the
// Gaussian's mean error 8.0e-17 against 7.5e-17.
__device__ __forceinline__ double cos_full_turn(double x, int top) {
    const int k = (top + 1) >> 1;
    const double kd = __hiloint2double(0x43300000, k) - 0x1p52;
    const double r = fma(-kd, 0x1.1a62633145c07p-54, fma(-kd, 0x1.921fb54442d18p+0, x));
    const double z = r * r;
    const bool odd = k & 1;
    double q = odd ? 0.0 : -0x1.8fa4800fb4bcbp-37;
    q = fma(q, z, odd ? 0x1.5d8fba92fea51p-33 : 0x1.1ee9d783e31abp-29);
    q = fma(q, z, odd ? -0x1.ae5e5a4426ab5p-26 : -0x1.27e4f7ea7e667p-22);
    q = fma(q, z, odd ? 0x1.71de3567738e7p-19 : 0x1.a01a019c83f08p-16);
    q = fma(q, z, odd ? -0x1.a01a019bfd844p-13 : -0x1.6c16c16c14f8ep-10);
    q = fma(q, z, odd ? 0x1.111111110f7cdp-7 : 0x1.555555555554bp-5);
    q = fma(q, z, odd ? -0x1.5555555555548p-3 : -0.5);
    const double v = fma(odd ? r * z : z, q, odd ? r : 1.0);
    return __hiloint2double(__double2hiint(v) ^ (((k + 1) & 2) << 30), __double2loint(v));
}

// sqrt w for w = 0 or 2^-60 < w < 2^60, correctly rounded: g = w y and h = y /
// 2 with y the hardware's approximation of 1 / sqrt(w) (better than 2^-19),
// the cubic Householder step (1 + e/2 + 3 e^2 / 8), e = 1 - g y, on both, and
// one correction with the exact residual, g + (w - g^2) h (Markstein, IBM J.
// Res. Dev. 34, 1990).  A zero of either sign gives itself (the
// approximation's infinity is made finite).
__device__ __forceinline__ double sqrt_radius(double w) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(w));
    const int hy = min(__double2hiint(y) & 0x7fffffff, 0x7fe00000);
    y = __hiloint2double(hy, 0);
    double g = w * y, h = __hiloint2double(hy - 0x00100000, 0);
    const double e = fma(-g, y, 1.0);
    const double s = e * fma(e, 0.375, 0.5);
    g = fma(g, s, g);
    h = fma(h, s, h);
    return fma(fma(-g, g, w), h, g);
}

// Box-Muller cosine branch from one key (src/util/rng.rs:43-49): the
// integer stream and the uniforms are exact (n 2^-53 with n = (bits >> 11) +
// 1); the transcendental factors are within a few ulp of exact, the Gaussian
// within 1e-12 relative of the reference's as required.
__device__ __forceinline__ double standard_normal(uint64_t key) {
    const uint64_t a = splitmix64(key);
    const uint64_t b = splitmix64(a ^ 0xD1B54A32D192ED03ull);
    const double nu = (double)((a >> 11) + 1), nv = (double)((b >> 11) + 1);
    // fl(2 pi v): the power of two scales exactly
    const double x = nv * (kTau * (1.0 / 9007199254740992.0));
    return sqrt_radius(-2.0 * log_unit_interval(nu)) * cos_full_turn(x, (int)(b >> 61));
}

// Single-precision Gaussian from the same two uniforms, for the FP32 path.
__device__ __forceinline__ float standard_normal_f32(uint64_t key) {
    uint64_t a = splitmix64(key);
    uint64_t b = splitmix64(a ^ 0xD1B54A32D192ED03ull);
    float u = (float)unit_open(a);
    float v = (float)unit_open(b);
    return sqrtf(-2.0f * logf(u)) * cospif(2.0f * v);
}

// Wiener stream tag of driver index j: (1 << 32) | j (driver.rs:134-140).
constexpr uint64_t kWienerStream0 = (1ull << 32) | 0ull;

// Streaming multiprocessors of the current device, queried once per device
// ordinal; the grid-sizing heuristics scale with it.
inline int device_sm_count() {
    static int cache[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
    int v = dev < 64 ? cache[dev] : 0;
    if (v > 0) return v;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 1;
    if (dev < 64) cache[dev] = v;
    return v;
}

}  // namespace lg
