// Halo fill, heat and Model C step kernels of the legendre B200 library.
//
// This translation unit is compiled with -fmad=false: the reference is Rust,
// which never contracts a*b+c into a fused multiply-add, so every product
// and sum below rounds separately and `fma` appears exactly where the
// reference calls `f64::mul_add`.  That is what makes the FP64 path
// bit-identical to the reference's SerialScheduler.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "lg_common.cuh"
#include "lg_kernels.h"
#include "lg_modelc_ops.cuh"

namespace lg {
namespace {

// Offset of interior-relative index l inside a ghost-inclusive slab
// (cartesian.rs:189-204).
template <int D>
__device__ __forceinline__ int64_t lin(const SlabLayout& L, const int* l) {
    int64_t o = l[0] + L.ghost;
    if (D > 1) o += (int64_t)(l[1] + L.ghost) * L.gdim[0];
    if (D > 2) o += (int64_t)(l[2] + L.ghost) * L.gdim[0] * L.gdim[1];
    return o;
}

// Write the value of interior cell `l` of block `b` into every ghost entry
// whose source it is.  The reference fills ghosts by a dimension sweep
// (cartesian.rs:439-526); its result is separable per dimension -- ghost
// (x, y, ...) holds the interior value at (map_0(x), map_1(y), ...), each
// map being the identity inside the block, the face neighbour's interior
// (wrapped in periodic dimensions) or the mirror image at a physical
// boundary.  Pushing along the pre-images of that map writes every ghost
// entry exactly once, with no ordering between blocks.
template <int D, class T>
__device__ __forceinline__ void push_ghost_images(T* __restrict__ arena, const CartTopo& topo,
                                                  const SlabLayout& L, int field, int b, const int* l, T val) {
    const int g = L.ghost;
    int step[D][3], cl[D][3], nc[D];
    bool any = false;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const int n = topo.n[d];
        nc[d] = 1;
        step[d][0] = 0;
        cl[d][0] = l[d];
        if (l[d] < g) {
            int nb = topo.nbr[(b * 3 + d) * 2 + 0];
            step[d][nc[d]] = nb >= 0 ? -1 : 0;
            cl[d][nc[d]] = nb >= 0 ? n + l[d] : -1 - l[d];
            ++nc[d];
            any = true;
        }
        if (l[d] >= n - g) {
            int nb = topo.nbr[(b * 3 + d) * 2 + 1];
            step[d][nc[d]] = nb >= 0 ? 1 : 0;
            cl[d][nc[d]] = nb >= 0 ? l[d] - n : 2 * n - 1 - l[d];
            ++nc[d];
            any = true;
        }
    }
    if (!any) return;
    int c[3] = {0, 0, 0};
    for (;;) {
        // advance the mixed-radix counter; the all-zero combination is the
        // cell itself and is skipped
        int d = 0;
        while (d < D) {
            if (++c[d] < nc[d]) break;
            c[d] = 0;
            ++d;
        }
        if (d == D) break;
        int blk = b;
        int tl[3] = {0, 0, 0};
#pragma unroll
        for (int e = 0; e < D; ++e) {
            int st = step[e][c[e]];
            if (st != 0) blk = topo.nbr[(blk * 3 + e) * 2 + (st > 0 ? 1 : 0)];
            tl[e] = cl[e][c[e]];
        }
        arena[slab_base(L, blk, field) + lin<D>(L, tl)] = val;
    }
}

// ------------------------------------------------------------- halo (b) --
// One CTA per block (several for large blocks), every ghost entry a copy of
// its source.  The
// reference's dimension sweep (cartesian.rs:439-526) is separable: ghost (x,
// y, ...) holds the interior value at (map_0(x), map_1(y), ...), each map the
// identity inside the block, the face neighbour's interior, or the mirror
// image.  The 3^D blocks those maps can lead to are looked up once per CTA.
// Ghost rows (a y or z outside the block) are copied whole, the x ghosts of
// the other rows one entry a thread.
//
// Bound: DRAM and L2 sectors (an x ghost costs a sector read and one written
// for its 8 bytes) and the latency of a copy, so each thread has four in
// flight: the fill of 32,768 blocks of 16^3 takes 470 us, one entry at a time
// 660.  All index arithmetic is 32 bit, two divisions an entry; with 64-bit
// divisions in every dimension it took 1650 us, three and a half heat steps.
// `dependent`: resident, its tables read, when the kernel before it drains (a
// run of one plain heat step and the fill, 64^3, 12.9 -> 10.8 us; after a graph
// it costs 2 us, and is not asked for).
// Index: 64 bit for blocks of more than 2^28 ghost entries, whose numbers and
// the strides beyond them could pass 32.
template <int D, class T, class Index>
__global__ void __launch_bounds__(256) halo_fill_kernel(T* __restrict__ arena, CartTopo topo, SlabLayout L,
                                                        int field) {
    constexpr int NS = D == 1 ? 3 : (D == 2 ? 9 : 27);
    __shared__ int64_t src_base[NS];  // slab of the block at (sx, sy, sz), sx fastest, each 0..2
    __shared__ int mirror[3][2];
    const int g = L.ghost;
    const int n0 = topo.n[0], n1 = D > 1 ? topo.n[1] : 1, n2 = D > 2 ? topo.n[2] : 1;
    const int G0 = L.gdim[0], G1 = D > 1 ? L.gdim[1] : 1;
    const int gy = D > 1 ? g : 0, gz = D > 2 ? g : 0;
    const Index first = blockIdx.y * blockDim.x + threadIdx.x, stride = gridDim.y * blockDim.x;
    for (int b = blockIdx.x; b < topo.nblocks; b += gridDim.x) {
        __syncthreads();  // the tables of the previous block are no longer read
        if (threadIdx.x < NS) {
            int src = b, code = threadIdx.x;
            for (int e = 0; e < D; ++e) {
                const int step = code % 3;
                code /= 3;
                if (step == 1) continue;
                const int nb = topo.nbr[(src * 3 + e) * 2 + (step >> 1)];
                if (nb >= 0) src = nb;
            }
            src_base[threadIdx.x] = slab_base(L, src, field);
        } else if (threadIdx.x >= 32 && threadIdx.x < 32 + 2 * D) {
            const int k = threadIdx.x - 32;
            mirror[k >> 1][k & 1] = topo.nbr[(b * 3 + (k >> 1)) * 2 + (k & 1)] < 0 ? 1 : 0;
        }
        __syncthreads();
        // the tables come from the topology alone: only now wait for the
        // predecessor, whose writes the copies read
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        T* const slab = arena + slab_base(L, b, field);
        // source index and step (0 low, 1 inside, 2 high) of index i, -g <= i < n + g
        auto map = [&](int e, int i, int n, int& step) {
            step = i < 0 ? 0 : (i >= n ? 2 : 1);
            if (step == 1) return i;
            if (mirror[e][step >> 1]) return step == 0 ? -1 - i : 2 * n - 1 - i;
            return step == 0 ? n + i : i - n;
        };
        // element offsets of ghost entry (x, y, z) in its slab and of its
        // source in the arena
        auto place = [&](int x, int y, int z, int64_t& to, int64_t& from) {
            int sx, sy = 1, sz = 1;
            const int mx = map(0, x, n0, sx);
            const int my = D > 1 ? map(1, y, n1, sy) : 0;
            const int mz = D > 2 ? map(2, z, n2, sz) : 0;
            const int code = sx + (D > 1 ? 3 * sy : 0) + (D > 2 ? 9 * sz : 0);
            to = (x + g) + (int64_t)G0 * ((y + gy) + (int64_t)G1 * (z + gz));
            from = src_base[code] + (mx + g) + (int64_t)G0 * ((my + gy) + (int64_t)G1 * (mz + gz));
        };
        // the entries in one sequence: x ghosts of the interior rows (2 g a
        // row), rows with y outside and z inside, planes with z outside
        const Index per = 2u * g, xs = (Index)n1 * n2 * per;
        const Index strip = D > 1 ? (Index)2 * g * G0 : 1, ys = D > 1 ? xs + strip * n2 : xs;
        const Index plane = D > 2 ? (Index)G0 * G1 : 1, all = D > 2 ? ys + plane * 2u * g : ys;
        auto entry = [&](Index k, int64_t& to, int64_t& from) {
            if (k < xs) {
                const Index row = k / per, i = k - row * per;
                const Index z = row / n1, y = row - z * n1;
                place((int)i < g ? (int)i - g : n0 + (int)i - g, (int)y, (int)z, to, from);
            } else if (D > 1 && k < ys) {
                k -= xs;
                const Index z = k / strip, q = k - z * strip;
                const Index r = q / G0, x = q - r * G0;
                place((int)x - g, (int)r < g ? (int)r - g : n1 + (int)r - g, (int)z, to, from);
            } else if (D > 2) {
                k -= ys;
                const Index p = k / plane, q = k - p * plane;
                const Index r = q / G0, x = q - r * G0;
                place((int)x - g, (int)r - g, (int)p < g ? (int)p - g : n2 + (int)p - g, to, from);
            }
        };
        constexpr int U = 4;  // entries in flight a thread
        for (Index k = first; k < all; k += U * stride) {
            int64_t to[U];
            T v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const Index e = k + u * stride;
                if (e < all) {
                    int64_t from = 0;
                    entry(e, to[u], from);
                    v[u] = arena[from];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + u * stride < all) slab[to[u]] = v[u];
        }
    }
}

// ------------------------------------ heat, one thread per cell (d) --
// Heat<D>::vector_field_block (examples/heat3d.rs:63-79): the central
// Laplacian (finite_difference.rs:49-67) times kappa, then ForwardEuler's
// axpy (integrators/euler.rs:51-53).  1-D, and single steps of small 2-D grids,
// which need no fill afterwards.
template <int D>
__device__ __forceinline__ double heat_drift(const double* s, int64_t o, int64_t st1, double kappa, double ih0,
                                             double ih1) {
    const double center = s[o];
    double acc = 0.0;
    acc += ((s[o + 1] - (center + center)) + s[o - 1]) * ih0;
    if (D > 1) acc += ((s[o + st1] - (center + center)) + s[o - st1]) * ih1;
    return acc * kappa;
}

template <int D>
__global__ void __launch_bounds__(256) heat_step_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                        CartTopo topo, SlabLayout L, int field, double kappa,
                                                        double dt, double ih0, double ih1) {
    const int64_t cells = (int64_t)topo.n[0] * (D > 1 ? topo.n[1] : 1);
    for (int b = blockIdx.y; b < topo.nblocks; b += gridDim.y) {
        const int64_t base = slab_base(L, b, field);
        const double* s = in + base;
        for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cells;
             c += (int64_t)gridDim.x * blockDim.x) {
            int l[2] = {(int)c, 0};
            if (D > 1) {
                l[1] = (int)(c / topo.n[0]);
                l[0] = (int)(c - (int64_t)l[1] * topo.n[0]);
            }
            const int64_t o = lin<D>(L, l);
            const double v = s[o] + dt * heat_drift<D>(s, o, L.gdim[0], kappa, ih0, ih1);
            out[base + o] = v;
            push_ghost_images<D, double>(out, topo, L, field, b, l, v);
        }
    }
}

// One stage of RungeKutta4 (rk4.rs:40-79) for the heat model, one thread
// per interior cell: k = kappa lap(in) as heat_step_kernel computes it, then
//   MODE 1: kout = k, out = y + c k          (y_tmp = y; y_tmp += c k_i)
//   MODE 2: out = (((y + s6 k1) + s3 k2) + s3 k3) + s6 k   (the four axpys)
// with the output's ghost images pushed for the next stage.
template <int MODE>
__global__ void __launch_bounds__(256) heat_rk_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                      const double* __restrict__ y, double* __restrict__ kout,
                                                      const double* __restrict__ k1, const double* __restrict__ k2,
                                                      const double* __restrict__ k3, CartTopo topo, SlabLayout L,
                                                      int field, double kappa, double ih, double c, double s6,
                                                      double s3) {
    for (int b = blockIdx.y; b < topo.nblocks; b += gridDim.y) {
        const int64_t base = slab_base(L, b, field);
        for (int64_t cc = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cc < topo.n[0];
             cc += (int64_t)gridDim.x * blockDim.x) {
            const int l[1] = {(int)cc};
            const int64_t o = lin<1>(L, l), e = base + o;
            const double k = heat_drift<1>(in + base, o, 0, kappa, ih, 0.0);
            double v;
            if (MODE == 1) {
                kout[e] = k;
                v = y[e] + c * k;
            } else {
                v = y[e];
                v = v + s6 * k1[e];
                v = v + s3 * k2[e];
                v = v + s3 * k3[e];
                v = v + s6 * k;
            }
            out[e] = v;
            push_ghost_images<1, double>(out, topo, L, field, b, l, v);
        }
    }
}

// Reference-order Model C step, one thread per interior cell: the flux
// kernel (finite_volume.rs:258-283), the local terms (phasefield.rs:395-404),
// the u Laplacian and coupling (phasefield.rs:412-421), the Time driver
// axpy (driver.rs:210-216) and the Wiener increment (driver.rs:218-236).
template <class T>
__global__ void __launch_bounds__(256) modelc_step_ref_kernel(const T* __restrict__ in, T* __restrict__ out,
                                                              CartTopo topo, SlabLayout L, MC<T> m, T dt,
                                                              double dt64, NoiseDev nz, T scale_amp, double* tdev,
                                                              int slot) {
    const int n0 = topo.n[0], n1 = topo.n[1];
    const int64_t sy = L.gdim[0];
    // Simulation::t lives on the device in two slots: this step reads
    // tdev[slot] (its bits are the Wiener salt, euler_maruyama.rs:73) and
    // writes t + dt to the other slot (simulation.rs:285), so a captured
    // sequence of steps needs no host-side time.
    const double t = tdev[slot];
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) tdev[slot ^ 1] = t + dt64;
    for (int b = blockIdx.y; b < topo.nblocks; b += gridDim.y) {
    const T* ph = in + slab_base(L, b, 0);
    const T* uu = in + slab_base(L, b, 1);
    T* phi_out = out + slab_base(L, b, 0);
    T* u_out = out + slab_base(L, b, 1);
    uint64_t block_key = 0;
    if (nz.on) block_key = wiener_block_key(nz.seed, (uint64_t)__double_as_longlong(t), kWienerStream0, (uint64_t)b);
    const T quarter = T(0.25), half = T(0.5);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n0 * n1; c += gridDim.x * blockDim.x) {
        const int i = c % n0, j = c / n0;
        const int64_t o = (int64_t)(i + 1) + (int64_t)(j + 1) * sy;
        auto P = [&](int di, int dj) { return ph[o + di + dj * sy]; };
        T derx_r = P(1, 0) - P(0, 0);
        T derx_l = P(0, 0) - P(-1, 0);
        T derx_t = quarter * (P(1, 1) - P(-1, 1) + P(1, 0) - P(-1, 0));
        T derx_b = quarter * (P(1, 0) - P(-1, 0) + P(1, -1) - P(-1, -1));
        T dery_t = P(0, 1) - P(0, 0);
        T dery_b = P(0, 0) - P(0, -1);
        T dery_r = quarter * (P(1, 1) - P(1, -1) + P(0, 1) - P(0, -1));
        T dery_l = quarter * (P(0, 1) - P(0, -1) + P(-1, 1) - P(-1, -1));
        T a_r, da_r, a_l, da_l, a_t, da_t, a_b, da_b;
        kr_face(m, derx_r, dery_r, a_r, da_r);
        kr_face(m, derx_l, dery_l, a_l, da_l);
        kr_face(m, derx_t, dery_t, a_t, da_t);
        kr_face(m, derx_b, dery_b, a_b, da_b);
        T j_r = a_r * (a_r * derx_r - da_r * dery_r);
        T j_l = a_l * (a_l * derx_l - da_l * dery_l);
        T j_t = a_t * (a_t * dery_t + da_t * derx_t);
        T j_b = a_b * (a_b * dery_b + da_b * derx_b);
        T flux = (j_r - j_l + j_t - j_b) * m.inv_h2_flux;

        T p = P(0, 0);
        T g_prime = fma_t(p * p, p, -p);
        T one_m_p2 = fma_t(p, -p, T(1));
        T p_prime = one_m_p2 * one_m_p2;
        // center_anisotropy (phasefield.rs:159-175)
        T cdx = half * (P(1, 0) - P(-1, 0));
        T cdy = half * (P(0, 1) - P(0, -1));
        T cdx2 = cdx * cdx;
        T cdy2 = cdy * cdy;
        T csum = cdx2 + cdy2;
        T cmag2 = csum * csum;
        T a = cmag2 <= m.tol ? m.a_bar : m.a_bar * (T(1) + m.eps_prime * (cdx2 * cdx2 + cdy2 * cdy2) / cmag2);
        T uc = uu[o];
        T kphi = fma_t(m.lambda * uc, -p_prime, flux - g_prime) / (a * a);

        T acc = T(0);
        acc += ((uu[o + 1] - (uc + uc)) + uu[o - 1]) * m.ih0;
        acc += ((uu[o + sy] - (uc + uc)) + uu[o - sy]) * m.ih1;
        T ku = fma_t(acc, m.d_thermal, half * kphi);

        T phin = p + dt * kphi;
        if (nz.on) {
            uint64_t key = splitmix64(block_key ^ (uint64_t)(i + j * n0));
            phin += scale_amp * normal_t(key, T(0));
        }
        T un = uc + dt * ku;
        phi_out[o] = phin;
        u_out[o] = un;
        int l[2] = {i, j};
        push_ghost_images<2, T>(out, topo, L, 0, b, l, phin);
        push_ghost_images<2, T>(out, topo, L, 1, b, l, un);
    }
    }
}

__global__ void standard_normal_kernel(const uint64_t* keys, double* out, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = standard_normal(keys[i]);
}

int grid_x_for(int64_t cells, int threads) {
    int64_t gx = (cells + threads - 1) / threads;
    return (int)(gx < 1 ? 1 : (gx > 65535 ? 65535 : gx));
}

int grid_y_for(int nblocks) { return nblocks < 1 ? 1 : (nblocks > 65535 ? 65535 : nblocks); }

}  // namespace

cudaError_t launch_halo_fill(void* arena, int elem_size, const CartTopo& topo, const SlabLayout& L, int field,
                             cudaStream_t s, bool dependent) {
    if (L.ghost == 0) return cudaSuccess;
    // entries of one block; a CTA for every 2048 of them
    int64_t inner = 1, whole = 1;
    for (int d = 0; d < topo.D; ++d) {
        inner *= topo.n[d];
        whole *= topo.n[d] + 2 * L.ghost;
    }
    const dim3 grid((unsigned)topo.nblocks,
                    (unsigned)std::max<int64_t>(1, std::min<int64_t>((whole - inner) / 2048, 1024)));
    const bool large = whole - inner > (int64_t)1 << 28;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
#define LG_HALO_T(DD, T)                                                                                         \
    (large ? cudaLaunchKernelEx(&cfg, halo_fill_kernel<DD, T, uint64_t>, static_cast<T*>(arena), topo, L, field) \
           : cudaLaunchKernelEx(&cfg, halo_fill_kernel<DD, T, unsigned>, static_cast<T*>(arena), topo, L, field))
#define LG_HALO(DD) (elem_size == 8 ? LG_HALO_T(DD, double) : LG_HALO_T(DD, float))
    return topo.D == 1 ? LG_HALO(1) : topo.D == 2 ? LG_HALO(2) : LG_HALO(3);
#undef LG_HALO
#undef LG_HALO_T
}

cudaError_t launch_heat_rk_stage(int mode, const double* in, double* out, const double* y, double* kout,
                                 const double* k1, const double* k2, const double* k3, const CartTopo& topo,
                                 const SlabLayout& L, int field, double kappa, const double* inv_h2, double c,
                                 double s6, double s3, cudaStream_t s) {
    if (topo.D != 1) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)std::min<int64_t>(((int64_t)topo.n[0] + 255) / 256, 1024),
                    (unsigned)std::min(topo.nblocks, 65535));
    if (mode == 1)
        heat_rk_kernel<1><<<grid, 256, 0, s>>>(in, out, y, kout, k1, k2, k3, topo, L, field, kappa, inv_h2[0], c, s6, s3);
    else
        heat_rk_kernel<2><<<grid, 256, 0, s>>>(in, out, y, kout, k1, k2, k3, topo, L, field, kappa, inv_h2[0], c, s6, s3);
    return cudaGetLastError();
}

cudaError_t launch_heat_step(const double* in, double* out, const CartTopo& topo, const SlabLayout& L, int field,
                             double kappa, double dt, const double inv_h2[3], cudaStream_t s) {
    if (topo.D > 2) return cudaErrorInvalidValue;
    dim3 grid(grid_x_for((int64_t)topo.n[0] * (topo.D > 1 ? topo.n[1] : 1), 256), grid_y_for(topo.nblocks));
    if (topo.D == 1)
        heat_step_kernel<1><<<grid, 256, 0, s>>>(in, out, topo, L, field, kappa, dt, inv_h2[0], 0.0);
    else
        heat_step_kernel<2><<<grid, 256, 0, s>>>(in, out, topo, L, field, kappa, dt, inv_h2[0], inv_h2[1]);
    return cudaGetLastError();
}

cudaError_t launch_modelc_step_f64(const double* in, double* out, const CartTopo& topo, const SlabLayout& L,
                                   const ModelCDev& m, double dt, const NoiseDev& nz, double* tdev, int slot,
                                   int variant, cudaStream_t s) {
    (void)variant;
    dim3 grid(grid_x_for((int64_t)topo.n[0] * topo.n[1], 256), grid_y_for(topo.nblocks));
    double scale_amp = std::sqrt(dt) * nz.amp;
    modelc_step_ref_kernel<double><<<grid, 256, 0, s>>>(in, out, topo, L, to_mc<double>(m), dt, dt, nz, scale_amp,
                                                        tdev, slot);
    return cudaGetLastError();
}

cudaError_t launch_modelc_step_f32(const float* in, float* out, const CartTopo& topo, const SlabLayout& L,
                                   const ModelCDev& m, double dt, const NoiseDev& nz, double* tdev, int slot,
                                   int variant, cudaStream_t s) {
    (void)variant;
    dim3 grid(grid_x_for((int64_t)topo.n[0] * topo.n[1], 256), grid_y_for(topo.nblocks));
    float scale_amp = (float)std::sqrt(dt) * (float)nz.amp;
    modelc_step_ref_kernel<float><<<grid, 256, 0, s>>>(in, out, topo, L, to_mc<float>(m), (float)dt, dt, nz,
                                                       scale_amp, tdev, slot);
    return cudaGetLastError();
}

cudaError_t launch_standard_normal(const uint64_t* keys, double* out, int64_t n, cudaStream_t s) {
    standard_normal_kernel<<<grid_x_for(n, 256), 256, 0, s>>>(keys, out, n);
    return cudaGetLastError();
}

}  // namespace lg
