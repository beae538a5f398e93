// Heat steps in 2-D and 3-D, two stages of a step sequence per launch.
//
// Compiled with -fmad=false: every product and sum rounds separately, in the
// reference's operand order (finite_difference.rs:49-67, euler.rs:51-53,
// rk4.rs:40-79), so the results are the reference's bits.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "lg_common.cuh"
#include "lg_heat_plan.h"
#include "lg_kernels.h"

namespace lg {
namespace {

// The four forms of the marching kernel.  kFe1: one forward-Euler step.
// kFe2: two of them, the state between them never leaving the SM.  kRkA:
// stages 1 and 2 of RungeKutta4 (in = y; out = y + c k2, aux = (y + s6 k1) +
// s3 k2).  kRkB: stages 3 and 4 (in = y + c k2 of kRkA, y, aux; out = ((aux +
// s3 k3) + s6 k4).  The running sum aux is rk4.rs's chain of axpys in its
// order, so no k is ever stored.
enum HeatForm { kFe1, kFe2, kRkA, kRkB };

struct HeatArgs {
    const double* in;   // the field's slab of block 0, in each arena
    double* out;
    const double* y;    // kRkB
    const double* aux_in;
    double* aux;        // kRkA
    int64_t N[3];       // global cells: x, y (1 in 2-D), march dimension
    int n[3];           // block cells in the same order
    int periodic[3];
    int64_t bstr[3];    // elements between neighbouring blocks of a dimension
    int64_t cstr[3];    // elements between neighbouring cells of a dimension inside a slab
    double ih[3];
    // The reference sums a cell's terms from zero, so that its sum is never -0;
    // here a sum of terms that all underflowed may be, and kappa sum + `zero` in
    // one fma has the reference's zero then (for kappa > 0; a sum from zero ran
    // 96^3 272 us instead of 244, the product alone 242).  Otherwise it is the
    // product: `zero` is -0 for other kappa.
    double kappa, zero, c1, c2, s6, s3;
    int tiles_x, tiles_y, zc;
};

// source coordinate of a window position: itself, wrapped, or the mirror
// image (cartesian.rs:439-526); positions that no result depends on are
// clamped into the domain
template <class Coord>
__device__ __forceinline__ Coord source_coord(Coord g, Coord N, int periodic) {
    if (periodic) {
        while (g < 0) g += N;
        while (g >= N) g -= N;
        return g;
    }
    if (g < 0) g = -1 - g;
    if (g >= N) g = N - 1 - (g - N);
    return min(max(g, (Coord)0), N - 1);
}

// element offset of global coordinate g of dimension d inside an arena
template <class Coord>
__device__ __forceinline__ int64_t coord_offset(const HeatArgs& a, int d, Coord g) {
    const Coord b = g / a.n[d];
    return (int64_t)b * a.bstr[d] + (int64_t)(g - b * a.n[d] + 1) * a.cstr[d];
}

// Tile geometry.  WX: window columns; TR: thread rows; R: window rows of a
// thread (TR = R = 1 in 2-D); PITCH: doubles between staged rows, such that
// lanes that wrap to the next thread row hit the following banks (R PITCH =
// WX mod 16).  A window is H cells wider than its tile on each side.
template <int FORM, int WX, int TR, int R, int PITCH>
struct MarchTile {
    static constexpr bool kHasY = TR * R > 1;
    static constexpr int kH = FORM == kFe1 ? 1 : 2;
    static constexpr int kWY = TR * R;
    static constexpr int kOX = WX - 2 * kH, kOY = kHasY ? kWY - 2 * kH : 1;
    static constexpr int kThreads = (WX * TR + 31) / 32 * 32;
    static constexpr int kGuard = PITCH + 1;  // the window's rim reads (and ignores) one row and one cell beyond it
    static constexpr int kPlane = kWY * PITCH + 2 * kGuard;
    static constexpr int kAhead = kHasY ? 1 : 3;  // planes in flight besides the newest
};

// One CTA owns a tile of columns of the global grid -- whatever blocks they
// lie in -- and marches along the last dimension over `zc` planes.  A thread
// owns R window rows of one column; the planes it has passed stay in its
// registers (the march neighbours), the newest plane and the first stage's
// result are staged in shared memory, double buffered, for the in-plane
// neighbours: one barrier per plane.  Iteration p starts the load of plane p
// + kAhead, applies the first stage to plane p - 1 and the second to plane p
// - 2.  The window is two cells wider than the tile on each side (one for
// kFe1): the first stage runs on a one-cell halo too, where it computes what
// the neighbour tile computes, from the same operands in the same order.  At
// a mirror boundary the first stage's ghost is the edge cell's own value.
//
// Bound (3-D, kFe2): the shared-memory pipe, 69 % busy at 416^3 with FP64 at
// 42 %, issue at 54 % and the DRAM at 42 %: each stage reads two x
// neighbours a cell from shared memory and a rows' global accesses straddle
// the 16-cell blocks.  More rows a thread means fewer y neighbours to read:
// at 512^3 394 us a step with R = 4, 420 with R = 3, 447 with R = 2.  Copying
// planes to shared memory asynchronously (four planes ahead, three CTAs per
// SM) ran at 411: the loads' latency is not the limit.
//
// No ghost entry is read.  The two ghost columns of each stored row are
// written with the row and refilled by the caller: without them the rows'
// ends are partly written sectors, which the DRAM reads back (512^3: 466
// instead of 394 us a step).
//
// The march is unrolled six times, so that the planes in registers, those of
// the first stage (three) and the double buffers keep their places and
// nothing is moved (rolled: 90 instead of 53 instructions per cell and
// step).  Off: the type of a column's byte offset inside one layer of blocks and,
// signed, of a cell's coordinate.
template <int FORM, int WX, int TR, int R, int PITCH, int MINB, class Off>
__global__ void __launch_bounds__(MarchTile<FORM, WX, TR, R, PITCH>::kThreads, MINB)
    heat_march_kernel(const __grid_constant__ HeatArgs a) {
    using G = MarchTile<FORM, WX, TR, R, PITCH>;
    using Coord = std::make_signed_t<Off>;
    constexpr bool HASY = G::kHasY;
    constexpr int H = G::kH, WY = G::kWY, PF = G::kAhead, UR = 6;
    __shared__ double A[2][G::kPlane];
    __shared__ double B[FORM == kFe1 ? 1 : 2][FORM == kFe1 ? 1 : G::kPlane];
    __shared__ int64_t plane_off[kMaxPlanes + 2 * H + PF + 1];  // bytes, of planes z0 - H ...

    const int t = threadIdx.x;
    const int cx = t % WX, ty = t / WX;
    const bool thread_in = ty < TR;
    const int wy0 = min(ty, TR - 1) * R;  // idle threads shadow the last rows
    const Coord NX = (Coord)a.N[0], NY = (Coord)a.N[1], NZ = (Coord)a.N[2];
    int item = blockIdx.x;
    const Coord tx0 = (Coord)(item % a.tiles_x) * G::kOX;
    item /= a.tiles_x;
    const Coord ty0 = HASY ? (Coord)(item % a.tiles_y) * G::kOY : 0;
    const Coord z0 = (Coord)(HASY ? item / a.tiles_y : item) * a.zc;
    const Coord z1 = min(z0 + a.zc, NZ);

    const Coord gx = tx0 - H + cx;
    const int64_t ox = coord_offset(a, 0, source_coord(gx, NX, a.periodic[0]));
    Off base[R];  // bytes
    bool store[R];
    const bool x_out = thread_in && cx >= H && cx < WX - H && gx < NX;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int64_t e = ox;
        store[r] = x_out;
        if (HASY) {
            const int wy = wy0 + r;
            const Coord gy = ty0 - H + wy;
            e += coord_offset(a, 1, source_coord(gy, NY, a.periodic[1]));
            store[r] = x_out && wy >= H && wy < WY - H && gy < NY;
        }
        base[r] = (Off)(e * 8);
    }
    // which of this thread's neighbours are mirror ghosts (second stage only)
    const bool mxlo = !a.periodic[0] && gx == 0, mxhi = !a.periodic[0] && gx == NX - 1;
    Coord mrow_lo = -1, mrow_hi = -1;
    if (HASY && !a.periodic[1]) {
        mrow_lo = H - ty0 - wy0;               // the r whose row is the first one
        mrow_hi = NY - 1 + H - ty0 - wy0;  // the r whose row is the last one
    }
    // ghost columns beside a block's first and last column
    const int ix = gx >= 0 && gx < NX ? (int)(gx % a.n[0]) : 1;
    const bool glo = x_out && ix == 0, ghi = x_out && ix == a.n[0] - 1;
    // plane offsets; those past the last plane needed stay valid addresses
    const Coord pend = z1 + H;
    const int planes = (int)(z1 - z0);
    for (int k = t; k < planes + 2 * H + PF + 1; k += G::kThreads)
        plane_off[k] = coord_offset(a, 2, source_coord(z0 - H + k, NZ, a.periodic[2])) * 8;
    const bool edge =
        __syncthreads_or(mxlo || mxhi || (mrow_lo >= 0 && mrow_lo < R) || (mrow_hi >= 0 && mrow_hi < R)) != 0;
    auto at = [](const double* p, int64_t plane, Off o) {
        return reinterpret_cast<const double*>(reinterpret_cast<const char*>(p) + plane + o);
    };
    auto put = [](double* p, int64_t plane, Off o) {
        return reinterpret_cast<double*>(reinterpret_cast<char*>(p) + plane + o);
    };
    // programmatic dependent launch: wait until the predecessor is complete
    // and its writes visible, then let the next launch become resident (not
    // before the wait: its CTAs would hold slots while two launches still run)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // loads bypass L1: an element is read once per CTA
    double U[UR][R], V[3][R], S[2][R], Y[2][R], X[2][R];
    const int64_t* po = plane_off;
#pragma unroll
    for (int k = 0; k < UR; ++k)
#pragma unroll
        for (int r = 0; r < R; ++r) U[k][r] = k < PF ? __ldcg(at(a.in, po[k], base[r])) : 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
        V[0][r] = V[1][r] = V[2][r] = S[0][r] = S[1][r] = Y[0][r] = Y[1][r] = X[0][r] = X[1][r] = 0.0;
    const int sidx = G::kGuard + wy0 * PITCH + cx;
    auto store_cell = [&](double* arena, int64_t off, Off o, double w) {
        double* q = put(arena, off, o);
        *q = w;
        if (glo) q[-1] = w;
        if (ghi) q[1] = w;
    };

    auto lap = [&](double c, double xm, double xp, double ym, double yp, double zm, double zp) {
        const double c2 = c + c;
        double acc = ((xp - c2) + xm) * a.ih[0];
        if (HASY) acc += ((yp - c2) + ym) * a.ih[1];
        acc += ((zp - c2) + zm) * a.ih[2];
        return fma(acc, a.kappa, a.zero);  // see HeatArgs
    };

    Coord p = z0 - H;
    for (;;) {
#pragma unroll
        for (int ph = 0; ph < UR; ++ph, ++p, ++po) {
            if (p >= pend) return;
            // places of planes p (newest), p - 1, p - 2 and of the load p + PF
            const int u0 = ph, u1 = (ph + 5) % UR, u2 = (ph + 4) % UR, ul = (ph + PF) % UR;
            const int v1 = ph % 3, v2 = (ph + 2) % 3, v3 = (ph + 1) % 3;  // first stage: planes p - 1, p - 2, p - 3
            const int e = ph & 1, o = e ^ 1;
#pragma unroll
            for (int r = 0; r < R; ++r) U[ul][r] = __ldcg(at(a.in, po[PF], base[r]));
            if (FORM == kRkB) {  // y and the running sum of plane p, for the next iteration
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    Y[e][r] = __ldcg(at(a.y, po[0], base[r]));
                    if (store[r]) X[e][r] = __ldcg(at(a.aux_in, po[0], base[r]));
                }
            }
            {
                // first stage, plane p - 1 (its rows are in A[o])
                const double* s = A[o] + sidx;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double xm = s[r * PITCH - 1], xp = s[r * PITCH + 1];
                    double ym = 0.0, yp = 0.0;
                    if (HASY) {
                        ym = r > 0 ? U[u1][r - 1] : s[-PITCH];
                        yp = r + 1 < R ? U[u1][r + 1] : s[R * PITCH];
                    }
                    const double c = U[u1][r];
                    const double k = lap(c, xm, xp, ym, yp, U[u2][r], U[u0][r]);
                    if (FORM == kRkB) {
                        V[v1][r] = Y[o][r] + a.c1 * k;
                        S[e][r] = X[o][r] + a.s3 * k;
                    } else {
                        V[v1][r] = c + a.c1 * k;
                        if (FORM == kRkA) S[e][r] = c + a.s6 * k;
                    }
                }
            }
            if (FORM == kFe1) {
                if (p - 1 >= z0 && p - 1 < z1) {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (store[r]) store_cell(a.out, po[-1], base[r], V[v1][r]);
                }
            } else {
                // second stage, plane p - 2 (the first stage's rows are in B[e])
                const double* s = B[e] + sidx;
                const bool zlo = !a.periodic[2] && p == 2, zhi = !a.periodic[2] && p - 2 == NZ - 1;
                const bool in = p - 2 >= z0;
                const int64_t off = in ? po[-2] : 0;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double c = V[v2][r];
                    double xm = s[r * PITCH - 1], xp = s[r * PITCH + 1];
                    double ym = 0.0, yp = 0.0;
                    if (HASY) {
                        ym = r > 0 ? V[v2][r - 1] : s[-PITCH];
                        yp = r + 1 < R ? V[v2][r + 1] : s[R * PITCH];
                    }
                    double zm = V[v3][r], zp = V[v1][r];
                    if (edge) {
                        if (mxlo) xm = c;
                        if (mxhi) xp = c;
                        if (HASY && r == mrow_lo) ym = c;
                        if (HASY && r == mrow_hi) yp = c;
                    }
                    if (zlo) zm = c;
                    if (zhi) zp = c;
                    const double k = lap(c, xm, xp, ym, yp, zm, zp);
                    double w;
                    if (FORM == kFe2) w = c + a.c2 * k;
                    if (FORM == kRkA) w = U[u2][r] + a.c2 * k;
                    if (FORM == kRkB) w = S[o][r] + a.s6 * k;
                    if (store[r] && in) {
                        store_cell(a.out, off, base[r], w);
                        if (FORM == kRkA) store_cell(a.aux, off, base[r], S[o][r] + a.s3 * k);
                    }
                }
                if (thread_in) {
                    double* sb = B[o] + sidx;
#pragma unroll
                    for (int r = 0; r < R; ++r) sb[r * PITCH] = V[v1][r];
                }
            }
            if (thread_in) {
                double* sa = A[e] + sidx;
#pragma unroll
                for (int r = 0; r < R; ++r) sa[r * PITCH] = U[u0][r];
            }
            __syncthreads();
        }
    }
}

// CTAs of a form that an SM holds, asked for once
template <int FORM, int WX, int TR, int R, int PITCH, int MINB, class Off>
cudaError_t march_occupancy(int& per_sm) {
    static std::atomic<int> known{0};
    per_sm = known.load(std::memory_order_relaxed);
    if (per_sm > 0) return cudaSuccess;
    auto* kernel = heat_march_kernel<FORM, WX, TR, R, PITCH, MINB, Off>;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, kernel, MarchTile<FORM, WX, TR, R, PITCH>::kThreads, 0);
    if (e != cudaSuccess) return e;
    per_sm = std::max(per_sm, 1);
    known.store(per_sm, std::memory_order_relaxed);
    return cudaSuccess;
}

// one tile shape: what it would cost (`factor`: what march_cost misses of it),
// and the launch
template <int FORM, class Off, int WX, int TR, int R, int PITCH, int MINB>
struct March {
    using G = MarchTile<FORM, WX, TR, R, PITCH>;
    static void tiles(HeatArgs& a) {
        a.tiles_x = (int)((a.N[0] + G::kOX - 1) / G::kOX);
        a.tiles_y = (int)((a.N[1] + G::kOY - 1) / G::kOY);
    }
    static cudaError_t consider(int tile, double factor, HeatArgs a, HeatPlan& plan) {
        int per_sm = 0;
        const cudaError_t e = march_occupancy<FORM, WX, TR, R, PITCH, MINB, Off>(per_sm);
        if (e != cudaSuccess) return e;
        tiles(a);
        const int64_t n = (int64_t)a.tiles_x * a.tiles_y, sms = device_sm_count();
        const int zc = march_planes(n, a.N[2], G::kH, sms * per_sm);
        const double cost = factor * march_cost(n, a.N[2], zc, G::kH, sms, per_sm, G::kThreads, R);
        if (plan.tile < 0 || cost < plan.cost) plan = HeatPlan{tile, zc, cost};
        return cudaSuccess;
    }
    static cudaError_t launch(HeatArgs a, const HeatPlan& plan, cudaStream_t s) {
        tiles(a);
        a.zc = plan.planes;
        const int64_t ctas = (int64_t)a.tiles_x * a.tiles_y * ((a.N[2] + a.zc - 1) / a.zc);
        if (ctas > (int64_t)0x7fffffff) return cudaErrorInvalidConfiguration;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ctas);
        cfg.blockDim = dim3(G::kThreads);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, heat_march_kernel<FORM, WX, TR, R, PITCH, MINB, Off>, a);
    }
};

// The tile shapes (window columns, thread rows, rows a thread) and the rule
// between them, march_cost.  2-D: a row of 128.  3-D: 32 x 16 columns with two
// rows a thread; Euler steps also 28 x 28 with four, where tiles are many
// (RungeKutta4 keeps two more arrays a row in registers: 256^3 375 us a step
// against 313); 8 x 80, 8 x 8 and (Euler) 60 x 8 for grids narrow in x, in both
// or in y, of which the others would fill a part of a window: 8 x 512 x 512 23.9
// -> 9.9 us a step, 8 x 8 x 4096 7.3 -> 4.3, 512 x 8 x 512 13.5 -> 9.4.
template <int FORM, class Off>
cudaError_t launch_form(int D, const HeatArgs& a, HeatPlan& plan, cudaStream_t s) {
    constexpr bool kEuler = FORM == kFe1 || FORM == kFe2, kNarrow = sizeof(Off) == 4;
    using Row = March<FORM, Off, 128, 1, 1, 128, 4>;
    using Few = March<FORM, Off, 36, 10, 2, 42, 2>;
    using Wide = March<FORM, Off, 32, 8, 4, 32, 2>;
    using NarrowX = March<FORM, Off, 12, 21, 4, 15, 2>;
    using Narrow = March<FORM, Off, 12, 3, 4, 15, 8>;
    using NarrowY = March<FORM, Off, 64, 3, 4, 64, 3>;
    if (plan.tile < 0) {
        cudaError_t e = D == 2 ? Row::consider(0, 1.0, a, plan) : Few::consider(1, 1.0, a, plan);
        if constexpr (kEuler)
            if (e == cudaSuccess && D == 3) e = Wide::consider(2, 1.0, a, plan);
        if constexpr (kNarrow) {
            if (e == cudaSuccess && D == 3) e = NarrowX::consider(3, kEuler ? 1.0 : 1.25, a, plan);
            if (e == cudaSuccess && D == 3) e = Narrow::consider(4, 1.0, a, plan);
            if constexpr (kEuler)
                if (e == cudaSuccess && D == 3) e = NarrowY::consider(5, 1.15, a, plan);
        }
        if (e != cudaSuccess) return e;
    }
    if constexpr (kEuler)
        if (plan.tile == 2) return Wide::launch(a, plan, s);
    if constexpr (kNarrow) {
        if (plan.tile == 3) return NarrowX::launch(a, plan, s);
        if (plan.tile == 4) return Narrow::launch(a, plan, s);
        if constexpr (kEuler)
            if (plan.tile == 5) return NarrowY::launch(a, plan, s);
    }
    return plan.tile == 0 ? Row::launch(a, plan, s) : Few::launch(a, plan, s);
}

template <int FORM>
cudaError_t launch_form(int D, const HeatArgs& a, HeatPlan& plan, cudaStream_t s) {
    // a column's byte offset inside one layer of blocks, and coordinates two
    // cells beyond the grid: 32 bits where they hold them
    const bool small = a.bstr[2] < (int64_t)1 << 28 && std::max({a.N[0], a.N[1], a.N[2]}) < (int64_t)1 << 30;
    return small ? launch_form<FORM, uint32_t>(D, a, plan, s)
                                       : launch_form<FORM, int64_t>(D, a, plan, s);
}

HeatArgs march_args(const CartTopo& topo, const SlabLayout& L, int field, const int periodic[3], double kappa,
                    const double inv_h2[3]) {
    HeatArgs a{};
    const int64_t blk = (int64_t)L.nfields * L.slab_stride;
    // dimensions of the kernel: x, y (absent in 2-D), march
    const int dim[3] = {0, topo.D == 3 ? 1 : -1, topo.D - 1};
    for (int k = 0; k < 3; ++k) {
        const int d = dim[k];
        if (d < 0) {
            a.N[k] = a.n[k] = 1;
            continue;
        }
        int64_t bs = blk, cs = 1;
        for (int e = 0; e < d; ++e) {
            bs *= topo.nb[e];
            cs *= L.gdim[e];
        }
        a.N[k] = (int64_t)topo.n[d] * topo.nb[d];
        a.n[k] = topo.n[d];
        a.periodic[k] = periodic[d];
        a.bstr[k] = bs;
        a.cstr[k] = cs;
        a.ih[k] = inv_h2[d];
    }
    a.kappa = kappa;
    a.zero = kappa > 0.0 ? 0.0 : -0.0;
    return a;
}
}  // namespace

bool heat_march_supported(const CartTopo& topo, const SlabLayout& L) { return topo.D >= 2 && L.ghost == 1; }

cudaError_t launch_heat_march_fe(int steps, const double* in, double* out, const CartTopo& topo, const SlabLayout& L,
                                 int field, const int periodic[3], double kappa, double dt, const double inv_h2[3],
                                 HeatPlan& plan, cudaStream_t s) {
    HeatArgs a = march_args(topo, L, field, periodic, kappa, inv_h2);
    a.in = in + (int64_t)field * L.slab_stride;
    a.out = out + (int64_t)field * L.slab_stride;
    a.c1 = a.c2 = dt;
    return steps == 2 ? launch_form<kFe2>(topo.D, a, plan, s) : launch_form<kFe1>(topo.D, a, plan, s);
}

cudaError_t launch_heat_march_rk4(int half, const double* in, double* out, const double* y, double* aux,
                                  const CartTopo& topo, const SlabLayout& L, int field, const int periodic[3],
                                  double kappa, double dt, const double inv_h2[3], HeatPlan& plan, cudaStream_t s) {
    HeatArgs a = march_args(topo, L, field, periodic, kappa, inv_h2);
    const int64_t f = (int64_t)field * L.slab_stride;
    a.in = in + f;
    a.out = out + f;
    a.s6 = dt / 6.0;  // rk4.rs:74-75
    a.s3 = dt / 3.0;
    if (half == 0) {
        a.aux = aux + f;
        a.c1 = a.c2 = 0.5 * dt;  // rk4.rs:57
        return launch_form<kRkA>(topo.D, a, plan, s);
    }
    a.y = y + f;
    a.aux_in = aux + f;
    a.c1 = dt;
    return launch_form<kRkB>(topo.D, a, plan, s);
}

}  // namespace lg
