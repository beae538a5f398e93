// Warp-strip Model C step kernel, generic over an arithmetic policy.
//
// Work unit: one warp owns a strip of 32 columns of one block over a run of
// rows and walks up the rows; lane l owns column 32 s + l.  Warps are
// independent -- no barriers, no shared memory.
//
// Every face flux of the Karma-Rappel divergence is computed once and
// shared by the two cells that touch it: the reference evaluates the right
// face of cell i and the left face of cell i+1 (and top of j / bottom of
// j+1) with the same expression in the same operand order
// (finite_volume.rs:261-280), so sharing is bit-exact and halves the face
// work.  Lane l computes the x face on the left of its column and receives
// its right face from lane l+1 by a shuffle; the strip's last lane takes it
// from a batch of 32 right-boundary faces that the warp evaluates with its
// lanes across rows (one extra face per 32 cells).  The y face below a cell
// is the y face above it in the previous row, carried in a register.
//
// The row loop keeps a window of four phi rows (j-1, j, j+1 and the
// prefetch of j+2).  It keeps one copy of the row code and shifts the window
// by register moves; only the FP32 oriented form unrolls it four times, so
// that the window rotates with no moves.
//
// Ops (the arithmetic policy) provides, for element type T:
//   xface(m, dn, d1, c, e)  flux A (A dn - A' dt) through an x face, with the
//                           normal difference dn and the transverse
//                           difference dt = 0.25 ((d1 + c) - e)
//   yface(m, dn, d1, c, e)  flux A (A dn + A' dt) through a y face
//   cell(...)               the cell's dphi/dt and du/dt from its four face
//                           fluxes, phi, the central differences and the
//                           five u values
//   axpy(dt, k, x)          x + dt k
//   noise(key)              N(key), the Gaussian of one cell
//   add_noise(x, s, n)      x + s n
//   oxface/oyface/ocell     the same in a cell's crystal frame (ORIENT)
// The operand lists keep the reference's evaluation order available to an
// exact policy.
//
// Template flags beside the arithmetic: ORIENT steps the multi-grain form
// (every face's anisotropy in its cell's crystal frame, cos/sin theta0 from a
// per-state table); MODE 0 is the Euler-Maruyama step, MODE 1 to 3 the
// RungeKutta4 stages (see RkArgs); BATCH serves ensembles; TAIL blocks lower
// than the row group.
#pragma once

#include <algorithm>
#include <type_traits>

#include "lg_common.cuh"
#include "lg_kernels.h"
#include "lg_strip_plan.h"
#include "lg_modelc_ops.cuh"

namespace lg {

struct TileArgs {
    CartTopo topo;
    SlabLayout L;
    double dt64;
    uint64_t seed;
    double* tdev;
    int slot;
    int rows;     // rows per work unit
    int strips;   // 32-column strips per block
    int chunks;   // row chunks per block
    int64_t units;
    // persistent work list (null: a static grid-stride schedule): one wave of
    // CTAs, each warp taking its first unit by position and every further one
    // from work[0].  work[1] counts the warps that are done; the last one sets
    // both back to zero for the next launch
    unsigned* work;
};

// Batched instances (BATCH kernels): block b belongs to instance b / bpi,
// whose parameters are params[instance] (an Ops::Params array on the
// device) and whose Wiener seed is seeds[instance]; its noise keys use the
// instance-local block index b % bpi.
struct BatchArgs {
    const void* params;
    const uint64_t* seeds;
    int bpi;
};

// RungeKutta4 stages (MODE 1, 2, 3; rk4.rs:40-79).  All arenas share the
// state's slab layout.  The step's result is the chain of axpys ((((y + dt/6
// k1) + dt/3 k2) + dt/3 k3) + dt/6 k4); `acc` carries it from stage to stage in
// that order, so no k is stored.  MODE 1 (stage 1, the input is y): the output
// is y + c k, acc = y + s k.  MODE 2 (stages 2 and 3): the output is y + c k,
// acc += s k.  MODE 3 (stage 4): the output is acc + s k.
template <class T>
struct RkArgs {
    const T* y;
    T* acc;
    T c, s;
};

// Ghost images of a strip's x-edge cells (the block's columns 0 and n0 - 1;
// rows 0 and n1 - 1, whose images include y ghosts and corners, are pushed in
// full).  FP64: the lane that owns an edge cell keeps the address of its image
// in the unit's first row -- the neighbour's ghost column, or this block's own
// at a mirror boundary -- and stores there as it stores the cell.  FP32: the
// images are gathered by shuffles, lane k holding those of row r0 + k (l0, l1:
// phi and u of the left edge cell, q0, q1: of the right one), and written once
// at the unit's end.  (The FP64 gather is 32 shuffles and selects a pass:
// 2002^2 in blocks of 91 x 77 without noise 61 -> 58 us a step with stores as
// the rows go, 10080^2 1357 -> 1327, but FP32 4096^2 in blocks of 256^2 143 ->
// 147.)
template <class T>
struct EdgeImages {
    static constexpr bool kGather = sizeof(T) == 4;
    T* p;  // this lane's image in row r0; null: not an edge cell
    T l0, l1, q0, q1;
    __device__ __forceinline__ EdgeImages(T* __restrict__ out, const SlabLayout& L, const Nbr2& nb, int n0, int r0,
                                          int col)
        : p(nullptr), l0(T(0)), l1(T(0)), q0(T(0)), q1(T(0)) {
        if constexpr (!kGather) {
            if (col == 0)
                p = out + slab_base(L, nb.l >= 0 ? nb.l : nb.b, 0) + (nb.l >= 0 ? n0 + 1 : 0);
            else if (col == n0 - 1)
                p = out + slab_base(L, nb.r >= 0 ? nb.r : nb.b, 0) + (nb.r >= 0 ? 0 : n0 + 1);
            if (p) p += (int64_t)(r0 + 1) * L.gdim[0];
        }
    }
    // one row of a strip on a block's x edge (the whole warp calls)
    __device__ __forceinline__ void row(T phin, T un, bool ok, bool live, int k, int lane, int last_lane, int sy,
                                        int64_t slab_stride) {
        if constexpr (kGather) {
            const T a0 = __shfl_sync(0xffffffffu, phin, 0), a1 = __shfl_sync(0xffffffffu, un, 0);
            const T b0 = __shfl_sync(0xffffffffu, phin, last_lane), b1 = __shfl_sync(0xffffffffu, un, last_lane);
            if (live && lane == (k & 31)) {
                l0 = a0;
                l1 = a1;
                q0 = b0;
                q1 = b1;
            }
        } else if (ok && p) {
            T* const q = p + (int64_t)k * sy;
            q[0] = phin;
            q[slab_stride] = un;
        }
    }
};

// store the cell, and take care of its ghost images (see EdgeImages;
// one-column blocks push every row in full)
template <class T>
__device__ __forceinline__ void store_cell(T* __restrict__ out, T* __restrict__ po, T* __restrict__ uo, int off,
                                           T phin, T un, bool ok, bool live, bool edge_x, int j, int r0, int n0,
                                           int n1, int col, int lane, int last_lane, int sy, const SlabLayout& L,
                                           const Nbr2& nb, EdgeImages<T>& eh) {
    if (ok) {
        po[off] = phin;
        uo[off] = un;
    }
    if (j == 0 || j == n1 - 1 || (!EdgeImages<T>::kGather && n0 == 1)) {  // warp-uniform
        if (ok) {
            push_ghosts_2d_g1(out, L, 0, nb, n0, n1, col, j, phin);
            push_ghosts_2d_g1(out, L, 1, nb, n0, n1, col, j, un);
        }
    } else if (edge_x) {  // warp-uniform
        eh.row(phin, un, ok, live, j - r0, lane, last_lane, sy, L.slab_stride);
    }
}

// the collected x-edge images of a unit's rows (r0 .. r1-1, not 0 or n1-1):
// the left edge's into the left neighbour's ghost column n0 (or this block's
// mirror ghost column -1), the right edge's likewise (push_ghosts_2d_g1); FP32 only
template <class T>
__device__ __forceinline__ void flush_edges(T* __restrict__ out, const SlabLayout& L, const Nbr2& nb, int n0, int n1,
                                            int r0, int r1, int lane, bool left, bool right, const EdgeImages<T>& eh,
                                            int rs = -1) {
    const int r = r0 + lane;
    if (r >= r1 || r < rs || r == 0 || r == n1 - 1) return;  // rows below rs: another unit's
    const int64_t row = (int64_t)(r + 1) * L.gdim[0];
    if (left) {
        const int tb = nb.l >= 0 ? nb.l : nb.b, ci = nb.l >= 0 ? n0 : -1;
        out[slab_base(L, tb, 0) + (ci + 1) + row] = eh.l0;
        out[slab_base(L, tb, 1) + (ci + 1) + row] = eh.l1;
    }
    if (right) {
        const int tb = nb.r >= 0 ? nb.r : nb.b, ci = nb.r >= 0 ? -1 : n0;
        out[slab_base(L, tb, 0) + (ci + 1) + row] = eh.q0;
        out[slab_base(L, tb, 1) + (ci + 1) + row] = eh.q1;
    }
}

// The new phi and u of a cell from its drift (kphi, ku): the Euler-Maruyama
// update (MODE 0) or a RungeKutta4 stage (MODE 1 to 3); e0/e1 index the cell's
// phi/u entries in any arena of the state's layout.
//
// RkCell: the other operands of a cell's stage, loaded before the drift they
// are added to is known.
template <class T>
struct RkCell {
    T y0, y1, a0, a1;
};
template <class T, int MODE>
__device__ __forceinline__ void rk_load(const RkArgs<T>& rk, int64_t e0, int64_t e1, RkCell<T>& c) {
    if constexpr (MODE >= 2) {
        c.a0 = rk.acc[e0];
        c.a1 = rk.acc[e1];
    }
    if constexpr (MODE == 2) {
        c.y0 = __ldg(rk.y + e0);
        c.y1 = __ldg(rk.y + e1);
    }
}
template <class T, class Ops, bool NOISE, int MODE>
__device__ __forceinline__ void cell_update(const RkArgs<T>& rk, const RkCell<T>& rc, T dt, T scale_amp, T nval,
                                            T kphi, T ku, T p, T uc, int64_t e0, int64_t e1, bool ok, T& phin,
                                            T& un) {
    if constexpr (MODE == 0) {
        phin = Ops::axpy(dt, kphi, p);
        if (NOISE) phin = Ops::add_noise(phin, scale_amp, nval);
        un = Ops::axpy(dt, ku, uc);
    } else if constexpr (MODE == 1) {
        phin = p + rk.c * kphi;
        un = uc + rk.c * ku;
        if (ok) {
            rk.acc[e0] = p + rk.s * kphi;
            rk.acc[e1] = uc + rk.s * ku;
        }
    } else {
        const T a0 = rc.a0 + rk.s * kphi, a1 = rc.a1 + rk.s * ku;
        if constexpr (MODE == 2) {
            phin = rc.y0 + rk.c * kphi;
            un = rc.y1 + rk.c * ku;
            if (ok) {
                rk.acc[e0] = a0;
                rk.acc[e1] = a1;
            }
        } else {
            phin = a0;
            un = a1;
        }
    }
}

// Multi-grain kernels (ORIENT): cos theta0 of every interior cell, blocks in
// order and each block's cells dimension-0-fastest, followed by sin theta0
// in the same order (ncells values each), in the kernel's element type.
struct OrientArgs {
    const void* trig;
    int64_t ncells;
};

template <class T>
struct Row3 {
    T a, b, c;  // columns c-1, c, c+1
};

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ bool same_bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_int(a) == __float_as_int(b); }

// One row: x face left of the lane's column, y face above cell (c, j), the
// cell update, stores and ghost pushes.  A, B, C = phi rows j-1, j, j+1 at
// columns c-1, c, c+1; UA, UB, UC = u at column c for the same rows; P / UP
// receive the prefetch of row j+1+PF.  `off` is the slab offset of (col, j); ph/uu/po/uo
// are the warp's slab bases.  NX > 0 fixes the block width (and the row
// stride) at compile time; FULL means every lane owns a column.
template <class T, class Ops, bool NOISE, int NX, bool FULL, int PF, bool TAIL, bool ORIENT, int MODE>
__device__ __forceinline__ void strip_row(const typename Ops::Params& m, const TileArgs& g, int j, int r0, int r1,
                                          int lane,
                                          int col, bool valid, int last_lane, int n0, int n1, int off,
                                          const T* __restrict__ ph, const T* __restrict__ uu, T* __restrict__ out,
                                          T* __restrict__ po, T* __restrict__ uo, const Nbr2& nb, bool edge_x,
                                          uint64_t block_key, T bnd, const Row3<T>& A, const Row3<T>& B,
                                          const Row3<T>& C, Row3<T>& P, T UA, T UB, T UC, T& UP, T& jb, T dt,
                                          T scale_amp, const T* __restrict__ trig_b, int64_t ncells, T& cprev,
                                          T& sprev, T& cnext, T& snext, const RkArgs<T>& rk,
                                          EdgeImages<T>& eh, int rs) {
    const int sy = NX > 0 ? NX + 2 : g.L.gdim[0];
    // lanes past the block's last column (valid false) run the same code on
    // a clamped column and only skip the stores: no branch splits the face,
    // noise and cell arithmetic.  Unit heights are whole groups of rows
    // (strip_group), so an unrolled row loop has no separate tail; only blocks
    // of fewer rows (TAIL) run rows past the unit's end, without stores.
    // rows below rs belong to the unit below (a block's last unit overlaps
    // it): computed for their faces, stored only by their own unit
    const bool live = (!TAIL || j < r1) && j >= rs;
    const bool ok = (FULL || valid) && live;
    if (j + 1 + PF <= n1) {
        const T* q = ph + off + (1 + PF) * sy;
        P.a = __ldg(q - 1);
        P.b = __ldg(q);
        P.c = __ldg(q + 1);
        UP = __ldg(uu + off + (1 + PF) * sy);
    }
    T ul = T(0), ur = T(0);
    if (live) {
        ul = __ldg(uu + off - 1);
        ur = __ldg(uu + off + 1);
    }
    RkCell<T> rc{};
    if (live) rk_load<T, MODE>(rk, (po - out) + off, (uo - out) + off, rc);
    T nval = T(0);
    if (NOISE) nval = Ops::noise(splitmix64(block_key ^ (uint64_t)(col + j * n0)));
    if constexpr (ORIENT) {
        // multi-grain: every face's anisotropy in the frame of the cell being
        // updated.  Within a grain two neighbours share theta0, and the
        // reference evaluates their common face from the same differences in
        // the same order, so it is computed once: the left face comes from
        // this lane, the right face from the next lane (or the strip's
        // boundary batch), the bottom face from the previous row.  Where the
        // neighbour's cos/sin theta0 differ (grain boundaries), the face is
        // evaluated again in this cell's frame.
        // this row's frame arrived with the previous row; fetch the next one
        const T c0 = cnext, s0 = snext;
        if (j + 1 < n1) {
            const int64_t ci = (int64_t)(j + 1) * n0 + (FULL ? col : min(col, n0 - 1));
            cnext = __ldg(trig_b + ci);
            snext = __ldg(trig_b + ncells + ci);
        }
        const T q = T(0.25);
        const T jl = Ops::oxface(m, c0, s0, B.b - B.a, q * (C.b - A.b + C.a - A.a));
        const T jt = Ops::oyface(m, c0, s0, q * (C.c - C.a + B.c - B.a), C.b - B.b);
        T jr = __shfl_down_sync(kFull, jl, 1);
        const T c0n = __shfl_down_sync(kFull, c0, 1), s0n = __shfl_down_sync(kFull, s0, 1);
        const T fb = __shfl_sync(kFull, bnd, (j - r0) & 31);
        if (lane == last_lane)
            jr = fb;
        else if (!(same_bits(c0n, c0) && same_bits(s0n, s0)))
            jr = Ops::oxface(m, c0, s0, B.c - B.b, q * (C.c - A.c + C.b - A.b));
        T jbot = jb;
        if (!(same_bits(cprev, c0) && same_bits(sprev, s0)))
            jbot = Ops::oyface(m, c0, s0, q * (B.c - B.a + A.c - A.a), B.b - A.b);
        T kphi, ku;
        Ops::ocell(m, jr, jl, jt, jbot, B.b, B.c - B.a, C.b - A.b, c0, s0, UB, ul, ur, UC, UA, kphi, ku);
        T phin, un;
        cell_update<T, Ops, NOISE, MODE>(rk, rc, dt, scale_amp, nval, kphi, ku, B.b, UB, (po - out) + off,
                                         (uo - out) + off, ok, phin, un);
        store_cell(out, po, uo, off, phin, un, ok, live, edge_x, j, r0, n0, n1, col, lane, last_lane, sy, g.L, nb, eh);
        jb = jt;
        cprev = c0;
        sprev = s0;
        return;
    }
    const T fl = Ops::xface(m, B.b - B.a, C.b - A.b, C.a, A.a);
    const T jt = Ops::yface(m, C.b - B.b, C.c - C.a, B.c, B.a);
    // right face: the next lane's left face, or the strip's boundary face of this row
    T fr = __shfl_down_sync(kFull, fl, 1);
    const T fb = __shfl_sync(kFull, bnd, (j - r0) & 31);
    if (lane == last_lane) fr = fb;
    T kphi, ku;
    Ops::cell(m, fr, fl, jt, jb, B.b, B.c - B.a, C.b - A.b, UB, ul, ur, UC, UA, kphi, ku);
    T phin, un;
    cell_update<T, Ops, NOISE, MODE>(rk, rc, dt, scale_amp, nval, kphi, ku, B.b, UB, (po - out) + off, (uo - out) + off,
                                     ok, phin, un);
    store_cell(out, po, uo, off, phin, un, ok, live, edge_x, j, r0, n0, n1, col, lane, last_lane, sy, g.L, nb, eh);
    jb = jt;
}

// One work unit of the strip kernel: the rows [r0, r1) of the 32-column
// strip at c0 of block b, with the parameter record m (the kernel parameter,
// or a batched instance's record) and the Wiener key of block key_block.
template <class T, class Ops, bool NOISE, int NX, bool FULL, int PF, bool TAIL, bool ORIENT, int MODE>
__device__ __forceinline__ void strip_unit(const typename Ops::Params& m, uint64_t seed, int key_block,
                                           const TileArgs& g, const T* __restrict__ ph, const T* __restrict__ uu,
                                           T* __restrict__ out, T* __restrict__ po, T* __restrict__ uo,
                                           const Nbr2& nb, int r0, int r1, int lane, int col, bool valid,
                                           int last_lane, int cr, bool edge_x, int n0, int n1, int sy, double tnow,
                                           T dt, T scale_amp, const T* __restrict__ trig_b, int64_t ncells, const RkArgs<T>& rk,
                                           int rs) {
    constexpr int NB = PF + 3;
    uint64_t block_key = 0;
    if (NOISE)
        block_key = wiener_block_key(seed, (uint64_t)__double_as_longlong(tnow), kWienerStream0,
                                     (uint64_t)key_block);

    // slab offset of (col, r0); a lane past the last column reads the last one
    int off = ((FULL ? col : min(col, n0 - 1)) + 1) + (r0 + 1) * sy;
    Row3<T> w[NB];
    T uw[NB];
    T jb = T(0);
    // window: rows r0-1 .. r0+PF in w[0..NB-2]; w[NB-1] is filled by the first row
#pragma unroll
    for (int q = 0; q < NB - 1; ++q) {
        w[q] = Row3<T>{};
        uw[q] = T(0);
        const int r = r0 - 1 + q;
        if (r <= n1) {
            const T* p = ph + off + (q - 1) * sy;
            w[q] = {__ldg(p - 1), __ldg(p), __ldg(p + 1)};
            uw[q] = __ldg(uu + off + (q - 1) * sy);
        }
    }
    w[NB - 1] = Row3<T>{};
    uw[NB - 1] = T(0);
    // right-boundary face of the strip for rows r0 .. r0+31 (lane = row)
    T bnd = T(0);
    if constexpr (!ORIENT) {
        const int r = r0 + lane;
        if (r < r1) {
            const T* q = ph + (cr + 1) + (r + 1) * sy;  // (column cr, row r)
            const T c0m = __ldg(q - sy), c1m = __ldg(q - sy + 1);
            const T c00 = __ldg(q), c10 = __ldg(q + 1);
            const T c0p = __ldg(q + sy), c1p = __ldg(q + sy + 1);
            bnd = Ops::xface(m, c10 - c00, c1p - c1m, c0p, c0m);
        }
    } else {  // the same faces in the frame of the strip's last cell of each row
        const int r = r0 + lane;
        if (r < r1) {
            const T* q = ph + (cr + 1) + (r + 1) * sy;
            const T c0m = __ldg(q - sy), c1m = __ldg(q - sy + 1);
            const T c00 = __ldg(q), c10 = __ldg(q + 1);
            const T c0p = __ldg(q + sy), c1p = __ldg(q + sy + 1);
            const int64_t ci = (int64_t)r * n0 + cr;
            bnd = Ops::oxface(m, __ldg(trig_b + ci), __ldg(trig_b + ncells + ci), c10 - c00,
                              T(0.25) * (c1p - c1m + c0p - c0m));
        }
    }
    // y face below the first row (between r0-1 and r0)
    T cpv = T(0), spv = T(0);  // cos/sin theta0 of the previous row's cell (multi-grain)
    T cnx = T(0), snx = T(0);  // and of the row about to be stepped
    if constexpr (!ORIENT) {
        jb = Ops::yface(m, w[1].b - w[0].b, w[1].c - w[1].a, w[0].c, w[0].a);
    } else {  // bottom face of the first row in its own frame
        const int64_t ci = (int64_t)r0 * n0 + (FULL ? col : min(col, n0 - 1));
        cpv = cnx = __ldg(trig_b + ci);
        spv = snx = __ldg(trig_b + ncells + ci);
        jb = Ops::oyface(m, cpv, spv, T(0.25) * (w[1].c - w[1].a + w[0].c - w[0].a), w[1].b - w[0].b);
    }

    EdgeImages<T> eh(out, g.L, nb, n0, r0, col);
#define LG_ROW(J, Q)                                                                                            \
    strip_row<T, Ops, NOISE, NX, FULL, PF, TAIL, ORIENT, MODE>(m, g, J, r0, r1, lane, col, valid, last_lane, n0, n1, off, ph, uu, out, po,  \
                                       uo, nb, edge_x, block_key, bnd, w[(Q) % NB], w[((Q) + 1) % NB],          \
                                       w[((Q) + 2) % NB], w[((Q) + 2 + PF) % NB], uw[(Q) % NB],                \
                                       uw[((Q) + 1) % NB], uw[((Q) + 2) % NB], uw[((Q) + 2 + PF) % NB], jb, dt, \
                                       scale_amp, trig_b, ncells, cpv, spv, cnx, snx, rk, eh, rs);                                                          \
    off += sy
    if constexpr (sizeof(T) == 8 || !ORIENT) {
        // one copy of the row code: the window shifts down by one row
        // through registers instead of rotating through NB unrolled copies,
        // which overflowed the instruction cache and spilled (FP64 4096^2:
        // 51.8 against 45.1 Gcell/s; 10080^2 with 1000 oriented grains: 33.7
        // against 25.3; FP32 4096^2: 100.1 against 94.2, and 3 CTAs per SM
        // without spills).  The FP32 oriented form is faster unrolled
        // (10080^2: 74.7 against 71.8).
#pragma unroll 1
        for (int j = r0; j < r1; ++j) {
            LG_ROW(j, 0);
#pragma unroll
            for (int q = 0; q + 1 < NB; ++q) {
                w[q] = w[q + 1];
                uw[q] = uw[q + 1];
            }
        }
    } else {
        for (int j = r0; j < r1; j += NB) {
#pragma unroll
            for (int q = 0; q < NB; ++q) { LG_ROW(j + q, q); }
        }
    }
#undef LG_ROW
    if constexpr (EdgeImages<T>::kGather)
        if (edge_x) flush_edges(out, g.L, nb, n0, n1, r0, r1, lane, col - lane == 0, cr == n0 - 1, eh, rs);
}

// The paired form of one work unit (an Euler-Maruyama step or an RK4 stage,
// axis-aligned or multi-grain; units of an even number of rows): each pass of
// the row loop steps rows j and j+1 together, so every lane carries two independent cells -- four face fluxes,
// two Gaussians, two cell updates -- whose dependency chains the scheduler
// interleaves; the y face between the two rows is computed once.  Each pass
// reads its four phi and u rows j-1 .. j+2 from L1, where the previous pass
// prefetched them, instead of carrying a six-row window in registers: the
// unit needs fewer registers (no spills at 3 CTAs per SM) and no register
// moves to shift the window.  Units are an even number of rows ending at or
// before the ghost row n1, so every row read lies inside the slab.
// Same arithmetic per cell, in the same operand order, as strip_row.
//
// ORIENT: the multi-grain faces (strip_row's ORIENT branch, for two rows):
// each face in the frame of the cell being updated, shared with the
// neighbour only where the neighbour's cos/sin theta0 are the same bits,
// else evaluated again in this cell's frame.
template <class T, class Ops, bool NOISE, int NX, bool FULL, bool ORIENT = false, int MODE = 0>
__device__ __forceinline__ void strip_unit_pair(const typename Ops::Params& m, uint64_t seed, int key_block,
                                                const TileArgs& g, const T* __restrict__ ph,
                                                const T* __restrict__ uu, T* __restrict__ out, T* __restrict__ po,
                                                T* __restrict__ uo, const Nbr2& nb, int r0, int r1, int lane,
                                                int col, bool valid, int last_lane, int cr, bool edge_x, int n0,
                                                int n1, int sy, double tnow, T dt, T scale_amp, int rs, const RkArgs<T>& rk,
                                                const T* __restrict__ trig_b = nullptr, int64_t ncells = 0) {
    uint64_t block_key = 0;
    if (NOISE)
        block_key = wiener_block_key(seed, (uint64_t)__double_as_longlong(tnow), kWienerStream0,
                                     (uint64_t)key_block);
    const bool ok = FULL || valid;
    // slab offset of (col, r0), fixed for the unit; `off` follows the row pair
    const int off0 = ((FULL ? col : min(col, n0 - 1)) + 1) + (r0 + 1) * sy;
    int off = off0;
    // phi (columns col-1, col, col+1) and u of row r, for -1 <= r <= n1 (row
    // n1 is the ghost row); rows past n1 read as zero and are never used
    auto load_row = [&](int r, Row3<T>& w, T& uw) {
        w = Row3<T>{};
        uw = T(0);
        if (r <= n1) {
            const T* q = ph + off0 + (r - r0) * sy;
            w = {__ldg(q - 1), __ldg(q), __ldg(q + 1)};
            uw = __ldg(uu + off0 + (r - r0) * sy);
        }
    };
    Row3<T> A, B, C, D;
    T UA, UB, UC, UD;
    load_row(r0 - 1, A, UA);
    load_row(r0, B, UB);
    T bnd = T(0);
    {
        const int r = r0 + lane;
        if (r < r1) {
            const T* q = ph + (cr + 1) + (r + 1) * sy;  // (column cr, row r)
            const T c0m = __ldg(q - sy), c1m = __ldg(q - sy + 1);
            const T c00 = __ldg(q), c10 = __ldg(q + 1);
            const T c0p = __ldg(q + sy), c1p = __ldg(q + sy + 1);
            if constexpr (ORIENT) {  // in the frame of the strip's last cell of the row
                const int64_t ci = (int64_t)r * n0 + cr;
                bnd = Ops::oxface(m, __ldg(trig_b + ci), __ldg(trig_b + ncells + ci), c10 - c00,
                                  T(0.25) * (c1p - c1m + c0p - c0m));
            } else {
                bnd = Ops::xface(m, c10 - c00, c1p - c1m, c0p, c0m);
            }
        }
    }
    const int ccol = FULL ? col : min(col, n0 - 1);
    T cprev = T(0), sprev = T(0);  // multi-grain: cos/sin theta0 of the row below the pass
    T jb;
    if constexpr (ORIENT) {  // the bottom face of the first row in its own frame
        const int64_t ci = (int64_t)r0 * n0 + ccol;
        cprev = __ldg(trig_b + ci);
        sprev = __ldg(trig_b + ncells + ci);
        jb = Ops::oyface(m, cprev, sprev, T(0.25) * (B.c - B.a + A.c - A.a), B.b - A.b);
    } else {
        jb = Ops::yface(m, B.b - A.b, B.c - B.a, A.c, A.a);
    }
    EdgeImages<T> eh(out, g.L, nb, n0, r0, col);
#pragma unroll 1
    for (int j = r0; j < r1; j += 2) {
        // the four rows of this pass (j-1 .. j+2 <= n1) from L1, and an L1
        // prefetch of the next pass's two new rows
        {
            const T* q = ph + off - sy;
            A = {__ldg(q - 1), __ldg(q), __ldg(q + 1)};
            B = {__ldg(q + sy - 1), __ldg(q + sy), __ldg(q + sy + 1)};
            C = {__ldg(q + 2 * sy - 1), __ldg(q + 2 * sy), __ldg(q + 2 * sy + 1)};
            D = {__ldg(q + 3 * sy - 1), __ldg(q + 3 * sy), __ldg(q + 3 * sy + 1)};
            const T* w = uu + off - sy;
            UA = __ldg(w);
            UB = __ldg(w + sy);
            UC = __ldg(w + 2 * sy);
            UD = __ldg(w + 3 * sy);
            const int64_t p3 = (int64_t)(min(j + 3, n1) - j) * sy, p4 = (int64_t)(min(j + 4, n1) - j) * sy;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(ph + off + p3));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(ph + off + p4));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(uu + off + p3));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(uu + off + p4));
        }
        RkCell<T> rc0{}, rc1{};
        rk_load<T, MODE>(rk, (po - out) + off, (uo - out) + off, rc0);
        rk_load<T, MODE>(rk, (po - out) + off + sy, (uo - out) + off + sy, rc1);
        const T ul0 = __ldg(uu + off - 1), ur0 = __ldg(uu + off + 1);
        const T ul1 = __ldg(uu + off + sy - 1), ur1 = __ldg(uu + off + sy + 1);
        T c0 = T(0), s0 = T(0), c1 = T(0), s1 = T(0);  // multi-grain: frames of rows j and j+1
        if constexpr (ORIENT) {
            const int64_t ci = (int64_t)j * n0 + ccol;
            if constexpr (sizeof(T) == 8) {
                // the next pass's frames (2520^2 167 -> 165 us a step; FP32,
                // whose passes are shorter on instructions, 92 -> 97)
                const int64_t p2 = ci + (int64_t)(min(j + 2, n1 - 1) - j) * n0;
                const int64_t p3 = ci + (int64_t)(min(j + 3, n1 - 1) - j) * n0;
                asm volatile("prefetch.global.L1 [%0];" ::"l"(trig_b + p2));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(trig_b + ncells + p2));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(trig_b + p3));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(trig_b + ncells + p3));
            }
            c0 = __ldg(trig_b + ci);
            s0 = __ldg(trig_b + ncells + ci);
            c1 = __ldg(trig_b + ci + n0);
            s1 = __ldg(trig_b + ncells + ci + n0);
        }
        // the Gaussians of the pass, drawn as soon as its loads are issued:
        // their integer and FP64 chains fill the loads' latency and the
        // anisotropy tests that follow, and are needed only at the end
        T nv0 = T(0), nv1 = T(0);
        auto draw = [&]() {
            if (NOISE) {
                nv0 = Ops::noise(splitmix64(block_key ^ (uint64_t)(col + j * n0)));
                nv1 = Ops::noise(splitmix64(block_key ^ (uint64_t)(col + (j + 1) * n0)));
            }
        };
        draw();
        const T fb0 = __shfl_sync(kFull, bnd, (j - r0) & 31), fb1 = __shfl_sync(kFull, bnd, (j + 1 - r0) & 31);
        T phin0, phin1, un0, un1, jt1;
        // rows below rs belong to the unit below (a block's last unit
        // overlaps it): computed for their faces, stored only once
        const bool own0 = j >= rs, own1 = j + 1 >= rs;
        auto update = [&](T kphi0, T ku0, T kphi1, T ku1) {
            const int64_t e0 = (po - out) + off, e1 = (uo - out) + off;
            cell_update<T, Ops, NOISE, MODE>(rk, rc0, dt, scale_amp, nv0, kphi0, ku0, B.b, UB, e0, e1, ok && own0, phin0,
                                             un0);
            cell_update<T, Ops, NOISE, MODE>(rk, rc1, dt, scale_amp, nv1, kphi1, ku1, C.b, UC, e0 + sy, e1 + sy,
                                             ok && own1, phin1, un1);
        };
        if constexpr (MODE >= 2) {  // the stage's other operands of the next pass
            const int64_t next = j + 3 < n1 ? 2 * (int64_t)sy : 0;
            const int64_t e0 = (po - out) + off + next, e1 = (uo - out) + off + next;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.acc + e0));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.acc + e1));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.acc + e0 + sy));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.acc + e1 + sy));
            if constexpr (MODE == 2) {
                asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.y + e0));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.y + e1));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.y + e0 + sy));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(rk.y + e1 + sy));
            }
        }
        if constexpr (ORIENT) {
            const T q = T(0.25);
            const T jl0 = Ops::oxface(m, c0, s0, B.b - B.a, q * (C.b - A.b + C.a - A.a));
            const T jt0 = Ops::oyface(m, c0, s0, q * (C.c - C.a + B.c - B.a), C.b - B.b);
            const T jl1 = Ops::oxface(m, c1, s1, C.b - C.a, q * (D.b - B.b + D.a - B.a));
            jt1 = Ops::oyface(m, c1, s1, q * (D.c - D.a + C.c - C.a), D.b - C.b);
            T jr0 = __shfl_down_sync(kFull, jl0, 1), jr1 = __shfl_down_sync(kFull, jl1, 1);
            const T c0n = __shfl_down_sync(kFull, c0, 1), s0n = __shfl_down_sync(kFull, s0, 1);
            const T c1n = __shfl_down_sync(kFull, c1, 1), s1n = __shfl_down_sync(kFull, s1, 1);
            if (lane == last_lane) {
                jr0 = fb0;
                jr1 = fb1;
            } else {
                if (!(same_bits(c0n, c0) && same_bits(s0n, s0)))
                    jr0 = Ops::oxface(m, c0, s0, B.c - B.b, q * (C.c - A.c + C.b - A.b));
                if (!(same_bits(c1n, c1) && same_bits(s1n, s1)))
                    jr1 = Ops::oxface(m, c1, s1, C.c - C.b, q * (D.c - B.c + D.b - B.b));
            }
            T jbot0 = jb, jbot1 = jt0;
            if (!(same_bits(cprev, c0) && same_bits(sprev, s0)))
                jbot0 = Ops::oyface(m, c0, s0, q * (B.c - B.a + A.c - A.a), B.b - A.b);
            if (!(same_bits(c0, c1) && same_bits(s0, s1)))
                jbot1 = Ops::oyface(m, c1, s1, q * (C.c - C.a + B.c - B.a), C.b - B.b);
            const auto o0 = Ops::ocell_open(m, jr0, jl0, jt0, jbot0, B.b, B.c - B.a, C.b - A.b, c0, s0, UB, ul0,
                                            ur0, UC, UA);
            const auto o1 = Ops::ocell_open(m, jr1, jl1, jt1, jbot1, C.b, C.c - C.a, D.b - B.b, c1, s1, UC, ul1,
                                            ur1, UD, UB);
            T kphi0, ku0, kphi1, ku1;
            Ops::close2(m, o0, o1, Ops::divides(m), kphi0, ku0, kphi1, ku1);
            update(kphi0, ku0, kphi1, ku1);
            cprev = c1;
            sprev = s1;
        } else {
            // the four faces' and two centres' gradients; where all are flat
            // for certain across the warp (the far field) the pass runs without
            // branches, with the general path's values; elsewhere the general
            // path leaves its range tests out where the gradients allow it
            const T xn0 = B.b - B.a, xt0 = Ops::quarter(C.b - A.b, C.a, A.a);
            const T yn0 = C.b - B.b, yt0 = Ops::quarter(C.c - C.a, B.c, B.a);
            const T xn1 = C.b - C.a, xt1 = Ops::quarter(D.b - B.b, D.a, B.a);
            const T yn1 = D.b - C.b, yt1 = Ops::quarter(D.c - D.a, C.c, C.a);
            const unsigned faces =
                max(max(Ops::key(xn0, xt0), Ops::key(yt0, yn0)), max(Ops::key(xn1, xt1), Ops::key(yt1, yn1)));
            const unsigned centers = max(Ops::key(B.c - B.a, C.b - A.b), Ops::key(C.c - C.a, D.b - B.b));
            typename Ops::Cell o0, o1;
            auto right_faces = [&](T fl0, T fl1, T& fr0, T& fr1) {
                fr0 = __shfl_down_sync(kFull, fl0, 1);
                fr1 = __shfl_down_sync(kFull, fl1, 1);
                if (lane == last_lane) {
                    fr0 = fb0;
                    fr1 = fb1;
                }
            };
            auto general = [&](auto safe) {
                constexpr bool S = decltype(safe)::value;
                const T fl0 = Ops::template xface<S>(m, B.b - B.a, C.b - A.b, C.a, A.a);
                const T jt0 = Ops::template yface<S>(m, C.b - B.b, C.c - C.a, B.c, B.a);
                const T fl1 = Ops::template xface<S>(m, C.b - C.a, D.b - B.b, D.a, B.a);
                jt1 = Ops::template yface<S>(m, D.b - C.b, D.c - D.a, C.c, C.a);
                T fr0, fr1;
                right_faces(fl0, fl1, fr0, fr1);
                o0 = Ops::template cell_open<S>(m, fr0, fl0, jt0, jb, B.b, B.c - B.a, C.b - A.b, UB, ul0, ur0, UC, UA);
                o1 = Ops::template cell_open<S>(m, fr1, fl1, jt1, jt0, C.b, C.c - C.a, D.b - B.b, UC, ul1, ur1, UD,
                                                UB);
            };
            if (__all_sync(kFull, Ops::far(m, faces, centers))) {
                const T fl0 = Ops::xface_far(m, xn0), jt0 = Ops::yface_far(m, yn0), fl1 = Ops::xface_far(m, xn1);
                jt1 = Ops::yface_far(m, yn1);
                T fr0, fr1;
                right_faces(fl0, fl1, fr0, fr1);
                o0 = Ops::cell_far(m, fr0, fl0, jt0, jb, B.b, UB, ul0, ur0, UC, UA);
                o1 = Ops::cell_far(m, fr1, fl1, jt1, jt0, C.b, UC, ul1, ur1, UD, UB);
            } else if (!Ops::kGuarded ||
                       __all_sync(kFull, Ops::safe(m, faces, centers, B.b, C.b))) {
                general(std::true_type{});
            } else {
                general(std::false_type{});
                Ops::divide(o0);
                Ops::divide(o1);
            }
            T kphi0, ku0, kphi1, ku1;
            Ops::close2(m, o0, o1, false, kphi0, ku0, kphi1, ku1);
            update(kphi0, ku0, kphi1, ku1);
        }
        store_cell(out, po, uo, off, phin0, un0, ok && own0, own0, edge_x, j, r0, n0, n1, col, lane, last_lane, sy,
                   g.L, nb, eh);
        store_cell(out, po, uo, off + sy, phin1, un1, ok && own1, own1, edge_x, j + 1, r0, n0, n1, col, lane,
                   last_lane, sy, g.L, nb, eh);
        jb = jt1;
        off += 2 * sy;
    }
    if constexpr (EdgeImages<T>::kGather)
        if (edge_x) flush_edges(out, g.L, nb, n0, n1, r0, r1, lane, col - lane == 0, cr == n0 - 1, eh, rs);
}

// strip, row chunk and block of a work unit
struct StripUnit {
    int s, k, b;
    // 32-bit divisions: a grid holds fewer than 2^32 units
    __device__ __forceinline__ void decode(const TileArgs& g, int64_t unit) {
        const unsigned bk = (unsigned)unit / (unsigned)g.strips;
        s = (int)((unsigned)unit - bk * (unsigned)g.strips);
        b = (int)(bk / (unsigned)g.chunks);
        k = (int)(bk - (unsigned)b * (unsigned)g.chunks);
    }
};

// Rows per work unit are at most 32, so one batch of boundary faces (lanes
// across rows) serves the whole unit.
template <class T, class Ops, bool NOISE, int MINB, int NX, int PF, bool BATCH = false, bool TAIL = false,
          bool ORIENT = false, int MODE = 0, bool PAIR = false>
__global__ void __launch_bounds__(256, MINB)
    modelc_strip_kernel(const T* __restrict__ in, T* __restrict__ out, TileArgs g, typename Ops::Params m0, T dt,
                        T scale_amp, BatchArgs bt, OrientArgs oa, RkArgs<T> rk) {
    constexpr bool FULL = NX > 0 && NX % 32 == 0;
    const CartTopo& topo = g.topo;
    const int n0 = NX > 0 ? NX : topo.n[0];
    const int n1 = topo.n[1];
    const int sy = NX > 0 ? NX + 2 : g.L.gdim[0];
    const int lane = threadIdx.x & 31;
    const int wpc = blockDim.x >> 5;

    const int64_t first_listed = (int64_t)gridDim.x * wpc;
    int64_t unit = (int64_t)blockIdx.x * wpc + (threadIdx.x >> 5);
    // what does not depend on the previous step: the first unit's place and
    // its neighbours in the topology
    StripUnit su;
    Nbr2 nb{};
    if (unit < g.units) {
        su.decode(g, unit);
        nb.load(topo, su.b);
    }
    // programmatic dependent launch: wait for the previous step's writes,
    // then let the next step's CTAs become resident
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // Simulation::t lives on the device in two slots: this step reads
    // tdev[slot] (its bits are the Wiener salt, euler_maruyama.rs:73) and
    // writes t + dt to the other slot (simulation.rs:285), so a captured
    // sequence of steps needs no host-side time.
    const double tnow = g.tdev[g.slot];
    if ((MODE == 0 || MODE == 3) && blockIdx.x == 0 && threadIdx.x == 0) {
        g.tdev[g.slot ^ 1] = tnow + g.dt64;
    }

    while (unit < g.units) {
        const int s = su.s, k = su.k, b = su.b;
        // units are g.rows high (whole groups of rows unless TAIL); a block's
        // last unit ends on its last row and may overlap the one before it,
        // whose rows it then recomputes to the same bits
        int r0 = k * g.rows;
        const int rs = r0;  // the unit's own rows start here
        int r1 = r0 + g.rows;
        if (r1 > n1) {
            r1 = n1;
            if (!TAIL) r0 = n1 - g.rows;
        }
        const int c0 = s * 32;
        const int col = c0 + lane;
        const bool valid = FULL || col < n0;
        const int last_lane = min(31, n0 - 1 - c0);
        const int cr = c0 + last_lane;  // last column of the strip; its right face is the boundary face
        const bool edge_x = s == 0 || s == g.strips - 1;

        const T* ph = in + slab_base(g.L, b, 0);
        const T* uu = in + slab_base(g.L, b, 1);
        T* po = out + slab_base(g.L, b, 0);
        T* uo = out + slab_base(g.L, b, 1);
        if constexpr (PAIR) {
            static_assert(!TAIL && !(ORIENT && BATCH), "the paired rows need whole groups");
            if constexpr (BATCH) {
                const int inst = b / bt.bpi;
                const typename Ops::Params mi = static_cast<const typename Ops::Params*>(bt.params)[inst];
                strip_unit_pair<T, Ops, NOISE, NX, FULL, false, MODE>(mi, bt.seeds[inst], b - inst * bt.bpi, g, ph, uu, out, po, uo,
                                                         nb, r0, r1, lane, col, valid, last_lane, cr, edge_x, n0, n1,
                                                         sy, tnow, dt, scale_amp, rs, rk);
            } else {
                const T* trig_b = ORIENT ? static_cast<const T*>(oa.trig) + (int64_t)b * n0 * n1 : nullptr;
                strip_unit_pair<T, Ops, NOISE, NX, FULL, ORIENT, MODE>(m0, g.seed, b, g, ph, uu, out, po, uo, nb, r0, r1,
                                                                 lane, col, valid, last_lane, cr, edge_x, n0, n1, sy,
                                                                 tnow, dt, scale_amp, rs, rk, trig_b, oa.ncells);
            }
        } else if constexpr (BATCH) {
            const int inst = b / bt.bpi;
            const typename Ops::Params mi = static_cast<const typename Ops::Params*>(bt.params)[inst];
            strip_unit<T, Ops, NOISE, NX, FULL, PF, TAIL, ORIENT, MODE>(
                mi, bt.seeds[inst], b - inst * bt.bpi, g, ph, uu, out, po, uo, nb, r0, r1, lane, col, valid, last_lane,
                cr, edge_x, n0, n1, sy, tnow, dt, scale_amp, nullptr, 0, rk, rs);
        } else {
            // multi-grain: this block's cos theta0 (sin theta0 follows ncells later)
            const T* trig_b = ORIENT ? static_cast<const T*>(oa.trig) + (int64_t)b * n0 * n1 : nullptr;
            strip_unit<T, Ops, NOISE, NX, FULL, PF, TAIL, ORIENT, MODE>(m0, g.seed, b, g, ph, uu, out, po, uo, nb,
                                                                        r0, r1, lane, col, valid, last_lane, cr,
                                                                        edge_x, n0, n1, sy, tnow, dt, scale_amp,
                                                                        trig_b, oa.ncells, rk, rs);
        }
        if (g.work) {  // the next unit of the list
            unsigned n = 0;
            if (lane == 0) n = atomicAdd(g.work, 1u);
            unit = first_listed + (int64_t)__shfl_sync(kFull, n, 0);
        } else {
            unit += first_listed;
        }
        if (unit < g.units) {
            su.decode(g, unit);
            nb.load(topo, su.b);
        }
    }
    if (g.work && lane == 0 && atomicAdd(g.work + 1, 1u) == gridDim.x * wpc - 1) {
        g.work[0] = 0u;
        g.work[1] = 0u;
    }
}

// Rows a unit's height is a multiple of: the paired rows step two at a time,
// the unrolled loop (FP32 multi-grain single rows) four.
template <class T, bool ORIENT, bool PAIR>
constexpr int strip_group() {
    return PAIR ? 2 : (sizeof(T) == 4 && ORIENT ? 4 : 1);
}

// Rows per work unit, where the caller leaves them open: of a few heights up
// to 32 (one batch of boundary faces per unit) the one that minimises the
// step's length.  A warp spends about two rows' time on starting a unit, and a
// row's time hardly depends on how many warps share the SM until the resident
// warps (`slots`) are all busy; from there on the units queue.
//
// FP64, and FP32 axis-aligned in one state: powers of two; FP32 rows are short enough to feel the
// queue from about three quarters on.  FP64 paired rows at 2, 4, 8, 16 rows a
// unit: 64^2 4.8, 6.8, 11.0, 19.4 us a step; 512^2 8.6, 8.4, 11.2, 19.5; 1008^2
// 25.0, 21.2, 19.8, 25.1; 2048^2 98, 77, 67, 63.
//
// FP32 multi-grain (TAILED): a single wave runs as fast as its units, but from
// one wave on half a unit's time is spent on the last, partly filled one, so
// heights between the powers of two pay.  With noise at 6, 8, 12, 16, 32 rows:
// 500^2 in blocks of 100^2 9.4, 11.3, 10.5, 12.5, 21.6 us a step; 1500^2 50.3,
// 47.5, 46.8, 53.2, 63.1; 2520^2 (126^2) 95.7, 91.0, 89.5, 84.8, 92.3.  Within
// 1 % of the best height on average over 500^2 to 3072^2, 7 % at most; the
// rule above chose up to 30 % off.
template <class T, bool TAILED>
inline int strip_auto_rows(const CartTopo& topo, int strips, int64_t slots) {
    const int n1 = topo.n[1];
    int best = 2;
    double best_cost = 0.0;
    for (int rows : {32, 24, 20, 16, 12, 10, 8, 6, 4, 2}) {
        if (!TAILED && (rows & (rows - 1)) != 0) continue;
        const int h = std::min(rows, n1);
        const double waves = (double)topo.nblocks * strips * ((n1 + h - 1) / h) / (double)slots;
        const double cost = TAILED ? (h + 1.5) * (waves <= 1.0 ? 1.0 : waves + 0.5)
                                   : (h + 2) * std::max(1.0, (sizeof(T) == 8 ? 1.0 : 1.36) * waves);
        if (best_cost == 0.0 || cost < best_cost) {
            best_cost = cost;
            best = h;
        }
    }
    return best;
}

// work decomposition of a launch: units of (block, strip, row chunk) of
// g.rows rows (at most 32; 0: chosen as above), a whole number of groups of
// nb rows; true when the block is lower than the row group (the TAIL kernels)
template <class T, bool TAILED = false>
inline bool strip_plan(TileArgs& g, int nb, int ctas_per_sm) {
    const int n0 = g.topo.n[0], n1 = g.topo.n[1];
    g.strips = (n0 + 31) / 32;
    const int64_t slots = (int64_t)device_sm_count() * ctas_per_sm * 8;
    int rows = g.rows > 0 ? g.rows : strip_auto_rows<T, TAILED>(g.topo, g.strips, slots);
    rows = std::max(1, std::min(std::min(rows, 32), n1));
    if (n1 >= nb) rows = std::max(nb, rows / nb * nb);
    g.rows = rows;
    g.chunks = (n1 + g.rows - 1) / g.rows;
    g.units = (int64_t)g.topo.nblocks * g.strips * g.chunks;
    // one wave or less needs no list (64^2: 4.8 against 5.1 us a step)
    if (g.units <= slots) g.work = nullptr;
    return n1 < nb;
}

// launch with programmatic dependent launch: consecutive steps overlap one
// step's tail with the next one's start-up (the kernel waits before it
// touches the state)
template <class... P, class... A>
cudaError_t strip_launch(void (*kernel)(P...), dim3 grid, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// CTAs of eight warps: one per eight units, or with a work list one wave
inline dim3 strip_ctas(const TileArgs& g, int ctas_per_sm) {
    const int wpc = 8;
    const int64_t wave = g.work ? (int64_t)device_sm_count() * ctas_per_sm : (int64_t)1 << 30;
    return dim3((unsigned)std::min<int64_t>((g.units + wpc - 1) / wpc, wave));
}

// batched instances: block widths 64 (the ensemble configuration) and 32
// get a compile-time row stride
// PAIR: the paired rows (256 instances of 256^2, FP32: 102.5 against 79.8 Gcell/s)
template <class T, class Ops, bool NOISE, int MINB, bool PAIR = false>
cudaError_t launch_strip_batch(const T* in, T* out, TileArgs g, BatchArgs bt, T dt, T scale_amp, cudaStream_t s) {
    constexpr bool kFixed = sizeof(T) == 4;
    if (kFixed && g.rows <= 0)
        g.rows = strip_batch_rows_f32(g.topo.nblocks, (g.topo.n[0] + 31) / 32, g.topo.n[1], device_sm_count());
    const bool tail = strip_plan<T>(g, kFixed ? 4 : strip_group<T, false, PAIR>(), MINB);
    const dim3 grid = strip_ctas(g, MINB);
    const typename Ops::Params m{};
    if (tail) {
        return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, 1, true, true>, grid, s, in, out, g, m, dt, scale_amp, bt, OrientArgs{}, RkArgs<T>{});
    }
    switch (g.topo.n[0]) {
        case 32: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 32, 1, true, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, bt, OrientArgs{}, RkArgs<T>{});
        case 64: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 64, 1, true, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, bt, OrientArgs{}, RkArgs<T>{});
        default: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, 1, true, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, bt, OrientArgs{}, RkArgs<T>{});
    }
}

template <class T, class Ops, bool NOISE, int MINB, int PF, bool PAIR = false>
cudaError_t launch_strip_minb(const T* in, T* out, TileArgs g, const typename Ops::Params& m, T dt, T scale_amp,
                              cudaStream_t s) {
    const bool tail = strip_plan<T>(g, strip_group<T, false, PAIR>(), MINB);
    const dim3 grid = strip_ctas(g, MINB);
    if (tail) {  // blocks lower than the row group: single rows (the paired form needs whole groups)
        return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, PF, false, true>, grid, s, in, out, g, m, dt, scale_amp, BatchArgs{}, OrientArgs{}, RkArgs<T>{});
    }
    const BatchArgs nob{};
    const OrientArgs noo{};
    const RkArgs<T> nork{};
    switch (g.topo.n[0]) {  // block widths of the shipped configurations get a compile-time row stride
        case 32: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 32, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
        case 64: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 64, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
        case 126: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 126, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
        case 128: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 128, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
        case 256: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 256, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
        default: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, PF, false, false, false, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, nob, noo, nork);
    }
}

// the multi-grain step: block widths 126 (the 101.6M-cell configuration)
// and 256 get a compile-time row stride; PAIR: the paired rows (10080^2
// with 1000 grains: FP64 37.6 against 36.4, FP32 81.7 against 77.0
// Gcell/s)
template <class T, class Ops, bool NOISE, int MINB, bool PAIR = false>
cudaError_t launch_strip_oriented(const T* in, T* out, TileArgs g, const typename Ops::Params& m, T dt, T scale_amp,
                                  OrientArgs oa, cudaStream_t s) {
    const bool tail = strip_plan<T, sizeof(T) == 4>(g, strip_group<T, true, PAIR>(), MINB);
    const dim3 grid = strip_ctas(g, MINB);
    if (tail) {  // blocks lower than the row group: single rows
        return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, 1, false, true, true>, grid, s, in, out, g, m, dt, scale_amp, BatchArgs{}, oa, RkArgs<T>{});
    }
    switch (g.topo.n[0]) {
        case 126: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 126, 1, false, false, true, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, BatchArgs{}, oa, RkArgs<T>{});
        case 256: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 256, 1, false, false, true, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, BatchArgs{}, oa, RkArgs<T>{});
        default: return strip_launch(modelc_strip_kernel<T, Ops, NOISE, MINB, 0, 1, false, false, true, 0, PAIR>, grid, s, in, out, g, m, dt, scale_amp, BatchArgs{}, oa, RkArgs<T>{});
    }
}

// RungeKutta4 stages of Model C (deterministic: no noise), axis-aligned or
// multi-grain, on the paired rows; the block widths of the Euler-Maruyama step
// get a compile-time row stride here too (2048^2 in blocks of 32, 64, 126, 128
// and 256 columns 5 to 7 % faster than without in FP64, 5 to 13 % in FP32)
template <class T, class Ops, int MODE, bool ORIENT>
cudaError_t launch_strip_rk(const T* in, T* out, TileArgs g, const typename Ops::Params& m, T dt, OrientArgs oa,
                            RkArgs<T> rk, cudaStream_t s) {
    const bool tail = strip_plan<T>(g, strip_group<T, ORIENT, true>(), 2);
    const dim3 grid = strip_ctas(g, 2);
    const BatchArgs nob{};
    if (tail)  // blocks of one row
        return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 0, 1, false, true, ORIENT, MODE>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
    switch (g.topo.n[0]) {
        case 32: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 32, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
        case 64: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 64, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
        case 126: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 126, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
        case 128: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 128, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
        case 256: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 256, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
        default: return strip_launch(modelc_strip_kernel<T, Ops, false, 2, 0, 1, false, false, ORIENT, MODE, true>, grid, s, in, out, g, m, dt, T(0), nob, oa, rk);
    }
}

// kind 2/3/4: single rows, CTAs of 256 threads per SM the register
// allocation must allow (2: up to 128 registers, 3: 80, 4: 64); kind 5/6/7:
// the paired rows (strip_unit_pair) at 2/3/4 CTAs per SM.
// PF: rows of prefetch ahead of the row being computed
template <class T, class Ops, bool NOISE, int PF>
cudaError_t launch_strip_ops(const T* in, T* out, TileArgs g, const typename Ops::Params& m, T dt, T scale_amp,
                             int kind, cudaStream_t s) {
    switch (kind) {
        case 3: return launch_strip_minb<T, Ops, NOISE, 3, PF>(in, out, g, m, dt, scale_amp, s);
        case 4: return launch_strip_minb<T, Ops, NOISE, 4, PF>(in, out, g, m, dt, scale_amp, s);
        case 5: return launch_strip_minb<T, Ops, NOISE, 2, PF, true>(in, out, g, m, dt, scale_amp, s);
        case 6: return launch_strip_minb<T, Ops, NOISE, 3, PF, true>(in, out, g, m, dt, scale_amp, s);
        case 7: return launch_strip_minb<T, Ops, NOISE, 4, PF, true>(in, out, g, m, dt, scale_amp, s);
        default: return launch_strip_minb<T, Ops, NOISE, 2, PF>(in, out, g, m, dt, scale_amp, s);
    }
}

}  // namespace lg
