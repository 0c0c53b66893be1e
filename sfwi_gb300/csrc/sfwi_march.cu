// sfwi_march.cu — whole time steps in one launch.
//
// A time step is a velocity and a stress sweep (sfwi_kernels.cu runs each as a
// launch of its own).  Here one launch runs both: a CTA takes an item, a strip
// of up to PC columns and a run of rows of one shot, and marches along x four
// rows (a group) at a time.  The first half-step's results of the last rows
// stay in shared memory, where the second half-step, which lags one group
// behind, differentiates them; nothing is exchanged between CTAs.
//
//   k_march_fwd   v' = v-sweep(v, sigma), sigma' = s-sweep(sigma, v'), background
//                 and scattered field (k_fwd_v + k_fwd_s)
//   k_march_bwd   sigma = s-sweep of the reconstruction and the adjoint, imaging,
//                 v = v-sweep of both (k_bwd_s + k_bwd_v); without PAIR the
//                 adjoint alone (snapshot runs: k_bwd_s_snap + k_bwd_v_snap)
//   k_snap_store, k_snap_image   the snapshot of a forward step, and the imaging
//                 of a backward step from its snapshot
//
// What bounds it: bytes, and the instructions that each cell takes.  The two
// sweeps of a Born forward step move 60 + 80 algorithmic bytes per cell, a
// step that reads every field once 100; the backward step 116 against 88 + 76.
// The price is the first half-step on a rim 4 cells wide around each item,
// recomputed by its neighbours, so an item's rows are long (a wave of items
// covers the batch) and its strip as wide as shared memory allows.  A CTA
// reads its rows through rings of four groups in shared memory filled by TMA
// one group ahead.
//
// State.  Neighbouring items read the fields that an item advances, so a step
// reads one copy of the totals and x-parts and writes the other; the imaging
// accumulators belong to one item each and are updated in place.  Two fields
// that advance together (background and scattered, reconstruction and adjoint) are
// stored as pairs, float2 per cell: every FP32x2 instruction then takes one
// cell of both, with no shuffling for the odd offsets of the z-derivatives.
// A single field (stage 1's forward, the adjoint alone) is stored plainly and two
// columns make the lanes.  The arithmetic is that of sfwi_cell.cuh, in the
// sweeps' order: a run gives the sweeps' bits.
#include <algorithm>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sfwi_cell.cuh"
#include "sfwi_launch.h"
#include "sfwi_pipe.cuh"

namespace sfwi {
namespace {

constexpr int G = G_ROWS;

__device__ __forceinline__ float2 ld2s(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ float2 ld2g(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void st2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ float2 sel(bool a, bool b, float2 x, float2 y) {
    return make_float2(a ? x.x : y.x, b ? x.y : y.y);
}

extern __shared__ __align__(1024) unsigned char march_smem[];
__device__ __forceinline__ float *smem() {
    // TMA destinations start on 128-byte boundaries
    return reinterpret_cast<float *>(march_smem + ((128 - (smem_u32(march_smem) & 127)) & 127));
}

// ---------------------------------------------------------------------------
// lanes: a thread's two adjacent columns of one row.  PAIR: two lanes, one per
// column, each both fields of the cell; else one lane, the two columns.
// ---------------------------------------------------------------------------
template <bool PAIR>
struct Lanes {
    static constexpr int N = PAIR ? 2 : 1;
    float2 v[N];
    __device__ __forceinline__ float2 &operator[](int i) { return v[i]; }
    __device__ __forceinline__ const float2 &operator[](int i) const { return v[i]; }
};
template <bool PAIR>
__device__ __forceinline__ Lanes<PAIR> ldl(const float *p) {
    Lanes<PAIR> o;
    if constexpr (PAIR) {
        const float4 a = ld4(p);
        o[0] = make_float2(a.x, a.y);
        o[1] = make_float2(a.z, a.w);
    } else {
        o[0] = ld2s(p);
    }
    return o;
}
template <bool PAIR>
__device__ __forceinline__ void stl(float *p, const Lanes<PAIR> &o) {
    if constexpr (PAIR)
        st4(p, make_float4(o[0].x, o[0].y, o[1].x, o[1].y));
    else
        st2(p, o[0]);
}
template <bool PAIR>
__device__ __forceinline__ Lanes<PAIR> zero_lanes() {
    Lanes<PAIR> o;
#pragma unroll
    for (int l = 0; l < Lanes<PAIR>::N; l++) o[l] = make_float2(0.f, 0.f);
    return o;
}
// a per-column value (c: the two columns) in the lanes
template <bool PAIR>
__device__ __forceinline__ float2 lane_of(float2 c, int l) {
    if constexpr (PAIR)
        return B2(l ? c.y : c.x);
    else
        return c;
}
// x where the column's mask holds, y elsewhere
template <bool PAIR>
__device__ __forceinline__ float2 pick(int l, bool m0, bool m1, float2 x, float2 y) {
    if constexpr (PAIR)
        return sel(l ? m1 : m0, l ? m1 : m0, x, y);
    else
        return sel(m0, m1, x, y);
}
// first field of the two columns (background, reconstruction, or the only one)
template <bool PAIR>
__device__ __forceinline__ float2 first_of(const Lanes<PAIR> &o) {
    if constexpr (PAIR)
        return make_float2(o[0].x, o[1].x);
    else
        return o[0];
}

// Offsets (floats) in a ring of the rows that the stencils of a thread's R rows
// reach: rows R ch - 4 .. R ch + R + 3 of group k, ch the thread's part of the group
template <int R>
struct RowOff {
    int o[R + 8];
};
template <int NSLOT, int SLOT, int PITCH, int R>
__device__ __forceinline__ RowOff<R> row_off(int k, int ch) {
    // the rows before, in and after group k, each as if it were the whole ring
    const int r0 = R * ch;
    const int a = ((k - 1) & (NSLOT - 1)) * SLOT + r0 * PITCH, b = (k & (NSLOT - 1)) * SLOT + (r0 - 4) * PITCH,
              c = ((k + 1) & (NSLOT - 1)) * SLOT + (r0 - 8) * PITCH;
    RowOff<R> r;
#pragma unroll
    for (int i = 0; i < R + 8; i++) r.o[i] = (i + r0 < 4 ? a : i + r0 < 8 ? b : c) + i * PITCH;
    return r;
}

// x-derivatives of the thread's columns on its R rows:
// D+x: sum_k K_k (f[r+k] - f[r-k+1]), D-x: sum_k K_k (f[r+k-1] - f[r-k])
template <bool PAIR, bool PLUS, int R>
__device__ __forceinline__ void ddx(const float *f, const RowOff<R> &ro, Lanes<PAIR> (&o)[R]) {
    Lanes<PAIR> w[R + 7];
#pragma unroll
    for (int i = 0; i < R + 7; i++) w[i] = ldl<PAIR>(f + ro.o[i + (PLUS ? 1 : 0)]);
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int l = 0; l < Lanes<PAIR>::N; l++) {
            float2 t = make_float2(0.f, 0.f);
            t = kdiff2(K1, w[i + 4][l], w[i + 3][l], t);
            t = kdiff2(K2, w[i + 5][l], w[i + 2][l], t);
            t = kdiff2(K3, w[i + 6][l], w[i + 1][l], t);
            t = kdiff2(K4, w[i + 7][l], w[i][l], t);
            o[i][l] = t;
        }
}
// z-derivatives of the thread's columns (q: its first column in the row)
template <bool PAIR, bool PLUS>
__device__ __forceinline__ Lanes<PAIR> ddz(const float *q) {
    constexpr int S = PLUS ? 0 : -1;
    Lanes<PAIR> o;
    if constexpr (PAIR) {
        float2 w[10];
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const Lanes<true> v = ldl<true>(q + 4 * (i - 2));
            w[2 * i] = v[0];
            w[2 * i + 1] = v[1];
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = 4 + j + S;
            float2 t = make_float2(0.f, 0.f);
            t = kdiff2(K1, w[c + 1], w[c], t);
            t = kdiff2(K2, w[c + 2], w[c - 1], t);
            t = kdiff2(K3, w[c + 3], w[c - 2], t);
            t = kdiff2(K4, w[c + 4], w[c - 3], t);
            o[j] = t;
        }
    } else {
        float w[10], d[2];
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const float2 v = ld2s(q + 2 * (i - 2));
            w[2 * i] = v.x;
            w[2 * i + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int c = 4 + j + S;
            float t = 0.f;
            t = kdiff2(K1, w[c + 1], w[c], t);
            t = kdiff2(K2, w[c + 2], w[c - 1], t);
            t = kdiff2(K3, w[c + 3], w[c - 2], t);
            t = kdiff2(K4, w[c + 4], w[c - 3], t);
            d[j] = t;
        }
        o[0] = make_float2(d[0], d[1]);
    }
    return o;
}

// ---------------------------------------------------------------------------
// where a thread's cells lie
// ---------------------------------------------------------------------------
struct Geo {
    int row0, nxpml, nzpml, pml, P, x0, x1, z0, zw;
};
// the two columns of a thread in one half-step, fixed for the march
struct Cols {
    // bits of f: the columns lie in the boxes; inside the update region; damped along
    // z; the item writes them; (backward) inside the imaging interior; over the
    // warp: no column of use inside the region; none damped, at an edge or special
    enum { ACTIVE = 1, OK0 = 2, OK1 = 4, SZ0 = 8, SZ1 = 16, OWN = 32, IM0 = 64, IM1 = 128, NONE = 256, PLAIN = 512 };
    int z, col;  // the first column, in the shot and in the half-step's boxes (0 where inactive)
    unsigned f;
    __device__ __forceinline__ bool is(unsigned m) const { return f & m; }
};
// columns z0 + col of a half-step whose boxes have ncol columns, of which those
// before `end` are of use
__device__ __forceinline__ Cols cols_at(const Geo &g, int z0, int col, int ncol, int end) {
    Cols c;
    const bool active = col < ncol;
    c.col = active ? col : 0;
    const int z = c.z = z0 + c.col;
    const bool ok0 = active && z >= NOP && z < g.nzpml - NOP, ok1 = active && z >= NOP && z + 1 < g.nzpml - NOP;
    const bool sz0 = ok0 && (z < g.pml || z > g.nzpml - g.pml);
    const bool sz1 = ok1 && (z + 1 < g.pml || z + 1 > g.nzpml - g.pml);
    const bool own = ok0 && z >= g.z0 && z < g.z0 + g.zw;
    auto in = [&](int w) { return own && w >= g.pml && w < g.nzpml - g.pml; };
    const unsigned all = 0xffffffffu;
    const bool none = !__any_sync(all, active && z >= NOP && z < end), plain = !__any_sync(all, active && (!ok1 || sz0 || sz1));
    c.f = active * Cols::ACTIVE | ok0 * Cols::OK0 | ok1 * Cols::OK1 | sz0 * Cols::SZ0 | sz1 * Cols::SZ1 |
          own * Cols::OWN | in(z) * Cols::IM0 | in(z + 1) * Cols::IM1 | none * Cols::NONE | plain * Cols::PLAIN;
    return c;
}
// no warp of special columns takes the LEAN form
__device__ __forceinline__ void special(Cols &c, bool any) {
    if (__any_sync(0xffffffffu, any)) c.f &= ~Cols::PLAIN;
}
// A half-step has three forms, and each warp picks one for its rows of a group:
//   LEAN   no cell damped, none that strips, receivers or the source touch
//   INNER  rows away from the PML and the strips along x, any columns
//   EDGE   any cells
// Most cells are LEAN's, whose instructions are little more than the stencils'
// and the update's.
enum Form { LEAN, INNER, EDGE };
// rows [lx0, lx0 + G) of a shot: away from the PML and the strips along x
__device__ __forceinline__ bool inner_rows(const Geo &g, int lx0) {
    return lx0 >= g.pml + NOP && lx0 + G <= g.nxpml - g.pml - NOP;
}
// a row
struct Row {
    int lx;
    bool ok, xd, own;
};
__device__ __forceinline__ Row row_at(const Geo &g, int lx) {
    return Row{lx, lx >= NOP && lx < g.nxpml - NOP, lx < g.pml || lx > g.nxpml - g.pml, lx >= g.x0 && lx < g.x1};
}
// PML factors 1 -+ (dt d)/2 and reciprocals of a thread's columns, from the
// factor arrays (fx: d1, r2 and fz: d3, r4 per cell); x: ones unless the row is
// damped along x
__device__ __forceinline__ void load_damp(const MarchArgs &a, unsigned i, bool xd, float4 &x, float4 &z) {
    if (xd) x = ld4(a.fx + 2 * (size_t)i);
    z = ld4(a.fz + 2 * (size_t)i);
}
template <bool PAIR>
__device__ __forceinline__ Damp2 lane_damp(const float4 &x, const float4 &z, int l) {
    return Damp2{lane_of<PAIR>(make_float2(x.x, x.z), l), lane_of<PAIR>(make_float2(x.y, x.w), l),
                 lane_of<PAIR>(make_float2(z.x, z.z), l), lane_of<PAIR>(make_float2(z.y, z.w), l)};
}

// A wait ran out: the copies in flight must land before the CTA leaves its
// shared memory.  Thread 0 waits for those of step t, which others waited for,
// thread 32 for those of step t + 1, if there is one.  (PIPE_WAIT_LIMIT whatever
// the bound of the wait that ran out was.  One thread waiting for both made the
// compiler's allocation of the Born march's registers 4 % slower, 92.5 -> 96.5 us.)
__device__ __forceinline__ void give_up(const Params &p, uint64_t (&full)[2], int t, int K) {
    const int tid = threadIdx.x;
    if ((tid & 31) == 0 && tid < 64 && t + (tid >> 5) < K) {
        atomicExch(p.err, 1);
        const int j = t + (tid >> 5);
        mbar_wait(&full[j & 1], ((j - 2) >> 1) & 1, PIPE_WAIT_LIMIT);
    }
}

struct Item {
    MarchItem m;
    Geo g;
    int K;    // groups: the item's rows and two more at either end
    int row;  // packed row of group 0
};
__device__ __forceinline__ Item load_item(const Params &p, const MarchItem *items) {
    Item it;
    const int4 *src = reinterpret_cast<const int4 *>(items + blockIdx.x);
    int4 w[sizeof(MarchItem) / 16];
#pragma unroll
    for (int i = 0; i < (int)(sizeof(MarchItem) / 16); i++) w[i] = __ldg(src + i);
    it.m = *reinterpret_cast<const MarchItem *>(w);
    it.g = Geo{it.m.g.row0, it.m.g.nxpml, it.m.g.nzpml, p.pml, p.P, it.m.x0, it.m.x1, it.m.z0, it.m.zw};
    it.K = (it.m.x1 - it.m.x0 + G - 1) / G + 4;
    it.row = it.m.g.row0 + it.m.x0 - 2 * G;
    return it;
}

// ---------------------------------------------------------------------------
// forward step
// ---------------------------------------------------------------------------
// Common to the two steps.  An item is worked on in one of two ways:
// marching, group by group through rings of four slots (three in use, one on
// its way; two for what only one half-step of a group reads), or, for small
// batches (BURST), all at once: every group of a short item has its slot, the
// warps share out the groups, and a step is one wait for the loads and one
// barrier between the half-steps.
template <int PS_, bool PAIR_, bool BURST_>
struct StepCfg {
    static constexpr bool PAIR = PAIR_, BURST = BURST_;
    static constexpr int E = PAIR ? 2 : 1;
    static constexpr int PS = PS_, PV = PS - 8, PC = PS - 16;  // columns of the view, the rim, the core
    static constexpr int NSLOT = BURST ? 8 : 4, CSLOT = BURST ? 8 : 2;
    // a warp takes all rows of a group in 16 columns (pairs) or 32, so few
    // warps hold the PML columns; a thread takes two columns of R rows
    static constexpr int R = PAIR ? 1 : 2, LPR = 32 * R / G;  // lanes of a row
    static constexpr int BLOCKS = PV / (2 * LPR);             // warps that cover the rim's columns
    static constexpr int NT = BURST ? 512 : 32 * BLOCKS;
};
template <int PS_, bool PAIR_, bool BURST_>
struct FwdCfg : StepCfg<PS_, PAIR_, BURST_> {
    using B = StepCfg<PS_, PAIR_, BURST_>;
    using B::E, B::PS, B::PV, B::PC, B::NSLOT, B::CSLOT, B::NT;
    static constexpr int ASIG = G * PS * E, AVEL = G * PV * E;  // floats of one array of a group
    static constexpr int SIG = 3 * ASIG, VEL = 2 * AVEL, IB = G * PV, CO = (PAIR_ ? 4 : 2) * G * PC;
    static constexpr int O_VEL = NSLOT * SIG, O_IB = O_VEL + NSLOT * VEL, O_CO = O_IB + CSLOT * IB;
    static constexpr int FLOATS = O_CO + CSLOT * CO;
    static constexpr size_t BYTES = (size_t)FLOATS * 4 + 128;
    static constexpr int FIT = (int)(228 * 1024 / (BYTES + 1024 + 64));
    static constexpr int CTAS = FIT > 512 / NT ? 512 / NT : FIT;
};

template <class C, bool SNAP>
struct FwdBody {
    static constexpr bool PAIR = C::PAIR;
    static constexpr int N = Lanes<PAIR>::N, E = C::E, R = C::R;
    using L = Lanes<PAIR>;
    const MarchArgs &a;
    const Item &im;
    float *sm;
    int it, ch;
    Cols vc, sc;        // columns of the velocity (rim) and the stress (core) half-step
    bool strip_z;       // a lane of the warp has columns in a top/bottom strip
    unsigned max_x = 0, max_z = 0;

    __device__ __forceinline__ FwdBody(const MarchArgs &a_, const Item &im_, float *sm_, int it_)
        : a(a_), im(im_), sm(sm_), it(it_) {
        const Geo &g = im.g;
        const int cp = (threadIdx.x >> 5) % C::BLOCKS * C::LPR + threadIdx.x % C::LPR;
        ch = (threadIdx.x & 31) / C::LPR;
        vc = cols_at(g, g.z0 - NOP, 2 * cp, C::PV, im.m.vend);
        sc = cols_at(g, g.z0, 2 * cp, C::PC, g.z0 + g.zw);
        const int d0 = vc.z - (g.pml - NOP), d1 = vc.z - (g.nzpml - g.pml - NOP);
        strip_z = __any_sync(0xffffffffu, vc.is(Cols::OWN) && ((d0 >= -1 && d0 < 2 * NOP) ||
                                                               (d1 >= -1 && d1 < 2 * NOP)));
        const bool src = im.m.flags & MARCH_SOURCE;
        auto holds = [](int z, int w) { return w == z || w == z + 1; };
        special(vc, strip_z || holds(vc.z, im.m.g.igz) || (src && holds(vc.z, im.m.g.isz)));
        special(sc, src && holds(sc.z, im.m.g.isz));
    }

    // the thread's rows of group k: new velocities into the ring (zero outside
    // the update region) and, where the item owns them, into memory
    __device__ __forceinline__ void velocity(int k) {
        const int g0 = im.g.x0 - 2 * G + G * k, lx0 = g0 + R * ch;
        if (vc.is(Cols::NONE)) return;
        if (!inner_rows(im.g, g0))
            velocity<EDGE>(k, lx0);
        else if (vc.is(Cols::PLAIN))
            velocity<LEAN>(k, lx0);
        else
            velocity<INNER>(k, lx0);
    }
    template <Form F>
    __device__ __forceinline__ void velocity(int k, int lx0) {
        const Params &p = a.p;
        const Geo &g = im.g;
        const FieldSet &in = a.in_bg, &out = p.bg;
        const int cv = vc.col;
        const unsigned o0 = (unsigned)((g.row0 + lx0) * g.P + vc.z);
        L mx[R], mz[R];
        float4 fx[R], fz[R];
        if constexpr (F != LEAN) {
#pragma unroll
            for (int i = 0; i < R; i++) {
                const Row r = row_at(g, lx0 + i);
                const bool xd = F == EDGE && r.xd;
                mx[i] = mz[i] = zero_lanes<PAIR>();
                fx[i] = fz[i] = make_float4(a.one, a.one, a.one, a.one);
                if ((F == INNER || r.ok) && vc.is(Cols::OK0) && (xd || vc.is(Cols::SZ0 | Cols::SZ1))) {
                    const size_t o = o0 + i * g.P;
                    load_damp(a, o, xd, fx[i], fz[i]);
                    mx[i] = ldl<PAIR>(in.mvx + o * E);
                    mz[i] = ldl<PAIR>(in.mvz + o * E);
                    if (!C::BURST && r.lx + G < g.nxpml) {
                        // the next group's, while this one is computed
                        const size_t n = o + G * g.P;
                        prefetch_l2(a.fz + 2 * n);
                        if (xd) prefetch_l2(a.fx + 2 * n);
                        prefetch_l2(in.mvx + n * E);
                        prefetch_l2(in.mvz + n * E);
                    }
                }
            }
        }
        const RowOff<R> ro = row_off<C::NSLOT, C::SIG, C::PS * E, R>(k, ch);
        const float *sig = sm + (cv + NOP) * E;
        L ax[R], dx[R], bz[R], dz[R];
        ddx<PAIR, true>(sig, ro, ax);
        ddx<PAIR, false>(sig + 2 * C::ASIG, ro, dx);
#pragma unroll
        for (int i = 0; i < R; i++) {
            bz[i] = ddz<PAIR, false>(sig + 2 * C::ASIG + ro.o[i + 4]);
            dz[i] = ddz<PAIR, true>(sig + C::ASIG + ro.o[i + 4]);
        }
        float *vel = sm + C::O_VEL + (k & (C::NSLOT - 1)) * C::VEL + (R * ch * C::PV + cv) * E;
        const float *ib = sm + C::O_IB + (k & (C::CSLOT - 1)) * C::IB + R * ch * C::PV + cv;
        const float2 tx = B2(p.dtdx), tz = B2(p.dtdz);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const bool row_ok = F != EDGE || r.ok, xd = F == EDGE && r.xd;
            const bool own = r.own && vc.is(Cols::OWN) && row_ok;
            const size_t o = o0 + i * g.P;
            const L ox = ldl<PAIR>(vel + i * C::PV * E), oz = ldl<PAIR>(vel + C::AVEL + i * C::PV * E);
            const float2 ic = ld2s(ib + i * C::PV);
            L vx, vz;
            float2 cx[N], cz[N];
#pragma unroll
            for (int l = 0; l < N; l++) {
                const float2 i2 = lane_of<PAIR>(ic, l);
                cx[l] = mul2(i2, tx), cz[l] = mul2(i2, tz);
                vx[l] = v_plain1(ox[l], cx[l], cz[l], ax[i][l], bz[i][l]);
                vz[l] = v_plain1(oz[l], cx[l], cz[l], dx[i][l], dz[i][l]);
            }
            const bool k1 = row_ok && vc.is(Cols::OK1);
            if constexpr (F != LEAN) {
                {
                    const bool s0 = row_ok && vc.is(Cols::OK0) && (xd || vc.is(Cols::SZ0));
                    const bool s1 = row_ok && vc.is(Cols::OK1) && (xd || vc.is(Cols::SZ1));
                    L nx, nz;
#pragma unroll
                    for (int l = 0; l < N; l++) {
                        const Damp2 d = lane_damp<PAIR>(fx[i], fz[i], l);
                        float2 x = mx[i][l], z = mz[i][l];
                        const float2 tx_ = v_split1(ox[l], x, d, cx[l], cz[l], ax[i][l], bz[i][l]);
                        const float2 tz_ = v_split1(oz[l], z, d, cx[l], cz[l], dx[i][l], dz[i][l]);
                        vx[l] = pick<PAIR>(l, s0, s1, tx_, vx[l]);
                        vz[l] = pick<PAIR>(l, s0, s1, tz_, vz[l]);
                        nx[l] = pick<PAIR>(l, s0, s1, x, mx[i][l]);
                        nz[l] = pick<PAIR>(l, s0, s1, z, mz[i][l]);
                    }
                    if (own && (s0 || s1)) {
                        stl<PAIR>(out.mvx + o * E, nx);
                        stl<PAIR>(out.mvz + o * E, nz);
                    }
                }
                const bool k0 = row_ok && vc.is(Cols::OK0);
#pragma unroll
                for (int l = 0; l < N; l++) {
                    vx[l] = pick<PAIR>(l, k0, k1, vx[l], make_float2(0.f, 0.f));
                    vz[l] = pick<PAIR>(l, k0, k1, vz[l], make_float2(0.f, 0.f));
                }
            }
            if (own) {
                stl<PAIR>(out.vx + o * E, vx);
                stl<PAIR>(out.vz + o * E, vz);
            }
            // a vertical force enters the total vz after this half-step: the
            // stress half-step, the records, the strips and the snapshot of
            // this step see it
            if (F != LEAN && (im.m.flags & MARCH_SOURCE) && p.src_kind == SRC_VZ_FORCE && r.lx == im.m.g.isx) {
                if (vc.z == im.m.g.isz) vz[0].x += p.sou[it];
                if (vc.z + 1 == im.m.g.isz) (PAIR ? vz[N - 1].x : vz[0].y) += p.sou[it];
            }
            if (vc.is(Cols::ACTIVE)) {
                stl<PAIR>(vel + i * C::PV * E, vx);
                stl<PAIR>(vel + C::AVEL + i * C::PV * E, vz);
            }
            if ((F != LEAN || SNAP) && own) {
                const float2 bx = first_of<PAIR>(vx), bz_ = first_of<PAIR>(vz);
                if constexpr (F != LEAN) {
                    const int dr = im.m.g.igz - vc.z;
                    if (dr == 0 || dr == 1) {
                        // receiver row: vz, vx (of the scattered field, then of the background)
                        float *rr = p.rrow + (size_t)it * p.nrc * p.X + g.row0 + r.lx;
                        if constexpr (PAIR) {
                            rr[0] = dr ? vz[N - 1].y : vz[0].y;
                            rr[p.X] = dr ? vx[N - 1].y : vx[0].y;
                            rr += 2 * (size_t)p.X;
                        }
                        rr[0] = dr ? bz_.y : bz_.x;
                        rr[p.X] = dr ? bx.y : bx.x;
                    }
                    if (p.tb) save_strips<F>(r.lx, bx, bz_);
                }
                if (SNAP) {
                    max_x = max(max_x, max(__float_as_uint(fabsf(bx.x)), k1 ? __float_as_uint(fabsf(bx.y)) : 0u));
                    max_z = max(max_z, max(__float_as_uint(fabsf(bz_.x)), k1 ? __float_as_uint(fabsf(bz_.y)) : 0u));
                }
            }
        }
    }
    // edge strips of the background velocity after this step
    template <Form F>
    __device__ __forceinline__ void save_strips(int lx, float2 vx, float2 vz) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const int sit = it % p.strip_steps, z = vc.z;
        if (strip_z && (F == INNER || (lx >= g.pml && lx < g.nxpml - g.pml))) {
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const int d = z - (b == 0 ? g.pml - NOP : g.nzpml - g.pml - NOP);
                if (d >= -1 && d < 2 * NOP) {
                    float *tx = p.tb + tb_row(sit, 0, b, p.X, g.row0 + lx) * 8;
                    float *tz = p.tb + tb_row(sit, 1, b, p.X, g.row0 + lx) * 8;
                    if (d >= 0) tx[d] = vx.x, tz[d] = vz.x;
                    if (d + 1 < 2 * NOP) tx[d + 1] = vx.y, tz[d + 1] = vz.y;
                }
            }
        }
        if (F == INNER) return;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int r = lx - (b == 0 ? g.pml - NOP : g.nxpml - g.pml - NOP);
            if (r >= 0 && r < 2 * NOP) {
                float *px = p.lr + lr_row(sit, 0, b, p.nshots, im.m.shot, r) * p.P;
                float *pz = p.lr + lr_row(sit, 1, b, p.nshots, im.m.shot, r) * p.P;
                if (z >= g.pml && z < g.nzpml - g.pml) px[z] = vx.x, pz[z] = vz.x;
                if (z + 1 >= g.pml && z + 1 < g.nzpml - g.pml) px[z + 1] = vx.y, pz[z + 1] = vz.y;
            }
        }
    }
    // scale of this step's snapshot: max |v| over the shot (the bits of
    // non-negative floats order as unsigned integers)
    __device__ __forceinline__ void snap_scale() const {
        const Params &p = a.p;
        const unsigned rx = __reduce_max_sync(0xffffffffu, max_x), rz = __reduce_max_sync(0xffffffffu, max_z);
        if ((threadIdx.x & 31) == 0) {
            unsigned *sc = reinterpret_cast<unsigned *>(p.sscale) +
                           ((size_t)im.m.shot * p.nsnap + it / p.snap_every) * 2;
            if (rx) atomicMax(sc, rx);
            if (rz) atomicMax(sc + 1, rz);
        }
    }

    // the thread's rows of group k: the new stresses
    __device__ __forceinline__ void stress(int k, const float *src_old) const {
        const int g0 = im.g.x0 - 2 * G + G * k, lx0 = g0 + R * ch;
        if (sc.is(Cols::NONE)) return;
        if (!inner_rows(im.g, g0))
            stress<EDGE>(k, lx0, src_old);
        else if (sc.is(Cols::PLAIN))
            stress<LEAN>(k, lx0, src_old);
        else
            stress<INNER>(k, lx0, src_old);
    }
    template <Form F>
    __device__ __forceinline__ void stress(int k, int lx0, const float *src_old) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const FieldSet &in = a.in_bg, &out = p.bg;
        const int cs = sc.col;
        const unsigned o0 = (unsigned)((g.row0 + lx0) * g.P + sc.z);
        L mxx[R], mzz[R], mxz[R];
        float4 fx[R], fz[R];
        if constexpr (F != LEAN) {
#pragma unroll
            for (int i = 0; i < R; i++) {
                const Row r = row_at(g, lx0 + i);
                const bool xd = F == EDGE && r.xd;
                mxx[i] = mzz[i] = mxz[i] = zero_lanes<PAIR>();
                fx[i] = fz[i] = make_float4(a.one, a.one, a.one, a.one);
                if ((F == INNER || r.ok) && r.own && sc.is(Cols::OWN) && (xd || sc.is(Cols::SZ0 | Cols::SZ1))) {
                    const size_t o = o0 + i * g.P;
                    load_damp(a, o, xd, fx[i], fz[i]);
                    mxx[i] = ldl<PAIR>(in.mtxx + o * E);
                    mzz[i] = ldl<PAIR>(in.mtzz + o * E);
                    mxz[i] = ldl<PAIR>(in.mtxz + o * E);
                    if (!C::BURST && r.lx + G < g.nxpml) {
                        const size_t n = o + G * g.P;
                        prefetch_l2(in.mtxx + n * E);
                        prefetch_l2(in.mtzz + n * E);
                        prefetch_l2(in.mtxz + n * E);
                    }
                }
            }
        }
        const RowOff<R> ro = row_off<C::NSLOT, C::VEL, C::PV * E, R>(k, ch);
        const float *vel = sm + C::O_VEL + (cs + NOP) * E;
        L av[R], bv[R], cv[R], dv[R];
        ddx<PAIR, false>(vel, ro, av);
        ddx<PAIR, true>(vel + C::AVEL, ro, dv);
#pragma unroll
        for (int i = 0; i < R; i++) {
            cv[i] = ddz<PAIR, true>(vel + ro.o[i + 4]);
            bv[i] = ddz<PAIR, false>(vel + C::AVEL + ro.o[i + 4]);
        }
        const float *sig = sm + (k & (C::NSLOT - 1)) * C::SIG + (R * ch * C::PS + cs + 2 * NOP) * E;
        const float2 tx = B2(p.dtdx), tz = B2(p.dtdz);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const bool row_ok = F != EDGE || r.ok, xd = F == EDGE && r.xd;
            const bool own = row_ok && r.own && sc.is(Cols::OWN);
            const size_t o = o0 + i * g.P;
            L xx = ldl<PAIR>(sig + i * C::PS * E), zz = ldl<PAIR>(sig + C::ASIG + i * C::PS * E),
              xz = ldl<PAIR>(sig + 2 * C::ASIG + i * C::PS * E);
            if (F != LEAN && (im.m.flags & MARCH_SOURCE) && p.src_kind == SRC_TXX_TZZ && r.lx == im.m.g.isx) {
                // the source was added to the velocity half-step's view only
                if (sc.z == im.m.g.isz) xx[0].x = src_old[0], zz[0].x = src_old[1];
                if (sc.z + 1 == im.m.g.isz) {
                    (PAIR ? xx[N - 1].x : xx[0].y) = src_old[0];
                    (PAIR ? zz[N - 1].x : zz[0].y) = src_old[1];
                }
            }
            float2 lc, uc, bp, bs;  // per column: lambda, mu, and the Born coefficients
            coefs(k, i, cs, lc, uc, bp, bs);
            Born2 q;  // lanes: the two columns
            L n[3] = {xx, zz, xz};
            if constexpr (PAIR) {
                // the scattered field takes the Born increments
                q = born2<float2>(bp, bs, p.idx, p.idz, p.dt, first_of<PAIR>(av[i]), first_of<PAIR>(bv[i]),
                                  first_of<PAIR>(cv[i]), first_of<PAIR>(dv[i]));
                n[0][0].y = add2(xx[0].y, q.xx.x), n[0][N - 1].y = add2(xx[N - 1].y, q.xx.y);
                n[1][0].y = add2(zz[0].y, q.zz.x), n[1][N - 1].y = add2(zz[N - 1].y, q.zz.y);
                n[2][0].y = add2(xz[0].y, q.xz.x), n[2][N - 1].y = add2(xz[N - 1].y, q.xz.y);
            }
#pragma unroll
            for (int l = 0; l < N; l++) {
                const float2 lam = lane_of<PAIR>(lc, l), mu = lane_of<PAIR>(uc, l);
                s_norm_plain(n[0][l], n[1][l], tx, tz, lam, mu, av[i][l], bv[i][l]);
                n[2][l] = s_shear_plain(n[2][l], tx, tz, mu, cv[i][l], dv[i][l]);
            }
            if constexpr (F != LEAN) {
                {
                    const bool s0 = row_ok && sc.is(Cols::OK0) && (xd || sc.is(Cols::SZ0));
                    const bool s1 = row_ok && sc.is(Cols::OK1) && (xd || sc.is(Cols::SZ1));
                    L m[3];
#pragma unroll
                    for (int l = 0; l < N; l++) {
                        const Damp2 d = lane_damp<PAIR>(fx[i], fz[i], l);
                        const float2 lam = lane_of<PAIR>(lc, l), mu = lane_of<PAIR>(uc, l);
                        S2 x{mxx[i][l], mzz[i][l], mxz[i][l]};
                        S2 y{zpart(xx[l], x.xx), zpart(zz[l], x.zz), zpart(xz[l], x.xz)};
                        if constexpr (PAIR) {
                            auto at = [&](float2 v) { return l ? v.y : v.x; };
                            x.xx.y = fma2(p.dt, at(q.xx_x), x.xx.y), y.xx.y = add2(y.xx.y, at(q.xx_z));
                            x.zz.y = fma2(p.dt, at(q.zz_x), x.zz.y), y.zz.y = add2(y.zz.y, at(q.zz_z));
                            x.xz.y = fma2(p.dt, at(q.xz_x), x.xz.y), y.xz.y = add2(y.xz.y, at(q.xz_z));
                        }
                        s_norm_split(x.xx, x.zz, y.xx, y.zz, d, tx, tz, lam, mu, av[i][l], bv[i][l]);
                        y.xz = s_shear_split(x.xz, y.xz, d, tx, tz, mu, cv[i][l], dv[i][l]);
                        n[0][l] = pick<PAIR>(l, s0, s1, y.xx, n[0][l]);
                        n[1][l] = pick<PAIR>(l, s0, s1, y.zz, n[1][l]);
                        n[2][l] = pick<PAIR>(l, s0, s1, y.xz, n[2][l]);
                        m[0][l] = pick<PAIR>(l, s0, s1, x.xx, mxx[i][l]);
                        m[1][l] = pick<PAIR>(l, s0, s1, x.zz, mzz[i][l]);
                        m[2][l] = pick<PAIR>(l, s0, s1, x.xz, mxz[i][l]);
                    }
                    if (own && (s0 || s1)) {
                        stl<PAIR>(out.mtxx + o * E, m[0]);
                        stl<PAIR>(out.mtzz + o * E, m[1]);
                        stl<PAIR>(out.mtxz + o * E, m[2]);
                    }
                }
                // a second column outside the update region keeps its zero
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int l = 0; l < N; l++)
                        n[c][l] = pick<PAIR>(l, true, sc.is(Cols::OK1), n[c][l], make_float2(0.f, 0.f));
            }
            if (own) {
                stl<PAIR>(out.txx + o * E, n[0]);
                stl<PAIR>(out.tzz + o * E, n[1]);
                stl<PAIR>(out.txz + o * E, n[2]);
            }
        }
    }
    // the coefficients of the thread's columns cs, cs+1 of its row i of group k
    __device__ __forceinline__ void coefs(int k, int i, int cs, float2 &lc, float2 &uc, float2 &bp, float2 &bs) const {
        const float *co = sm + C::O_CO + (k & (C::CSLOT - 1)) * C::CO;
        const float *c = co + (R * ch + i) * C::PC + cs;
        lc = ld2s(c), uc = ld2s(c + G * C::PC);
        if constexpr (PAIR) bp = ld2s(c + 2 * G * C::PC), bs = ld2s(c + 3 * G * C::PC);
    }
};

// Measured against the two sweeps, per step: 38 Born shots at 376x201
// 107 -> 92 us (4.1 TB/s of the 100 bytes a cell needs, 152 SMs), two stage-1 shots at
// 2001x801 51 -> 49 us.  The rest is the instructions of the INNER and EDGE warps, which a
// group's barrier makes the others wait for (all warps LEAN: 72 us), and the
// shared-memory loads of the stencils.  128 registers a thread are a hard limit: any
// spill cost more than it saved (134 us), so flags are bits and the item is in shared memory.
template <int PS, bool PAIR, bool SNAP>
__global__ void __launch_bounds__((FwdCfg<PS, PAIR, false>::NT), (FwdCfg<PS, PAIR, false>::CTAS))
    k_march_fwd(const __grid_constant__ MarchArgs a, const __grid_constant__ MarchMaps tm, int it) {
    using C = FwdCfg<PS, PAIR, false>;
    __shared__ uint64_t full[2];
    __shared__ float src_old[2];
    const Params &p = a.p;
    float *sm = smem();
    const int tid = threadIdx.x;
    __shared__ Item im;
    if (threadIdx.x == 0) im = load_item(p, a.items);
    if (tid == 0) {
        mbar_init(&full[0], PAIR ? 5 : 4);
        mbar_init(&full[1], PAIR ? 5 : 4);
        fence_mbar_init();
    }
    __syncthreads();
    griddep_launch();
    griddep_wait();
    const int K = im.K;
    // what step t of the march adds: sigma group t, v and 1/rho of group t-1,
    // the coefficients of group t-2; one load a warp, each on its own account
    constexpr int LOADS = PAIR ? 5 : 4, LW = C::NT / 32;
    auto issue = [&](int t) {
        if (tid & 31) return;
        uint64_t *bar = &full[t & 1];
        const int r1 = im.row + G * (t - 1), z1 = im.g.z0 - NOP, r2 = im.row + G * (t - 2);
        for (int w = tid >> 5; w < LOADS; w += LW) {
            if (w == 0) {
                mbar_expect_tx(bar, (t == 2 ? 3 : 1) * C::SIG * 4u);
                for (int q = t == 2 ? 0 : t; q <= t; q++)
                    tma_load(sm + (q & (C::NSLOT - 1)) * C::SIG, &tm.view3, im.g.z0 - 2 * NOP, im.row + G * q, BG_TXX, bar);
            } else if (w == 1) {
                mbar_expect_tx(bar, C::VEL * 4u);
                tma_load(sm + C::O_VEL + ((t - 1) & (C::NSLOT - 1)) * C::VEL, &tm.rim2, z1, r1, BG_VX, bar);
            } else if (w == 2) {
                mbar_expect_tx(bar, C::IB * 4u);
                tma_load(sm + C::O_IB + ((t - 1) & 1) * C::IB, &tm.rim1c, z1, r1, C_IB, bar);
            } else {  // (the first two groups take no stress half-step)
                float *c = sm + C::O_CO + (t & 1) * C::CO + (w - 3) * 2 * G * C::PC;
                mbar_expect_tx(bar, t >= 4 ? 2 * G * C::PC * 4u : 0u);
                if (t >= 4) tma_load(c, &tm.core2c, im.g.z0, r2, w == 3 ? C_LAM : C_BP, bar);
            }
        }
    };
    issue(2);
    if (K > 3) issue(3);
    FwdBody<C, SNAP> body(a, im, sm, it);
    // group of the source row, if the item's view holds the source cell
    const int gsrc = (im.m.flags & MARCH_SOURCE) && p.src_kind == SRC_TXX_TZZ ? (im.m.g.isx - im.g.x0 + 2 * G) / G : -1;
    for (int t = 2; t < K; t++) {
        const bool ok = mbar_wait(&full[t & 1], ((t - 2) >> 1) & 1, p.wait_limit);
        if (gsrc >= 0 && (t == 2 ? gsrc <= 2 : gsrc == t)) {
            if (tid == 0 && ok) {
                // explosive source into the total txx and tzz of the
                // background, seen by the velocity half-step only
                const int r = im.m.g.isx - im.g.x0 + 2 * G - G * gsrc, c = im.m.g.isz - im.g.z0 + 2 * NOP;
                float *s = sm + (gsrc & (C::NSLOT - 1)) * C::SIG + (r * PS + c) * C::E;
                src_old[0] = s[0];
                src_old[1] = s[C::ASIG];
                s[0] += p.sou[it];
                s[C::ASIG] += p.sou[it];
            }
            __syncthreads();
        }
        body.velocity(t - 1);
        if (__syncthreads_or(!ok)) {
            give_up(p, full, t, K);
            return;
        }
        if (t >= 4) body.stress(t - 2, src_old);
        // this thread's accesses of the freed groups come before the
        // asynchronous-proxy writes that refill them
        fence_proxy_async();
        __syncthreads();
        if (t + 2 < K) issue(t + 2);
    }
    if (SNAP) body.snap_scale();
}

// The groups of a short item all at once.  Bound by latency: a launch, the
// loads, two half-steps of one or two groups a warp.  One stage-1 shot at 376x201
// 8.3 -> 5.0 us a step, at 149x83 7.7 -> 4.4 us (Born 9.1 -> 4.4 us).  No prefetches: the
// next group is at work next door, and they cost 0.4 us a step.
template <int PS, bool PAIR, bool SNAP>
__global__ void __launch_bounds__((FwdCfg<PS, PAIR, true>::NT), 1)
    k_burst_fwd(const __grid_constant__ MarchArgs a, const __grid_constant__ MarchMaps tm, int it) {
    using C = FwdCfg<PS, PAIR, true>;
    __shared__ uint64_t full;
    __shared__ float src_old[2];
    const Params &p = a.p;
    float *sm = smem();
    const int tid = threadIdx.x, warp = tid >> 5;
    __shared__ Item im;
    if (threadIdx.x == 0) im = load_item(p, a.items);
    if (tid == 0) {
        mbar_init(&full, 1);
        fence_mbar_init();
        const int K = im.K;
        mbar_expect_tx(&full, (K * C::SIG + (K - 2) * (C::VEL + C::IB) + (K - 4) * C::CO) * 4u);
    }
    __syncthreads();
    const int K = im.K;
    griddep_launch();
    griddep_wait();
    if ((tid & 31) == 0)
        // (group, array) pairs over the warps
        for (int w = warp; w < K * 5; w += C::NT / 32) {
            const int q = w / 5, r = im.row + G * q, z1 = im.g.z0 - NOP;
            const bool rim = q >= 1 && q < K - 1, core = q >= 2 && q < K - 2;
            switch (w % 5) {
            case 0: tma_load(sm + q * C::SIG, &tm.view3, im.g.z0 - 2 * NOP, r, BG_TXX, &full); break;
            case 1:
                if (rim) tma_load(sm + C::O_VEL + q * C::VEL, &tm.rim2, z1, r, BG_VX, &full);
                break;
            case 2:
                if (rim) tma_load(sm + C::O_IB + q * C::IB, &tm.rim1c, z1, r, C_IB, &full);
                break;
            case 3:
                if (core) tma_load(sm + C::O_CO + q * C::CO, &tm.core2c, im.g.z0, r, C_LAM, &full);
                break;
            default:
                if (PAIR && core)
                    tma_load(sm + C::O_CO + q * C::CO + 2 * G * C::PC, &tm.core2c, im.g.z0, r, C_BP, &full);
            }
        }
    FwdBody<C, SNAP> body(a, im, sm, it);
    const bool ok = mbar_wait(&full, 0, p.wait_limit);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicExch(p.err, 1);
            mbar_wait(&full, 0, PIPE_WAIT_LIMIT);  // the copies must land before the CTA leaves
        }
        return;
    }
    if ((im.m.flags & MARCH_SOURCE) && p.src_kind == SRC_TXX_TZZ) {
        if (tid == 0) {
            // explosive source into the total txx and tzz of the background,
            // seen by the velocity half-step only
            const int d = im.m.g.isx - im.g.x0 + 2 * G, c = im.m.g.isz - im.g.z0 + 2 * NOP;
            float *s = sm + d / G * C::SIG + (d % G * PS + c) * C::E;
            src_old[0] = s[0];
            src_old[1] = s[C::ASIG];
            s[0] += p.sou[it];
            s[C::ASIG] += p.sou[it];
        }
        __syncthreads();
    }
    constexpr int TEAMS = C::NT / 32 / C::BLOCKS;
    for (int k = 1 + warp / C::BLOCKS; k < K - 1; k += TEAMS) body.velocity(k);
    __syncthreads();
    for (int k = 2 + warp / C::BLOCKS; k < K - 2; k += TEAMS) body.stress(k, src_old);
    if (SNAP) body.snap_scale();
}

// ---------------------------------------------------------------------------
// backward step
// ---------------------------------------------------------------------------
// PAIR: reconstruction and adjoint; else the adjoint alone
template <int PS_, bool PAIR_, bool BURST_>
struct BwdCfg : StepCfg<PS_, PAIR_, BURST_> {
    using B = StepCfg<PS_, PAIR_, BURST_>;
    using B::E, B::PS, B::PV, B::PC, B::NSLOT, B::CSLOT, B::NT;
    static constexpr int AVEL = G * PS * E, ASIG = G * PV * E, AOWN = G * PC * E;
    static constexpr int VEL = 2 * AVEL, SIG = 3 * ASIG, LM = 2 * G * PV, IB = G * PC, OWN = 2 * AOWN;
    static constexpr int O_SIG = NSLOT * VEL, O_LM = O_SIG + NSLOT * SIG, O_IB = O_LM + CSLOT * LM,
                         O_OWN = O_IB + CSLOT * IB;
    static constexpr int FLOATS = O_OWN + CSLOT * OWN;
    static constexpr size_t BYTES = (size_t)FLOATS * 4 + 128;
    static constexpr int FIT = (int)(228 * 1024 / (BYTES + 1024 + 64));
    static constexpr int CTAS = FIT > 512 / NT ? 512 / NT : FIT;
};
// bit pattern marking a packed row without a receiver in the residual source
constexpr uint32_t NO_RECEIVER_BITS = 0xFFFFFFFFu;

template <class C, bool RHO>
struct BwdBody {
    static constexpr bool PAIR = C::PAIR;
    static constexpr int N = Lanes<PAIR>::N, E = C::E, R = C::R;
    using L = Lanes<PAIR>;
    const MarchArgs &a;
    const Item &im;
    float *sm;
    int it, ch;
    float adj_dir;
    Cols sc, vc;      // columns of the stress (rim) and the velocity (core) half-step

    __device__ __forceinline__ BwdBody(const MarchArgs &a_, const Item &im_, float *sm_, int it_, float adj)
        : a(a_), im(im_), sm(sm_), it(it_), adj_dir(adj) {
        const Geo &g = im.g;
        const int cp = (threadIdx.x >> 5) % C::BLOCKS * C::LPR + threadIdx.x % C::LPR;
        ch = (threadIdx.x & 31) / C::LPR;
        sc = cols_at(g, g.z0 - NOP, 2 * cp, C::PV, min(g.z0 + g.zw, g.nzpml - 2 * NOP) + NOP);
        vc = cols_at(g, g.z0, 2 * cp, C::PC, g.z0 + g.zw);
        // (a column the item owns but does not image: undamped, at the interior's edge)
        special(sc, sc.is(Cols::OWN) && !(sc.is(Cols::IM0) && sc.is(Cols::IM1)));
        special(vc, vc.is(Cols::OWN) && !(vc.is(Cols::IM0) && vc.is(Cols::IM1)));
    }
    template <Form F>
    __device__ __forceinline__ bool image_row(const Row &r) const {
        return r.own && (F != EDGE || (r.lx >= im.g.pml && r.lx < im.g.nxpml - im.g.pml));
    }

    // The transient writes of this step on the view: the saved edge strips
    // replace the reconstructed velocity, the residual the adjoint velocity at
    // the receivers.  A thread fetches what it writes into group t (a value of a
    // top or bottom strip, a receiver's residual) an iteration ahead; the rare
    // rows of a left or right strip are read when they are written.
    struct Patch {
        float strip, rz, rx;
        bool has_strip, has_res;
    };
    __device__ __forceinline__ Patch fetch(int t) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const int zv = g.z0 - 2 * NOP, lx0 = g.x0 - 2 * G + G * t;  // first column and row of the view
        Patch q;
        q.has_strip = q.has_res = false;
        if (PAIR && threadIdx.x < 128) {
            const int i = threadIdx.x, b = i >> 6, comp = (i >> 5) & 1, r = (i >> 3) & 3, c = i & 7;
            const int lx = lx0 + r, col = strip_z0(b) + c - zv;
            if (lx >= g.pml && lx < g.nxpml - g.pml && col >= 0 && col < C::PS) {
                q.strip = p.tb[tb_row(it % p.strip_steps, comp, b, p.X, g.row0 + lx) * 8 + c];
                q.has_strip = true;
            }
        }
        if ((im.m.flags & MARCH_RECV) && threadIdx.x >= C::NT - G) {
            const int lx = lx0 + (int)threadIdx.x - (C::NT - G);
            if (lx >= 0 && lx < g.nxpml) {
                const float2 rs = ld2g(a.rsrc + (size_t)(g.row0 + lx) * a.rsp + 2 * it);
                q.rz = rs.x, q.rx = rs.y;
                q.has_res = __float_as_uint(q.rz) != NO_RECEIVER_BITS;
            }
        }
        return q;
    }
    __device__ __forceinline__ int strip_z0(int b) const {
        return b == 0 ? im.g.pml - NOP : im.g.nzpml - im.g.pml - NOP;
    }
    __device__ __forceinline__ void patch(int t, const Patch &q) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const int zv = g.z0 - 2 * NOP, lx0 = g.x0 - 2 * G + G * t;
        float *v = sm + (t & (C::NSLOT - 1)) * C::VEL;
        if (PAIR) {
            if (q.has_strip) {
                const int i = threadIdx.x, b = i >> 6, comp = (i >> 5) & 1, r = (i >> 3) & 3, c = i & 7;
                v[comp * C::AVEL + (r * C::PS + strip_z0(b) + c - zv) * E] = q.strip;
            }
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const int xb = b == 0 ? g.pml - NOP : g.nxpml - g.pml - NOP;
                if (lx0 + G > xb && lx0 < xb + 2 * NOP) {
                    for (int r = 0; r < G; r++) {
                        const int br = lx0 + r - xb;
                        if (br < 0 || br >= 2 * NOP) continue;
                        for (int i = threadIdx.x; i < 2 * C::PS; i += C::NT) {
                            const int comp = i >= C::PS, col = i - comp * C::PS, z = zv + col;
                            if (z >= g.pml && z < g.nzpml - g.pml)
                                v[comp * C::AVEL + (r * C::PS + col) * E] =
                                    p.lr[lr_row(it % p.strip_steps, comp, b, p.nshots, im.m.shot, br) * p.P + z];
                        }
                    }
                }
            }
        }
        if (q.has_res) {
            const int r = threadIdx.x - (C::NT - G);
            float *av = v + (r * C::PS + im.m.g.igz - zv) * E + (PAIR ? 1 : 0);
            av[C::AVEL] = q.rz;
            av[0] = q.rx;
        }
    }

    // The same for all groups of a short item at once: a thread fetches up to
    // BZ values of the top and bottom strips, BX of the left and right ones and a
    // row's residual while the groups are on their way.
    static constexpr int ROWS = G * C::NSLOT, BZ = 32 * ROWS / C::NT;
    static constexpr int XN = 2 * 2 * 2 * NOP * C::PS, BX = (XN + C::NT - 1) / C::NT;
    struct Patches {
        float z[BZ], x[BX];
        int zo[BZ], xo[BX];  // where they go (-1: nowhere)
        float rz, rx;
        int ro;
    };
    __device__ __forceinline__ void fetch_all(int K, Patches &q) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const int zv = g.z0 - 2 * NOP, xv = g.x0 - 2 * G, sit = it % p.strip_steps;
        if constexpr (PAIR) {
#pragma unroll
            for (int j = 0; j < BZ; j++) {
                const int i = threadIdx.x + j * C::NT, r = i >> 5, b = (i >> 4) & 1, comp = (i >> 3) & 1, c = i & 7;
                const int lx = xv + r, col = strip_z0(b) + c - zv;
                q.zo[j] = -1;
                if (r < G * K && lx >= g.pml && lx < g.nxpml - g.pml && col >= 0 && col < C::PS) {
                    q.z[j] = p.tb[tb_row(sit, comp, b, p.X, g.row0 + lx) * 8 + c];
                    q.zo[j] = at(r, comp, col);
                }
            }
#pragma unroll
            for (int j = 0; j < BX; j++) {
                const int i = threadIdx.x + j * C::NT, f = i / C::PS, col = i - f * C::PS;
                const int b = f >> 4, comp = (f >> 3) & 1, br = f & 7;
                const int r = (b == 0 ? g.pml - NOP : g.nxpml - g.pml - NOP) + br - xv, z = zv + col;
                q.xo[j] = -1;
                if (i < XN && r >= 0 && r < G * K && z >= g.pml && z < g.nzpml - g.pml) {
                    q.x[j] = p.lr[lr_row(sit, comp, b, p.nshots, im.m.shot, br) * p.P + z];
                    q.xo[j] = at(r, comp, col);
                }
            }
        }
        q.ro = -1;
        if ((im.m.flags & MARCH_RECV) && threadIdx.x < G * K) {
            const int r = threadIdx.x, lx = xv + r;
            if (lx >= 0 && lx < g.nxpml) {
                const float2 rs = ld2g(a.rsrc + (size_t)(g.row0 + lx) * a.rsp + 2 * it);
                q.rz = rs.x, q.rx = rs.y;
                if (__float_as_uint(q.rz) != NO_RECEIVER_BITS) q.ro = at(r, 0, im.m.g.igz - zv) + (PAIR ? 1 : 0);
            }
        }
    }
    __device__ __forceinline__ static int at(int r, int comp, int col) {
        return (r / G) * C::VEL + comp * C::AVEL + (r % G * C::PS + col) * E;
    }
    __device__ __forceinline__ void patch_all(const Patches &q) const {
        if constexpr (PAIR) {
#pragma unroll
            for (int j = 0; j < BZ; j++)
                if (q.zo[j] >= 0) sm[q.zo[j]] = q.z[j];
#pragma unroll
            for (int j = 0; j < BX; j++)
                if (q.xo[j] >= 0) sm[q.xo[j]] = q.x[j];
        }
        if (q.ro >= 0) {
            sm[q.ro] = q.rx;
            sm[q.ro + C::AVEL] = q.rz;
        }
    }

    // the thread's rows of group k: reconstructed and adjoint stresses, imaging
    // of the columns the item owns; the ring keeps the reconstructed stresses
    // and the Lame-weighted adjoint ones
    __device__ __forceinline__ void stress(int k) const {
        const int g0 = im.g.x0 - 2 * G + G * k, lx0 = g0 + R * ch;
        if (sc.is(Cols::NONE)) return;
        if (!inner_rows(im.g, g0))
            stress<EDGE>(k, lx0);
        else if (sc.is(Cols::PLAIN))
            stress<LEAN>(k, lx0);
        else
            stress<INNER>(k, lx0);
    }
    template <Form F>
    __device__ __forceinline__ void stress(int k, int lx0) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const FieldSet &in = PAIR ? a.in_bg : a.in_ad, &out = PAIR ? p.bg : p.ad;
        const int cv = sc.col;
        const unsigned o0 = (unsigned)((g.row0 + lx0) * g.P + sc.z);
        L mxx[R], mzz[R], mxz[R];
        float4 fx[R], fz[R];
        float2 gl[R], gm[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const size_t o = o0 + i * g.P;
            if constexpr (F != LEAN) {
                const bool xd = F == EDGE && r.xd;
                mxx[i] = mzz[i] = mxz[i] = zero_lanes<PAIR>();
                fx[i] = fz[i] = make_float4(a.one, a.one, a.one, a.one);
                if ((F == INNER || r.ok) && sc.is(Cols::OK0) && (xd || sc.is(Cols::SZ0 | Cols::SZ1))) {
                    load_damp(a, o, xd, fx[i], fz[i]);
                    mxz[i] = ldl<PAIR>(in.mtxz + o * E);
                    if (PAIR) {
                        mxx[i] = ldl<PAIR>(in.mtxx + o * E);
                        mzz[i] = ldl<PAIR>(in.mtzz + o * E);
                    }
                    if (!C::BURST && r.lx + G < g.nxpml) {
                        // the next group's, while this one is computed
                        const size_t n = o + G * g.P;
                        prefetch_l2(a.fz + 2 * n);
                        if (xd) prefetch_l2(a.fx + 2 * n);
                        prefetch_l2(in.mtxz + n * E);
                        if (PAIR) {
                            prefetch_l2(in.mtxx + n * E);
                            prefetch_l2(in.mtzz + n * E);
                        }
                    }
                }
            }
            if (PAIR && image_row<F>(r) && (sc.is(Cols::IM0 | Cols::IM1))) {
                gl[i] = ld2g(p.glam + o);
                gm[i] = ld2g(p.gmu + o);
                if (!C::BURST && r.lx + G < g.nxpml) {
                    prefetch_l2(p.glam + o + G * g.P);
                    prefetch_l2(p.gmu + o + G * g.P);
                }
            }
        }
        const RowOff<R> ro = row_off<C::NSLOT, C::VEL, C::PS * E, R>(k, ch);
        const float *vel = sm + (cv + NOP) * E;
        L av[R], bv[R], cc[R], dv[R];
        ddx<PAIR, false>(vel, ro, av);
        ddx<PAIR, true>(vel + C::AVEL, ro, dv);
#pragma unroll
        for (int i = 0; i < R; i++) {
            cc[i] = ddz<PAIR, true>(vel + ro.o[i + 4]);
            bv[i] = ddz<PAIR, false>(vel + C::AVEL + ro.o[i + 4]);
        }
        const float *lm = sm + C::O_LM + (k & (C::CSLOT - 1)) * C::LM + R * ch * C::PV + cv;
        float *sig = sm + C::O_SIG + (k & (C::NSLOT - 1)) * C::SIG + (R * ch * C::PV + cv) * E;
        const float rtx = -p.dtdx, rtz = -p.dtdz, atx = adj_dir * p.dtdx, atz = adj_dir * p.dtdz;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const bool row_ok = F != EDGE || r.ok, xd = F == EDGE && r.xd;
            const size_t o = o0 + i * g.P;
            const L xx = ldl<PAIR>(sig + i * C::PV * E), zz = ldl<PAIR>(sig + C::ASIG + i * C::PV * E),
                    xz = ldl<PAIR>(sig + 2 * C::ASIG + i * C::PV * E);
            const float2 lc = ld2s(lm + i * C::PV), uc = ld2s(lm + (G + i) * C::PV);
            const bool s0 = row_ok && sc.is(Cols::OK0) && (xd || sc.is(Cols::SZ0));
            const bool s1 = row_ok && sc.is(Cols::OK1) && (xd || sc.is(Cols::SZ1));
            const bool k0 = row_ok && sc.is(Cols::OK0), k1 = row_ok && sc.is(Cols::OK1);
            const bool own = row_ok && r.own && sc.is(Cols::OWN);
            L n[3], w[3];  // the new stresses, and what the ring keeps
            if constexpr (PAIR) {
                // lanes: the two columns of one field
                auto cols = [](const L &v, bool ad) {
                    return ad ? make_float2(v[0].y, v[N - 1].y) : make_float2(v[0].x, v[N - 1].x);
                };
                const float2 ga = cols(av[i], false), gb = cols(bv[i], false), gc = cols(cc[i], false),
                             gd = cols(dv[i], false);
                const float2 aa = cols(av[i], true), ab = cols(bv[i], true), ac = cols(cc[i], true),
                             ad = cols(dv[i], true);
                const S2 ob{cols(xx, false), cols(zz, false), cols(xz, false)};
                const S2 oa{cols(xx, true), cols(zz, true), cols(xz, true)};
                S2 nb = s_plain2<false>(ob, B2(rtx), B2(rtz), lc, uc, ga, gb, gc, gd, Born2{});
                S2 na = as_plain2(oa, B2(atx), B2(atz), aa, ab, ac, ad);
                if constexpr (F != LEAN) {
                    const Damp2 d = lane_damp<false>(fx[i], fz[i], 0);
                    const S2 mb{cols(mxx[i], false), cols(mzz[i], false), cols(mxz[i], false)};
                    const float2 ma = cols(mxz[i], true);
                    S2 xb = mb;
                    float2 xa = ma;
                    const S2 tb = s_split2<false>(ob, xb, d, B2(rtx), B2(rtz), lc, uc, ga, gb, gc, gd, Born2{});
                    const S2 ta = as_split2(oa, xa, d, B2(atx), B2(atz), aa, ab, ac, ad);
                    nb = S2{sel(s0, s1, tb.xx, nb.xx), sel(s0, s1, tb.zz, nb.zz), sel(s0, s1, tb.xz, nb.xz)};
                    na = S2{sel(s0, s1, ta.xx, na.xx), sel(s0, s1, ta.zz, na.zz), sel(s0, s1, ta.xz, na.xz)};
                    if (own && (s0 || s1)) {
                        xb = S2{sel(s0, s1, xb.xx, mb.xx), sel(s0, s1, xb.zz, mb.zz), sel(s0, s1, xb.xz, mb.xz)};
                        xa = sel(s0, s1, xa, ma);
                        st4(out.mtxx + o * E, make_float4(xb.xx.x, 0.f, xb.xx.y, 0.f));
                        st4(out.mtzz + o * E, make_float4(xb.zz.x, 0.f, xb.zz.y, 0.f));
                        st4(out.mtxz + o * E, make_float4(xb.xz.x, xa.x, xb.xz.y, xa.y));
                    }
                }
                if constexpr (F != LEAN) {
                    const float2 zero = make_float2(0.f, 0.f);
                    nb = S2{sel(k0, k1, nb.xx, zero), sel(k0, k1, nb.zz, zero), sel(k0, k1, nb.xz, zero)};
                    na = S2{sel(k0, k1, na.xx, zero), sel(k0, k1, na.zz, zero), sel(k0, k1, na.xz, zero)};
                }
                if (image_row<F>(r) && (sc.is(Cols::IM0 | Cols::IM1))) {
                    const Img2 q = image2(p.idx, p.idz, ga, gb, gc, gd, na);
                    const float2 nl = fma2(B2(-1.f), q.lg, gl[i]), nm = fma2(B2(-1.f), q.mg, gm[i]);
                    st2(p.glam + o, F == LEAN ? nl : sel(sc.is(Cols::IM0), sc.is(Cols::IM1), nl, gl[i]));
                    st2(p.gmu + o, F == LEAN ? nm : sel(sc.is(Cols::IM0), sc.is(Cols::IM1), nm, gm[i]));
                }
                const S2 wa = lame2(na, lc, uc);
                auto pairs = [](float2 b, float2 c) {
                    L v;
                    v[0] = make_float2(b.x, c.x), v[N - 1] = make_float2(b.y, c.y);
                    return v;
                };
                n[0] = pairs(nb.xx, na.xx), n[1] = pairs(nb.zz, na.zz), n[2] = pairs(nb.xz, na.xz);
                w[0] = pairs(nb.xx, wa.xx), w[1] = pairs(nb.zz, wa.zz), w[2] = pairs(nb.xz, wa.xz);
            } else {
                const S2 old{xx[0], zz[0], xz[0]};
                S2 t = as_plain2(old, B2(atx), B2(atz), av[i][0], bv[i][0], cc[i][0], dv[i][0]);
                if constexpr (F != LEAN) {
                    float2 x = mxz[i][0];
                    const S2 u = as_split2(old, x, lane_damp<false>(fx[i], fz[i], 0), B2(atx), B2(atz), av[i][0],
                                           bv[i][0], cc[i][0], dv[i][0]);
                    t = S2{sel(s0, s1, u.xx, t.xx), sel(s0, s1, u.zz, t.zz), sel(s0, s1, u.xz, t.xz)};
                    if (own && (s0 || s1)) st2(out.mtxz + o, sel(s0, s1, x, mxz[i][0]));
                }
                if constexpr (F != LEAN) {
                    const float2 zero = make_float2(0.f, 0.f);
                    t = S2{sel(k0, k1, t.xx, zero), sel(k0, k1, t.zz, zero), sel(k0, k1, t.xz, zero)};
                }
                n[0][0] = t.xx, n[1][0] = t.zz, n[2][0] = t.xz;
                const S2 q = lame2(t, lc, uc);
                w[0][0] = q.xx, w[1][0] = q.zz, w[2][0] = q.xz;
            }
            if (own) {
                stl<PAIR>(out.txx + o * E, n[0]);
                stl<PAIR>(out.tzz + o * E, n[1]);
                stl<PAIR>(out.txz + o * E, n[2]);
            }
            if (sc.is(Cols::ACTIVE))
#pragma unroll
                for (int c = 0; c < 3; c++) stl<PAIR>(sig + c * C::ASIG + i * C::PV * E, w[c]);
        }
    }

    // the thread's rows of group k: reconstructed and adjoint velocities,
    // illumination, density kernel
    __device__ __forceinline__ void velocity(int k) const {
        const int g0 = im.g.x0 - 2 * G + G * k, lx0 = g0 + R * ch;
        if (vc.is(Cols::NONE)) return;
        if (!inner_rows(im.g, g0))
            velocity<EDGE>(k, lx0);
        else if (vc.is(Cols::PLAIN))
            velocity<LEAN>(k, lx0);
        else
            velocity<INNER>(k, lx0);
    }
    template <Form F>
    __device__ __forceinline__ void velocity(int k, int lx0) const {
        const Params &p = a.p;
        const Geo &g = im.g;
        const FieldSet &in = PAIR ? a.in_bg : a.in_ad, &out = PAIR ? p.bg : p.ad;
        const int cs = vc.col;
        const unsigned o0 = (unsigned)((g.row0 + lx0) * g.P + vc.z);
        L mx[R], mz[R];
        float4 fx[R], fz[R];
        float2 il[R], gr[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const size_t o = o0 + i * g.P;
            if constexpr (F != LEAN) {
                const bool xd = F == EDGE && r.xd;
                mx[i] = mz[i] = zero_lanes<PAIR>();
                fx[i] = fz[i] = make_float4(a.one, a.one, a.one, a.one);
                if ((F == INNER || r.ok) && r.own && vc.is(Cols::OWN) && (xd || vc.is(Cols::SZ0 | Cols::SZ1))) {
                    load_damp(a, o, xd, fx[i], fz[i]);
                    mx[i] = ldl<PAIR>(in.mvx + o * E);
                    mz[i] = ldl<PAIR>(in.mvz + o * E);
                    if (!C::BURST && r.lx + G < g.nxpml) {
                        prefetch_l2(in.mvx + (o + G * g.P) * E);
                        prefetch_l2(in.mvz + (o + G * g.P) * E);
                    }
                }
            }
            if (PAIR && image_row<F>(r) && (vc.is(Cols::IM0 | Cols::IM1))) {
                il[i] = ld2g(p.illum + o);
                if (RHO) gr[i] = ld2g(p.grho + o);
                if (!C::BURST && r.lx + G < g.nxpml) {
                    prefetch_l2(p.illum + o + G * g.P);
                    if (RHO) prefetch_l2(p.grho + o + G * g.P);
                }
            }
        }
        const RowOff<R> ro = row_off<C::NSLOT, C::SIG, C::PV * E, R>(k, ch);
        const float *sig = sm + C::O_SIG + (cs + NOP) * E;
        L ax[R], dx[R], bz[R], dz[R];
        ddx<PAIR, true>(sig, ro, ax);
        ddx<PAIR, false>(sig + 2 * C::ASIG, ro, dx);
#pragma unroll
        for (int i = 0; i < R; i++) {
            bz[i] = ddz<PAIR, false>(sig + 2 * C::ASIG + ro.o[i + 4]);
            dz[i] = ddz<PAIR, true>(sig + C::ASIG + ro.o[i + 4]);
        }
        const float *ib = sm + C::O_IB + (k & (C::CSLOT - 1)) * C::IB + R * ch * C::PC + cs;
        const float *own_v = sm + C::O_OWN + (k & (C::CSLOT - 1)) * C::OWN + (R * ch * C::PC + cs) * E;
        const float atx = adj_dir * p.dtdx, atz = adj_dir * p.dtdz;
        const float2 tx = PAIR ? make_float2(-p.dtdx, atx) : B2(atx), tz = PAIR ? make_float2(-p.dtdz, atz) : B2(atz);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const Row r = row_at(g, lx0 + i);
            const bool row_ok = F != EDGE || r.ok, xd = F == EDGE && r.xd;
            const size_t o = o0 + i * g.P;
            const L ox = ldl<PAIR>(own_v + i * C::PC * E), oz = ldl<PAIR>(own_v + C::AOWN + i * C::PC * E);
            const float2 ic = ld2s(ib + i * C::PC);
            const bool own = row_ok && r.own && vc.is(Cols::OWN);
            L vx, vz;
            float2 cx[N], cz[N];
#pragma unroll
            for (int l = 0; l < N; l++) {
                const float2 i2 = lane_of<PAIR>(ic, l);
                cx[l] = mul2(i2, tx), cz[l] = mul2(i2, tz);
                vx[l] = v_plain1(ox[l], cx[l], cz[l], ax[i][l], bz[i][l]);
                vz[l] = v_plain1(oz[l], cx[l], cz[l], dx[i][l], dz[i][l]);
            }
            if constexpr (F != LEAN) {
                {
                    const bool s0 = row_ok && vc.is(Cols::OK0) && (xd || vc.is(Cols::SZ0));
                    const bool s1 = row_ok && vc.is(Cols::OK1) && (xd || vc.is(Cols::SZ1));
                    L nx, nz;
#pragma unroll
                    for (int l = 0; l < N; l++) {
                        V2 m{mx[i][l], mz[i][l]};
                        const V2 v = v_split2(V2{ox[l], oz[l]}, m, lane_damp<PAIR>(fx[i], fz[i], l), cx[l], cz[l],
                                              ax[i][l], bz[i][l], dx[i][l], dz[i][l]);
                        vx[l] = pick<PAIR>(l, s0, s1, v.x, vx[l]);
                        vz[l] = pick<PAIR>(l, s0, s1, v.z, vz[l]);
                        nx[l] = pick<PAIR>(l, s0, s1, m.x, mx[i][l]);
                        nz[l] = pick<PAIR>(l, s0, s1, m.z, mz[i][l]);
                    }
                    if (own && (s0 || s1)) {
                        stl<PAIR>(out.mvx + o * E, nx);
                        stl<PAIR>(out.mvz + o * E, nz);
                    }
                }
                // a second column outside the update region keeps its zero
#pragma unroll
                for (int l = 0; l < N; l++) {
                    vx[l] = pick<PAIR>(l, true, vc.is(Cols::OK1), vx[l], make_float2(0.f, 0.f));
                    vz[l] = pick<PAIR>(l, true, vc.is(Cols::OK1), vz[l], make_float2(0.f, 0.f));
                }
            }
            if (own) {
                stl<PAIR>(out.vx + o * E, vx);
                stl<PAIR>(out.vz + o * E, vz);
            }
            if constexpr (PAIR) {
                if (image_row<F>(r) && (vc.is(Cols::IM0 | Cols::IM1))) {
                    const float2 bx = first_of<PAIR>(vx), by = first_of<PAIR>(vz);
                    const float2 e = add2(il[i], fma2(bx, bx, mul2(by, by)));
                    st2(p.illum + o, F == LEAN ? e : sel(vc.is(Cols::IM0), vc.is(Cols::IM1), e, il[i]));
                    if (RHO) {
                        // the density kernel's velocity step, (v(it) - v(it-1)) / dt:
                        // imaging cells lie outside the PML, where the
                        // reconstruction subtracts dt (1/rho) D sigma, so it is
                        // formed from that increment, not as a difference of
                        // two nearly equal velocities
                        const float2 idx = B2(p.idx), idz = B2(p.idz);
                        const float2 gvx = mul2(ic, fma2(first_of<PAIR>(ax[i]), idx, mul2(first_of<PAIR>(bz[i]), idz)));
                        const float2 gvz = mul2(ic, fma2(first_of<PAIR>(dx[i]), idx, mul2(first_of<PAIR>(dz[i]), idz)));
                        // G_rho -= v_adj . (v(it) - v(it-1)) / dt
                        const float2 s = fma2(make_float2(vx[0].y, vx[N - 1].y), gvx,
                                              mul2(make_float2(vz[0].y, vz[N - 1].y), gvz));
                        const float2 f = fma2(B2(-1.f), s, gr[i]);
                        st2(p.grho + o, F == LEAN ? f : sel(vc.is(Cols::IM0), vc.is(Cols::IM1), f, gr[i]));
                    }
                }
            }
        }
    }
};

// Measured against the two sweeps, per step: 38 shots at 376x201 with the density
// kernel 126 -> 116 us, two shots at 2001x801 97 -> 93 us; the adjoint alone (and the imaging
// of every fourth step) of two shots at 2001x801 57.5 -> 55 us.
template <int PS, bool PAIR, bool RHO>
__global__ void __launch_bounds__((BwdCfg<PS, PAIR, false>::NT), (BwdCfg<PS, PAIR, false>::CTAS))
    k_march_bwd(const __grid_constant__ MarchArgs a, const __grid_constant__ MarchMaps tm, int it, float adj_dir) {
    using C = BwdCfg<PS, PAIR, false>;
    __shared__ uint64_t full[2];
    const Params &p = a.p;
    float *sm = smem();
    const int tid = threadIdx.x;
    const Item im = load_item(p, a.items);
    if (tid == 0) {
        mbar_init(&full[0], 5);
        mbar_init(&full[1], 5);
        fence_mbar_init();
    }
    __syncthreads();
    griddep_launch();
    griddep_wait();
    const int K = im.K;
    // what step t of the march adds: the velocities' view of group t, the
    // stresses and Lame parameters of group t-1, 1/rho and the stored
    // velocities (the view is overwritten at strips and receivers) of group
    // t-2; one load a warp, each on its own account
    constexpr int LOADS = 5, LW = C::NT / 32;
    auto issue = [&](int t) {
        if (tid & 31) return;
        uint64_t *bar = &full[t & 1];
        const int r1 = im.row + G * (t - 1), z1 = im.g.z0 - NOP, r2 = im.row + G * (t - 2);
        for (int w = tid >> 5; w < LOADS; w += LW) {
            if (w == 0) {
                mbar_expect_tx(bar, (t == 2 ? 3 : 1) * C::VEL * 4u);
                for (int q = t == 2 ? 0 : t; q <= t; q++)
                    tma_load(sm + (q & (C::NSLOT - 1)) * C::VEL, &tm.view2, im.g.z0 - 2 * NOP, im.row + G * q, BG_VX, bar);
            } else if (w == 1) {
                mbar_expect_tx(bar, C::SIG * 4u);
                tma_load(sm + C::O_SIG + ((t - 1) & (C::NSLOT - 1)) * C::SIG, &tm.rim3, z1, r1, BG_TXX, bar);
            } else if (w == 2) {
                mbar_expect_tx(bar, C::LM * 4u);
                tma_load(sm + C::O_LM + ((t - 1) & 1) * C::LM, &tm.rim2c, z1, r1, C_LAM, bar);
            } else if (w == 3) {  // (the first two groups take no velocity half-step)
                mbar_expect_tx(bar, t >= 4 ? C::OWN * 4u : 0u);
                if (t >= 4) tma_load(sm + C::O_OWN + (t & 1) * C::OWN, &tm.core2, im.g.z0, r2, BG_VX, bar);
            } else {
                mbar_expect_tx(bar, t >= 4 ? C::IB * 4u : 0u);
                if (t >= 4) tma_load(sm + C::O_IB + (t & 1) * C::IB, &tm.core1c, im.g.z0, r2, C_IB, bar);
            }
        }
    };
    issue(2);
    if (K > 3) issue(3);
    const BwdBody<C, RHO> body(a, im, sm, it, adj_dir);
    // a group is patched as soon as it has landed, an iteration before its use
    bool ok = mbar_wait(&full[0], 0, p.wait_limit);
    for (int q = 0; q < 3; q++) body.patch(q, body.fetch(q));
    __syncthreads();
    for (int t = 2; t < K; t++) {
        typename BwdBody<C, RHO>::Patch next;
        next.has_strip = next.has_res = false;
        if (t + 1 < K) next = body.fetch(t + 1);
        body.stress(t - 1);
        if (__syncthreads_or(!ok)) {
            give_up(p, full, t, K);
            return;
        }
        if (t >= 4) body.velocity(t - 2);
        if (t + 1 < K) {
            ok = mbar_wait(&full[(t + 1) & 1], ((t - 1) >> 1) & 1, p.wait_limit);
            body.patch(t + 1, next);
        }
        fence_proxy_async();
        __syncthreads();
        if (t + 2 < K) issue(t + 2);
    }
}

// One shot at 376x201 11.1 -> 6.9 us a step, at 149x83 10.4 -> 5.1 us.  The strips and
// residuals are fetched while the loads are on their way: read row by row after
// them they cost 6 us.
template <int PS, bool PAIR, bool RHO>
__global__ void __launch_bounds__((BwdCfg<PS, PAIR, true>::NT), 1)
    k_burst_bwd(const __grid_constant__ MarchArgs a, const __grid_constant__ MarchMaps tm, int it, float adj_dir) {
    using C = BwdCfg<PS, PAIR, true>;
    __shared__ uint64_t full;
    const Params &p = a.p;
    float *sm = smem();
    const int tid = threadIdx.x, warp = tid >> 5;
    __shared__ Item im;
    if (threadIdx.x == 0) im = load_item(p, a.items);
    if (tid == 0) {
        mbar_init(&full, 1);
        fence_mbar_init();
        const int K = im.K;
        mbar_expect_tx(&full, (K * C::VEL + (K - 2) * (C::SIG + C::LM) + (K - 4) * (C::IB + C::OWN)) * 4u);
    }
    __syncthreads();
    const int K = im.K;
    griddep_launch();
    griddep_wait();
    if ((tid & 31) == 0)
        for (int w = warp; w < K * 5; w += C::NT / 32) {
            const int q = w / 5, r = im.row + G * q, z1 = im.g.z0 - NOP;
            const bool rim = q >= 1 && q < K - 1, core = q >= 2 && q < K - 2;
            switch (w % 5) {
            case 0: tma_load(sm + q * C::VEL, &tm.view2, im.g.z0 - 2 * NOP, r, BG_VX, &full); break;
            case 1:
                if (rim) tma_load(sm + C::O_SIG + q * C::SIG, &tm.rim3, z1, r, BG_TXX, &full);
                break;
            case 2:
                if (rim) tma_load(sm + C::O_LM + q * C::LM, &tm.rim2c, z1, r, C_LAM, &full);
                break;
            case 3:
                if (core) tma_load(sm + C::O_OWN + q * C::OWN, &tm.core2, im.g.z0, r, BG_VX, &full);
                break;
            default:
                if (core) tma_load(sm + C::O_IB + q * C::IB, &tm.core1c, im.g.z0, r, C_IB, &full);
            }
        }
    const BwdBody<C, RHO> body(a, im, sm, it, adj_dir);
    // (the fetches of the patches overlap the loads)
    typename BwdBody<C, RHO>::Patches q;
    body.fetch_all(K, q);
    const bool ok = mbar_wait(&full, 0, p.wait_limit);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicExch(p.err, 1);
            mbar_wait(&full, 0, PIPE_WAIT_LIMIT);  // the copies must land before the CTA leaves
        }
        return;
    }
    body.patch_all(q);
    __syncthreads();
    constexpr int TEAMS = C::NT / 32 / C::BLOCKS;
    for (int k = 1 + warp / C::BLOCKS; k < K - 1; k += TEAMS) body.stress(k);
    __syncthreads();
    for (int k = 2 + warp / C::BLOCKS; k < K - 2; k += TEAMS) body.velocity(k);
}

// ---------------------------------------------------------------------------
// between the passes
// ---------------------------------------------------------------------------
// What the steps read per cell as pairs: the PML factors, rounded as
// make_damp2 rounds them, fx = (d1, r2) and fz = (d3, r4)
__global__ void k_march_factors(const MarchFactors f) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < f.n; i += (size_t)gridDim.x * blockDim.x) {
        const float x = f.dampx[i], z = f.dampz[i];
        st2(f.fx + 2 * i, make_float2(damp_minus(f.dt, x), damp_plus_rcp(f.dt, x)));
        st2(f.fz + 2 * i, make_float2(damp_minus(f.dt, z), damp_plus_rcp(f.dt, z)));
    }
}

// The state that the backward steps start from: the background's last forward
// state as the reconstruction and, in pairs, a zero adjoint.  A shot's forward
// steps end in copy nt & 1 of its own length (blockIdx.y: the shot).
__global__ void k_pair_start(const PairStart s) {
    const ShotGeo g = s.geo[blockIdx.y];
    const int c = s.aux[blockIdx.y].nt & 1;
    const size_t n = (size_t)g.nxpml * s.P, off = (size_t)g.row0 * s.P;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
#pragma unroll
        for (int k = 0; k < 10; k++) {
            const size_t o = k * s.cells + off + i;
            if (s.from_pairs && s.to_pairs)
                s.dst[c][2 * o + 1] = 0.f;
            else if (s.from_pairs)
                s.dst[c][o] = s.src[c][2 * o];
            else if (s.to_pairs)
                st2(s.dst[c] + 2 * o, make_float2(s.src[c][o], 0.f));
            else if (s.src[c] != s.dst[c])
                s.dst[c][o] = s.src[c][o];
        }
}

// ---------------------------------------------------------------------------
// snapshots
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t to16(float v, int fmt) {
    return fmt == SNAP_F16 ? (uint32_t)__half_as_ushort(__float2half_rn(v))
                           : (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float from16(uint16_t u, int fmt) {
    return fmt == SNAP_F16 ? __half2float(__ushort_as_half(u)) : __bfloat162float(__ushort_as_bfloat16(u));
}

// the background velocity after step `it` as snapshot it / snap_every: every
// cell of the padded grid (blockIdx.y: the shot), four columns a thread; a vertical force of
// this step is part of it
template <bool PAIR>
__global__ void k_snap_store(const __grid_constant__ MarchArgs a, int it) {
    griddep_launch();
    griddep_wait();
    const Params &p = a.p;
    const ShotGeo g = p.geo[blockIdx.y];
    const int k = it / p.snap_every, q = p.P / 4;
    const bool force = p.src_kind == SRC_VZ_FORCE;
    const float *sc = p.sscale + ((size_t)blockIdx.y * p.nsnap + k) * 2;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.nxpml * q; i += gridDim.x * blockDim.x) {
        const int lx = i / q, z = 4 * (i - lx * q);
        const size_t gi = (size_t)(g.row0 + lx) * p.P + z;
#pragma unroll
        for (int comp = 0; comp < 2; comp++) {
            const float *src = comp ? p.bg.vz : p.bg.vx;
            float4 v;
            if constexpr (PAIR) {
                const float4 u = ld4(src + 2 * gi), w = ld4(src + 2 * gi + 4);
                v = make_float4(u.x, u.z, w.x, w.z);
            } else {
                v = ld4(src + gi);
            }
            if (comp && force && lx == g.isx && g.isz >= z && g.isz < z + 4) {
                float *e = g.isz == z ? &v.x : g.isz == z + 1 ? &v.y : g.isz == z + 2 ? &v.z : &v.w;
                *e += p.sou[it];
            }
            const size_t o = ((size_t)(2 * k + comp) * p.X + g.row0 + lx) * p.PS + z;
            if (p.snap_fmt == SNAP_F32) {
                st4(reinterpret_cast<float *>(p.snap) + o, v);
            } else {
                const float s = sc[comp], inv = s > 0.f ? 1.0f / s : 0.f;
                const uint32_t w0 = to16(v.x * inv, p.snap_fmt) | (to16(v.y * inv, p.snap_fmt) << 16);
                const uint32_t w1 = to16(v.z * inv, p.snap_fmt) | (to16(v.w * inv, p.snap_fmt) << 16);
                *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(p.snap) + o) = make_uint2(w0, w1);
            }
        }
    }
}

// imaging of backward step `it` from its snapshot, after the adjoint step: the
// strains of the stored velocities by the reconstruction's stencils, weight
// snap_every.  A block takes 32 x 64 interior cells of one shot, with their
// rim decompressed into shared memory.
constexpr int IX = 32, IZ = 64, IP = IZ + 2 * NOP;
template <int FMT>
__global__ void __launch_bounds__(256) k_snap_image(const __grid_constant__ MarchArgs a, int it) {
    __shared__ float sv[2][(IX + 2 * NOP) * IP];
    griddep_launch();
    griddep_wait();
    const Params &p = a.p;
    const ShotGeo g = p.geo[blockIdx.z];
    const int k = it / p.snap_every;
    const int x0 = p.pml + blockIdx.x * IX, z0 = (p.pml & ~3) + blockIdx.y * IZ;
    if (x0 >= g.nxpml - p.pml || z0 >= g.nzpml - p.pml) return;
    const float w = (float)p.snap_every;
    const float *sc = p.sscale + ((size_t)blockIdx.z * p.nsnap + k) * 2;
    for (int i = threadIdx.x; i < 2 * (IX + 2 * NOP) * (IP / 4); i += blockDim.x) {
        const int comp = i / ((IX + 2 * NOP) * (IP / 4)), j = i - comp * (IX + 2 * NOP) * (IP / 4);
        const int r = j / (IP / 4), c = 4 * (j - r * (IP / 4));
        const int lx = x0 - NOP + r, z = z0 - NOP + c;  // z is a multiple of 4, at least 0 (pml >= 8)
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lx < g.nxpml && z < p.P) {
            const size_t o = ((size_t)(2 * k + comp) * p.X + g.row0 + lx) * p.PS + z;
            if (FMT == SNAP_F32) {
                v = ld4(reinterpret_cast<const float *>(p.snap) + o);
            } else {
                const uint2 u = *reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(p.snap) + o);
                const float s = sc[comp];
                v = make_float4(from16(u.x & 0xffffu, FMT) * s, from16(u.x >> 16, FMT) * s,
                                from16(u.y & 0xffffu, FMT) * s, from16(u.y >> 16, FMT) * s);
            }
        }
        st4(&sv[comp][r * IP + c], v);
    }
    __syncthreads();
    // 32 column pairs x 8 runs of four rows, two rows at a time
    const int cp = threadIdx.x & 31, ch = threadIdx.x >> 5;
    const int z = z0 + 2 * cp;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int r0 = 4 * ch + 2 * h;  // first row in the block
        constexpr int R = 2;
        RowOff<R> ro;
#pragma unroll
        for (int i = 0; i < R + 8; i++) ro.o[i] = (r0 + i) * IP + 2 * cp + NOP;
        Lanes<false> av[R], dv[R];
        ddx<false, false>(sv[0], ro, av);
        ddx<false, true>(sv[1], ro, dv);
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int lx = x0 + r0 + i;
            const bool row = lx < g.nxpml - p.pml;
            const bool i0 = row && z >= p.pml && z < g.nzpml - p.pml;
            const bool i1 = row && z + 1 >= p.pml && z + 1 < g.nzpml - p.pml;
            if (!i0 && !i1) continue;
            const size_t gi = (size_t)(g.row0 + lx) * p.P + z;
            const float *vx = sv[0] + ro.o[i + 4], *vz = sv[1] + ro.o[i + 4];
            const float2 cc = ddz<false, true>(vx)[0], bv = ddz<false, false>(vz)[0];
            const S2 s{ld2g(p.ad.txx + gi), ld2g(p.ad.tzz + gi), ld2g(p.ad.txz + gi)};
            const float2 gl = ld2g(p.glam + gi), gm = ld2g(p.gmu + gi), il = ld2g(p.illum + gi);
            const Img2 q = image2(p.idx, p.idz, av[i][0], bv, cc, dv[i][0], s);
            const float2 nl = fma2(B2(-w), q.lg, gl), nm = fma2(B2(-w), q.mg, gm);
            const float2 x = ld2s(vx), y = ld2s(vz);
            const float2 ni = fma2(B2(w), fma2(x, x, mul2(y, y)), il);
            st2(p.glam + gi, sel(i0, i1, nl, gl));
            st2(p.gmu + gi, sel(i0, i1, nm, gm));
            st2(p.illum + gi, sel(i0, i1, ni, il));
        }
    }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
template <class... KArgs, class... Args>
cudaError_t launch(void (*k)(KArgs...), dim3 grid, int threads, size_t bytes, bool overlap, cudaStream_t st,
                   Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

// one way of working on the items: the kernels of a strip width
template <int PS, bool BURST>
struct Way {
    using F1 = FwdCfg<PS, false, BURST>;
    using F2 = FwdCfg<PS, true, BURST>;
    using B1 = BwdCfg<PS, false, BURST>;
    using B2_ = BwdCfg<PS, true, BURST>;
    using Fwd = void (*)(const MarchArgs, const MarchMaps, int);
    using Bwd = void (*)(const MarchArgs, const MarchMaps, int, float);
    template <bool PAIR, bool SNAP>
    static Fwd fwd_kernel() {
        if constexpr (BURST)
            return k_burst_fwd<PS, PAIR, SNAP>;
        else
            return k_march_fwd<PS, PAIR, SNAP>;
    }
    template <bool PAIR, bool RHO>
    static Bwd bwd_kernel() {
        if constexpr (BURST)
            return k_burst_bwd<PS, PAIR, RHO>;
        else
            return k_march_bwd<PS, PAIR, RHO>;
    }
    static cudaError_t configure() {
        cudaError_t e = cudaSuccess;
        auto set = [&](auto *k, size_t bytes) {
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        };
        set(fwd_kernel<false, false>(), F1::BYTES);
        set(fwd_kernel<false, true>(), F1::BYTES);
        set(fwd_kernel<true, false>(), F2::BYTES);
        set(fwd_kernel<true, true>(), F2::BYTES);
        set(bwd_kernel<true, false>(), B2_::BYTES);
        set(bwd_kernel<true, true>(), B2_::BYTES);
        set(bwd_kernel<false, false>(), B1::BYTES);
        return e;
    }
    static void fwd(const MarchArgs &a, const MarchMaps &tm, int nitems, int it, bool born, cudaStream_t st) {
        // the snapshot scale of a step is found by the step itself
        const bool sm = a.p.snap && a.p.snap_fmt != SNAP_F32 && it % a.p.snap_every == 0;
        if (born)
            launch(sm ? fwd_kernel<true, true>() : fwd_kernel<true, false>(), dim3(nitems), F2::NT, F2::BYTES, a.p.overlap,
                   st, a, tm, it);
        else
            launch(sm ? fwd_kernel<false, true>() : fwd_kernel<false, false>(), dim3(nitems), F1::NT, F1::BYTES,
                   a.p.overlap, st, a, tm, it);
    }
    static void bwd(const MarchArgs &a, const MarchMaps &tm, int nitems, int it, float adj_dir, cudaStream_t st) {
        if (a.p.snap)
            launch(bwd_kernel<false, false>(), dim3(nitems), B1::NT, B1::BYTES, a.p.overlap, st, a, tm, it, adj_dir);
        else
            launch(a.p.grho ? bwd_kernel<true, true>() : bwd_kernel<true, false>(), dim3(nitems), B2_::NT, B2_::BYTES,
                   a.p.overlap, st, a, tm, it, adj_dir);
    }
    static const MarchVariant *variant() {
        static const MarchVariant v{PS,          BURST,  {F1::CTAS, F2::CTAS}, {B1::CTAS, B2_::CTAS},
                                    &configure, &fwd, &bwd};
        return &v;
    }
};

}  // namespace

const MarchVariant *march_wide() { return Way<136, false>::variant(); }
const MarchVariant *march_burst() { return Way<72, true>::variant(); }

void launch_march_factors(const MarchFactors &f, cudaStream_t st) {
    k_march_factors<<<(int)std::min<size_t>((f.n + 255) / 256, 8192), 256, 0, st>>>(f);
}
void launch_pair_start(const PairStart &s, int max_nxpml, int nshots, cudaStream_t st) {
    const size_t n = (size_t)max_nxpml * s.P;
    k_pair_start<<<dim3((int)std::min<size_t>((n + 255) / 256, 1024), nshots), 256, 0, st>>>(s);
}
void launch_snap_store(const MarchArgs &a, int max_nxpml, int it, bool pairs, cudaStream_t st) {
    const int n = max_nxpml * (a.p.P / 4);
    const dim3 grid(std::min((n + 255) / 256, 2048), a.p.nshots);
    launch(pairs ? k_snap_store<true> : k_snap_store<false>, grid, 256, 0, a.p.overlap, st, a, it);
}
void launch_snap_image(const MarchArgs &a, int max_nx, int max_nz, int it, cudaStream_t st) {
    const dim3 grid((max_nx + IX - 1) / IX, (max_nz + 3 + IZ - 1) / IZ, a.p.nshots);
    if (a.p.snap_fmt == SNAP_F32)
        launch(k_snap_image<SNAP_F32>, grid, 256, 0, a.p.overlap, st, a, it);
    else if (a.p.snap_fmt == SNAP_F16)
        launch(k_snap_image<SNAP_F16>, grid, 256, 0, a.p.overlap, st, a, it);
    else
        launch(k_snap_image<SNAP_BF16>, grid, 256, 0, a.p.overlap, st, a, it);
}

}  // namespace sfwi
