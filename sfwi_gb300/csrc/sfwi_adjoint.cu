// sfwi_adjoint.cu — the exact discrete adjoint of the Born modelling operator.
//
// The stage-2 forward (sfwi-stage2/FD2DGPU.cu:1814-1843, born.cu:749-801) maps
// a model perturbation (dVp, dVs) linearly to the scattered records: each
// time step runs the scattered velocity sweep, records the scattered
// velocities, then adds the Born virtual source (dt * 2 rho vp dVp, 2 rho vs
// dVs times strains of the background velocity) to the split parts of the
// scattered stresses inside the stress sweep.  The reference's Hessian
// products (ELSRTM_CALCULATE_Hessian_vector*, sfwi-stage1/FD2DGPU.cu:
// 5236-5774, with add_born_source_adjoint_components, born.cu:886-958)
// approximate its transpose with the continuous adjoint equations.  The
// kernels here are the transpose of the forward sweeps this library runs
// (k_fwd_v, k_fwd_s: the same stencils, the same split-field PML update in
// damped cells and plain update elsewhere, the same update region), so
// <L m, d> = <m, L^T d> holds to rounding: reverse-mode differentiation of
// one time step, run backwards from the last step.
//
// Per reverse step `it` (forward step: V' = V-sweep(V, S); record V';
// S' = S-sweep(S, V', born(m, background V'))), two launches:
//   k_adj_velocity  adjoint of V': gathers of G (transposed stencils: the
//                   transpose of D+ is -D-), the records' data at the
//                   receiver cells, then the own-cell transpose of the
//                   velocity sweep: the adjoint of V and the fields H
//   k_adj_stress    the adjoint of S gathers H, which ends step `it`; then, of step
//                   it - 1, the own-cell transpose of the stress sweep: the
//                   adjoint of S (and its x-parts), the fields G to be scattered
//                   into the adjoint of V', and the Born-source adjoint folded into
//                   per-cell accumulators of d(2 rho vp dVp) and d(2 rho vs dVs) with
//                   the background strains of step it - 1
// The adjoint of S is zero before the last step, so that step has no stress
// part, and nothing reads what the velocity part of step 0 would leave.
// The transposed stencil gathers read G/H of the cells up to 4 away, which
// are zero outside the update region [4, n-4), so they stay within a shot.
//
// A thread takes two adjacent columns of a row and reads its stencils straight
// from memory: at the sizes of a Hessian product the fields live in L2, a
// block's rows share lines in L1, and what counts is the number of launches
// and the loads in flight.  five shots at 251x121: 32.4 -> 9.2 us a step, eight at
// 376x201 73.9 -> 24.9 us, against three launches with a cell a thread and
// the accumulators' twenty FP64 operations a cell, which alone kept the FP64 pipe 69 % busy
// for half of the step; they are float pairs of 48 bits now.  So that their
// products keep clear of FP32's smallest numbers whatever the units of the source
// and the records, the records enter times a power of two that makes the
// largest about 1, the strains likewise, and k_born_image divides by both.
#include "sfwi_d2.cuh"
#include "sfwi_launch.h"
#include "sfwi_pipe.cuh"

namespace sfwi {

namespace {

constexpr float AK1 = (float)(1225.0 / 1024.0);
constexpr float AK2 = (float)(-245.0 / 3072.0);
constexpr float AK3 = (float)(49.0 / 5120.0);
constexpr float AK4 = (float)(-5.0 / 7168.0);
__device__ __forceinline__ float kk(int k) { return k == 1 ? AK1 : k == 2 ? AK2 : k == 3 ? AK3 : AK4; }

__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void st2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ float2 mask2(bool a, bool b, float2 v) { return make_float2(a ? v.x : 0.f, b ? v.y : 0.f); }

// Staggered first derivatives at columns z, z+1 of a row (f: at z, z even; rows
// `s` floats apart): dp sum K_k (f[+k] - f[-k+1]), dm sum K_k (f[+k-1] - f[-k]), along
// x (rows) and z (columns).
template <bool PLUS>
__device__ __forceinline__ float2 ddx(const float *f, long long s) {
    float2 w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = ld2(f + (i - (PLUS ? 3 : 4)) * s);
    float2 a = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= NOP; k++) {
        a.x += kk(k) * (w[3 + k].x - w[4 - k].x);
        a.y += kk(k) * (w[3 + k].y - w[4 - k].y);
    }
    return a;
}
template <bool PLUS>
__device__ __forceinline__ float2 ddz(const float *f) {
    float w[10];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const float2 v = ld2(f + 2 * i - 4);
        w[2 * i] = v.x, w[2 * i + 1] = v.y;
    }
    constexpr int c = PLUS ? 4 : 3;
    float2 a = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= NOP; k++) {
        a.x += kk(k) * (w[c + k] - w[c + 1 - k]);
        a.y += kk(k) * (w[c + 1 + k] - w[c + 2 - k]);
    }
    return a;
}

// the two columns of a thread
struct Cells {
    int row, lz;      // packed row, first column
    size_t i;         // packed index in [X][P]
    int igz;          // the shot's receiver depth
    bool live0, live1;        // inside the update region
    bool damped0, damped1;
};
constexpr int BZ = 16, BX = 16;  // threads of a block: column pairs, rows
__device__ __forceinline__ Cells cells_at(const AdjArgs &a) {
    Cells c;
    c.row = blockIdx.x * BX + threadIdx.y;
    c.lz = 2 * (blockIdx.y * BZ + threadIdx.x);
    c.live0 = c.live1 = false;
    if (c.row >= a.X) return c;
    const ShotGeo g = a.geo[a.rowshot[c.row]];
    const int lx = c.row - g.row0, nx = g.nxpml, nz = g.nzpml, pml = a.pml;
    c.i = (size_t)c.row * a.P + c.lz;
    c.igz = g.igz;
    const bool row = lx >= NOP && lx < nx - NOP, dx = lx < pml || lx > nx - pml;
    c.live0 = row && c.lz >= NOP && c.lz < nz - NOP;
    c.live1 = c.live0 && c.lz + 1 < nz - NOP;
    c.damped0 = c.live0 && (dx || c.lz < pml || c.lz > nz - pml);
    c.damped1 = c.live1 && (dx || c.lz + 1 < pml || c.lz + 1 > nz - pml);
    return c;
}

// peak[0]: max |record|, peak[1]: max |background velocity| over every 16th step
// back from the last one that the stress part reads, as bits (a wave's amplitude
// changes little in 16 steps once it is under way; of a run of a few steps
// the last has it, the first may have none)
__global__ void k_adj_peaks(const __grid_constant__ AdjArgs a, long long nrec) {
    float m = 0.f, v = 0.f;
    const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (long long i = i0; i < nrec; i += step) m = fmaxf(m, fmaxf(fabsf(a.dz[i]), fabsf(a.dx[i])));
    const long long n = (long long)2 * a.X * a.PS / 4;  // a step's velocities, four at a time
    for (int it = a.nt - 2; it >= 0; it -= 16) {
        const float4 *q = reinterpret_cast<const float4 *>(a.snap + (size_t)it * 2 * a.X * a.PS);
        for (long long i = i0; i < n; i += step) {
            const float4 w = q[i];
            v = fmaxf(v, fmaxf(fmaxf(fabsf(w.x), fabsf(w.y)), fmaxf(fabsf(w.z), fabsf(w.w))));
        }
    }
    const unsigned r = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    const unsigned s = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    if ((threadIdx.x & 31) == 0) {
        atomicMax(a.peak, r);
        atomicMax(a.peak + 1, s);
    }
}
// the power of two that brings a peak to [1, 2) (1 where there is none, or none finite)
__device__ __forceinline__ float unit_scale(unsigned peak) {
    const unsigned e = peak >> 23;
    return e == 0 || e >= 254 ? 1.f : __uint_as_float((254u - e) << 23);
}

// the PML factors of the forward update: 1 - dt d / 2 and 1 / (1 + dt d / 2)
struct Fac {
    float d1, r2, d3, r4;
};
__device__ __forceinline__ Fac damp_factors(const AdjArgs &a, float dx, float dz) {
    const float tx = a.dt * dx, tz = a.dt * dz;
    return Fac{fmaf(tx, -0.5f, 1.f), __frcp_rn(fmaf(tx, 0.5f, 1.f)), fmaf(tz, -0.5f, 1.f),
               __frcp_rn(fmaf(tz, 0.5f, 1.f))};
}

// own-cell transpose of the stress sweep of one cell: the adjoint stresses A and
// x-parts M in place, the fields G, and what the Born source's x- and
// z-parts (xx, zz, xz) are weighted with
struct StressCell {
    float axx, azz, axz, mxx, mzz, mxz;
    float gax, gbz, gcz, gdx, b[6];
};
__device__ __forceinline__ void stress_cell(StressCell &s, bool damped, const Fac &f, float l, float u) {
    const float l2m = l + 2.f * u;
    const float Axx = s.axx, Azz = s.azz, Axz = s.axz;
    if (damped) {
        const float Bxx = s.mxx + Axx, Bzz = s.mzz + Azz, Bxz = s.mxz + Axz;
        s.mxx = f.r2 * f.d1 * Bxx - f.r4 * f.d3 * Axx;
        s.mzz = f.r2 * f.d1 * Bzz - f.r4 * f.d3 * Azz;
        s.mxz = f.r2 * f.d1 * Bxz - f.r4 * f.d3 * Axz;
        s.axx = s.b[1] = f.r4 * f.d3 * Axx;
        s.azz = s.b[3] = f.r4 * f.d3 * Azz;
        s.axz = s.b[5] = f.r4 * f.d3 * Axz;
        s.b[0] = f.r2 * f.d1 * Bxx;
        s.b[2] = f.r2 * f.d1 * Bzz;
        s.b[4] = f.r2 * f.d1 * Bxz;
        s.gax = f.r2 * (l2m * Bxx + l * Bzz);
        s.gbz = f.r4 * (l * Axx + l2m * Azz);
        s.gdx = f.r2 * u * Bxz;
        s.gcz = f.r4 * u * Axz;
    } else {
        s.b[0] = s.b[1] = Axx;
        s.b[2] = s.b[3] = Azz;
        s.b[4] = s.b[5] = Axz;
        s.gax = l2m * Axx + l * Azz;
        s.gbz = l * Axx + l2m * Azz;
        s.gdx = s.gcz = u * Axz;
    }
}

// the gathers of step it + 1, then the stress part of step `it`
__global__ void __launch_bounds__(BZ *BX) k_adj_stress(const __grid_constant__ AdjArgs a, int it) {
    griddep_launch();
    const Cells c = cells_at(a);
    if (!c.live0) return;
    const size_t i = c.i;
    // strains of the background velocity after the velocity sweep of step `it`
    // (the Born source's: Dx- vx, Dz- vz, Dx+ vz, Dz+ vx), not written by the adjoint
    const float *svx = a.snap + (size_t)(2 * it) * a.X * a.PS + (size_t)c.row * a.PS + c.lz,
                *svz = svx + (size_t)a.X * a.PS;
    const float2 AX = ddx<false>(svx, a.PS), BZ_ = ddz<false>(svz), DX = ddx<true>(svz, a.PS), CZ = ddz<true>(svx);
    const float2 l = ld2(a.lam + i), u = ld2(a.mu + i);
    const bool damped = c.damped0 || c.damped1;
    float2 fx = make_float2(0.f, 0.f), fz = fx;
    if (damped) fx = ld2(a.dampx + i), fz = ld2(a.dampz + i);
    griddep_wait();
    const float unit = unit_scale(a.peak[1]), idx = a.idx * unit, idz = a.idz * unit;
    // the velocity sweep read S through Dx+ txx, Dz- txz, Dx- txz, Dz+ tzz
    const float2 hx = ddx<false>(a.hax + i, a.P), hz = ddz<false>(a.hcz + i), bz = ddz<true>(a.hbz + i),
                 dx = ddx<true>(a.hdx + i, a.P);
    const float2 xx = ld2(a.atxx + i), zz = ld2(a.atzz + i), xz = ld2(a.atxz + i);
    float2 mxx = make_float2(0.f, 0.f), mzz = mxx, mxz = mxx;
    if (damped) mxx = ld2(a.amxx + i), mzz = ld2(a.amzz + i), mxz = ld2(a.amxz + i);
    float4 bp = *reinterpret_cast<const float4 *>(a.dbp + i), bs = *reinterpret_cast<const float4 *>(a.dbs + i);
    StressCell s[2] = {{xx.x - hx.x, zz.x - hz.x, xz.x - (bz.x + dx.x), mxx.x, mzz.x, mxz.x},
                       {xx.y - hx.y, zz.y - hz.y, xz.y - (bz.y + dx.y), mxx.y, mzz.y, mxz.y}};
    stress_cell(s[0], c.damped0, c.damped0 ? damp_factors(a, fx.x, fz.x) : Fac{}, l.x, u.x);
    stress_cell(s[1], c.damped1, c.damped1 ? damp_factors(a, fx.y, fz.y) : Fac{}, l.y, u.y);
    const bool k1 = c.live1;
    auto both = [&](float StressCell::*m) { return make_float2(s[0].*m, k1 ? s[1].*m : 0.f); };
    st2(a.atxx + i, both(&StressCell::axx));
    st2(a.atzz + i, both(&StressCell::azz));
    st2(a.atxz + i, both(&StressCell::axz));
    if (damped) {
        st2(a.amxx + i, both(&StressCell::mxx));
        st2(a.amzz + i, both(&StressCell::mzz));
        st2(a.amxz + i, both(&StressCell::mxz));
    }
    st2(a.gax + i, both(&StressCell::gax));
    st2(a.gbz + i, both(&StressCell::gbz));
    st2(a.gcz + i, both(&StressCell::gcz));
    st2(a.gdx + i, both(&StressCell::gdx));
    // (dt and the units are applied in k_born_image)
    auto image = [&](float ax, float bz2, float dx2, float cz, const StressCell &q, D2 &p, D2 &h) {
        const float AXi = ax * idx, BZi = bz2 * idz, DXi = dx2 * idx, CZi = cz * idz;
        const D2 mix = add_product(add_product(D2{0.f, 0.f}, BZi, q.b[1]), AXi, q.b[2]);
        p = add_product(add_product(p, AXi, q.b[0]), BZi, q.b[3]) + mix;
        h = add_product(add_product(h, DXi, q.b[4]), CZi, q.b[5]) + D2{-2.f * mix.h, -2.f * mix.l};
    };
    D2 p0{bp.x, bp.y}, p1{bp.z, bp.w}, s0{bs.x, bs.y}, s1{bs.z, bs.w};
    image(AX.x, BZ_.x, DX.x, CZ.x, s[0], p0, s0);
    if (k1) image(AX.y, BZ_.y, DX.y, CZ.y, s[1], p1, s1);
    *reinterpret_cast<float4 *>(a.dbp + i) = make_float4(p0.h, p0.l, p1.h, p1.l);
    *reinterpret_cast<float4 *>(a.dbs + i) = make_float4(s0.h, s0.l, s1.h, s1.l);
}

__global__ void __launch_bounds__(BZ *BX) k_adj_velocity(const __grid_constant__ AdjArgs a, int it) {
    griddep_launch();
    const Cells c = cells_at(a);
    if (!c.live0) return;
    const size_t i = c.i;
    const float2 ib = ld2(a.ib + i);
    const bool damped = c.damped0 || c.damped1;
    float2 fx = make_float2(0.f, 0.f), fz = fx;
    if (damped) fx = ld2(a.dampx + i), fz = ld2(a.dampz + i);
    griddep_wait();
    // the stress sweep read V' through tx Dx- vx, tz Dz+ vx, tz Dz- vz, tx Dx+ vz
    const float2 gx = ddx<true>(a.gax + i, a.P), gc = ddz<false>(a.gcz + i), gb = ddz<true>(a.gbz + i),
                 gd = ddx<false>(a.gdx + i, a.P);
    const float2 vx = ld2(a.avx + i), vz = ld2(a.avz + i);
    float2 mx = make_float2(0.f, 0.f), mz = mx;
    if (damped) mx = ld2(a.amx + i), mz = ld2(a.amz + i);
    float2 AX = make_float2(vx.x - a.dtdx * gx.x - a.dtdz * gc.x, vx.y - a.dtdx * gx.y - a.dtdz * gc.y);
    float2 AZ = make_float2(vz.x - a.dtdz * gb.x - a.dtdx * gd.x, vz.y - a.dtdz * gb.y - a.dtdx * gd.y);
    // the records of step it read V' at the receiver cells (every trace
    // recorded there, in trace order)
    if (c.lz == c.igz || c.lz + 1 == c.igz) {
        const float unit = unit_scale(a.peak[0]);
        for (int k = a.rstart[c.row]; k < a.rstart[c.row + 1]; k++) {
            const size_t o = (size_t)a.rtr[k] * a.nt + it;
            (c.lz == c.igz ? AZ.x : AZ.y) += unit * a.dz[o];
            (c.lz == c.igz ? AX.x : AX.y) += unit * a.dx[o];
        }
    }
    // own-cell transpose of the velocity sweep: A and the x-part M in place, the fields H
    auto cell = [&](float &ax, float &az, float &qx, float &qz, float b, bool d, float dx, float dz, float4 &h) {
        const float cx = b * a.dtdx, cz = b * a.dtdz;
        if (d) {
            const Fac f = damp_factors(a, dx, dz);
            const float Bx = qx + ax, Bz = qz + az;
            qx = f.r2 * f.d1 * Bx - f.r4 * f.d3 * ax;
            qz = f.r2 * f.d1 * Bz - f.r4 * f.d3 * az;
            h = make_float4(f.r2 * cx * Bx, f.r4 * cz * ax, f.r2 * cx * Bz, f.r4 * cz * az);
            ax = f.r4 * f.d3 * ax;
            az = f.r4 * f.d3 * az;
        } else {
            h = make_float4(cx * ax, cz * ax, cx * az, cz * az);
        }
    };
    float4 h0, h1;
    cell(AX.x, AZ.x, mx.x, mz.x, ib.x, c.damped0, fx.x, fz.x, h0);
    cell(AX.y, AZ.y, mx.y, mz.y, ib.y, c.damped1, fx.y, fz.y, h1);
    const bool k1 = c.live1;
    st2(a.avx + i, mask2(true, k1, AX));
    st2(a.avz + i, mask2(true, k1, AZ));
    if (damped) {
        st2(a.amx + i, mask2(true, k1, mx));
        st2(a.amz + i, mask2(true, k1, mz));
    }
    st2(a.hax + i, mask2(true, k1, make_float2(h0.x, h1.x)));
    st2(a.hbz + i, mask2(true, k1, make_float2(h0.y, h1.y)));
    st2(a.hdx + i, mask2(true, k1, make_float2(h0.z, h1.z)));
    st2(a.hcz + i, mask2(true, k1, make_float2(h0.w, h1.w)));
}

template <class K>
cudaError_t launch(K k, const AdjArgs &a, int it, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((a.X + BX - 1) / BX, (a.P / 2 + BZ - 1) / BZ);
    cfg.blockDim = dim3(BZ, BX);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, it);
}

int grid_blocks(long long n) {
    long long b = (n + 255) / 256;
    return (int)(b < 8192 ? (b > 0 ? b : 1) : 8192);
}

}  // namespace

int launch_adjoint(const AdjArgs &a, long long nrec, cudaStream_t st) {
    k_adj_peaks<<<1024, 256, 0, st>>>(a, nrec);
    for (int it = a.nt - 1; it >= 1; it--) {
        launch(k_adj_velocity, a, it, st);
        launch(k_adj_stress, a, it - 1, st);
    }
    return 2 * a.nt - 1;
}

// L^T d on the global model: each window cell's accumulated d(2 rho vp dVp),
// d(2 rho vs dVs) times 2 rho vp, 2 rho vs goes to the model cell it was cut
// from (k_setup cuts the window with the PML cells taking the nearest edge
// value, so an edge model cell collects the PML cells beyond it), shots in
// order, FP64.  A thread has a model cell; the cells that collect a
// rectangle of PML cells (up to 21 x 21 at PML 20) are summed by their whole warp:
// one thread's loop over a corner took 1400 us, all of it now 300 us.
__global__ void k_born_image(ImageArgs a) {
    const long long n = (long long)a.allnx * a.allnz, step = (long long)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    const double f = a.dt / ((double)unit_scale(a.peak[0]) * (double)unit_scale(a.peak[1]));
    for (long long w = blockIdx.x * (long long)blockDim.x + (threadIdx.x - lane); w < n; w += step) {
        const long long i = w + lane;
        const bool live = i < n;
        const int gx = (int)(i / a.allnz), gz = (int)(i - (long long)gx * a.allnz);
        double sp = live ? a.img_vp[i] : 0.0, ss = live ? a.img_vs[i] : 0.0;
        auto add = [&](size_t o, double &x, double &y) {
            const double rho = a.rho[o];
            const float2 p = a.dbp[o], q = a.dbs[o];
            x += 2.0 * (rho * a.vp[o]) * (f * ((double)p.x + (double)p.y));
            y += 2.0 * (rho * a.vs[o]) * (f * ((double)q.x + (double)q.y));
        };
        for (int s = 0; s < a.nshots; s++) {
            const ShotGeo g = a.geo[s];
            const int cx = gx - g.win0, nzm = g.nzpml - 2 * a.pml;
            const bool in = live && cx >= 0 && cx < g.nx && gz < nzm;
            const int x0 = cx == 0 ? 0 : a.pml + cx, x1 = cx == g.nx - 1 ? g.nxpml - 1 : a.pml + cx;
            const int z0 = gz == 0 ? 0 : a.pml + gz, z1 = gz == nzm - 1 ? g.nzpml - 1 : a.pml + gz;
            const bool one = x0 == x1 && z0 == z1;
            if (in && one) add((size_t)(g.row0 + x0) * a.P + z0, sp, ss);
            for (unsigned todo = __ballot_sync(0xffffffffu, in && !one); todo; todo &= todo - 1) {
                const int l = __ffs(todo) - 1;
                const int bx0 = __shfl_sync(0xffffffffu, x0, l), bx1 = __shfl_sync(0xffffffffu, x1, l);
                const int bz0 = __shfl_sync(0xffffffffu, z0, l), bz = __shfl_sync(0xffffffffu, z1, l) - bz0 + 1;
                double x = 0.0, y = 0.0;
                for (int k = lane; k < (bx1 - bx0 + 1) * bz; k += 32)
                    add((size_t)(g.row0 + bx0 + k / bz) * a.P + bz0 + k % bz, x, y);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                    y += __shfl_xor_sync(0xffffffffu, y, o);
                }
                if (lane == l) sp += x, ss += y;
            }
        }
        if (live) {
            a.img_vp[i] = sp;
            a.img_vs[i] = ss;
        }
    }
}

void launch_born_image(const ImageArgs &a, cudaStream_t st) {
    k_born_image<<<grid_blocks((long long)a.allnx * a.allnz), 256, 0, st>>>(a);
}

}  // namespace sfwi
