// uns_cc.cu -- cell-centred (CCFVM) residual-and-update hot path on GB300.
//
// Design:
//   * structure-of-arrays in HBM with small per-entity vectors: double4 for
//     the four conserved / primitive / gradient / limiter values of a cell,
//     so a gathered neighbour costs one 32-byte sector;
//   * face kernels compute every per-face quantity once (flux, spectral
//     radius, face gradient) and write it to a face array; cell kernels then
//     gather their faces from an index-sorted face list.  That is atomic-free
//     and deterministic, and the per-cell summation order is exactly the
//     reference's face-loop order (boundary faces, then interior faces, then
//     the viscous loop), so there is no colour pass and no reordering error;
//   * cell kernels fuse what the reference runs as separate cell loops
//     (con2prim + save_old + the limiter's global min/max; spectral radius
//     gather + dt + gradient + limiter; residual gather + RK stage + norm);
//   * LU-SGS forward/backward sweeps run as a list-scheduled dataflow sweep
//     over the cell DAG of the reference ordering inside one cooperative
//     launch: each warp works through its own list of (cell, pass) items and
//     waits (bounded) on the published records of the items it depends on,
//     which reproduces the sequential sweep exactly;
//   * one iteration of the main loop is captured once as a CUDA graph and
//     replayed; iteration number, CFL schedule and the convergence stop live
//     in device memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "uns_cc_impl.cuh"
#include "uns_common.cuh"
#include "uns_packed.hpp"
#include "uns_phys.cuh"
#include "uns_sched.hpp"
#include "uns_sweep.cuh"
#include "unsflow_gpu.h"

using namespace uns;

namespace {


__device__ __forceinline__ bool stopped(const CCView& v, int inst) {
    return v.done != nullptr && ((volatile int*)v.done)[inst] != 0;
}
__device__ __forceinline__ bool stopped(const CCView& v) { return stopped(v, 0); }
__device__ __forceinline__ double cur_cfl(const CCView& v, int inst, double cfl) {
    return v.cfl_sched ? v.cfl_sched[(size_t)inst * v.cfl_stride + v.iter[inst]] : cfl;
}
// Instance of a cell / face / vertex (0 for a single case; -1 for padding).
__device__ __forceinline__ int cell_inst(const CCView& v, int i) { return v.ninst ? v.cinst[i] : 0; }
__device__ __forceinline__ int face_inst(const CCView& v, int f) { return v.ninst ? v.finst[f] : 0; }
__device__ __forceinline__ int vert_inst(const CCView& v, int k) { return v.ninst ? v.pinst[k] : 0; }
// Instance of a block of interior cells, of any width up to kBlock (every
// case has cells, so never -1).
static_assert(kBlock == kCasePad, "the norm's blocks are a case's own");
__device__ __forceinline__ int block_inst(const CCView& v) {
    return v.ninst ? v.cinst[block_case_cell(blockIdx.x, blockDim.x)] : 0;
}
__device__ __forceinline__ const Gas& gas_of(const CCView& v, int inst) { return v.ninst ? v.gas[inst] : v.g; }

// Minimum / maximum of a 64-bit key over a group of lanes (all of which call
// it with the same mask): the extreme high word, then the extreme low word
// among the lanes holding it.
__device__ __forceinline__ unsigned long long grp_min_u64(unsigned grp, unsigned long long e) {
    const unsigned hi = (unsigned)(e >> 32), lo = (unsigned)e;
    const unsigned mh = __reduce_min_sync(grp, hi);
    const unsigned ml = __reduce_min_sync(grp, hi == mh ? lo : 0xffffffffu);
    return ((unsigned long long)mh << 32) | ml;
}
__device__ __forceinline__ unsigned long long grp_max_u64(unsigned grp, unsigned long long e) {
    const unsigned hi = (unsigned)(e >> 32), lo = (unsigned)e;
    const unsigned mh = __reduce_max_sync(grp, hi);
    const unsigned ml = __reduce_max_sync(grp, hi == mh ? lo : 0u);
    return ((unsigned long long)mh << 32) | ml;
}

static __device__ __noinline__ double pow_rare(double a, double b) { return pow(a, b); }
static __device__ __noinline__ double mean_rare(double a, double b) { return 0.5 * (a + b); }
__device__ __forceinline__ void d4get(const double4& q, double o[4]) { o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w; }
__device__ __forceinline__ double4 d4(const double o[4]) { return make_double4(o[0], o[1], o[2], o[3]); }
__device__ __forceinline__ void f4get(const double4& q, F64 o[4]) { o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w; }
__device__ __forceinline__ void f4get(const double4& q, F64I o[4]) { o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w; }
__device__ __forceinline__ double4 f4(const F64I o[4]) { return make_double4(o[0].v, o[1].v, o[2].v, o[3].v); }
__device__ __forceinline__ double4 f4(const F64 o[4]) { return make_double4(o[0].v, o[1].v, o[2].v, o[3].v); }

// ---------------------------------------------------------------- kernels
// con2prim (main.F90:62-67) + save_old (solution.F90:118-132) + the global
// min/max of every cell's primitives incl. ghosts (limiter.F90:146-149) +
// the positivity check of main.F90:384-411, fused over one pass of the cells.
// The eight ranges reduce over a warp by its integer reductions, on the high
// and then the low word (4.2 M cells: 133 -> 107 us, mixed form 96 -> 81,
// against five exchanges of both words each); an atomic skipped where the
// stored range already covers a block's gained nothing.
enum { BEGIN_PRIM = 1, BEGIN_OLD = 2, BEGIN_MINMAX = 4, BEGIN_POS = 8 };

__global__ void __launch_bounds__(kBlock) k_begin(CCView v, int flags) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int inst = i < v.ntot ? cell_inst(v, i) : (v.ninst ? -1 : 0);
    const bool live = inst >= 0 && !stopped(v, inst);
    if (!v.ninst && !live) return;  // one case: the whole grid stops together
    unsigned long long emx[4] = {0ULL, 0ULL, 0ULL, 0ULL};
    unsigned long long emn[4] = {~0ULL, ~0ULL, ~0ULL, ~0ULL};
    bool have = false;  // the primitives below are this thread's qp (no read-back for the limiter range)
    double pr[4];
    if (live && i < v.noc) {
        const Gas& gi = gas_of(v, inst);
        double4 q = v.qc[i];
        if ((flags & BEGIN_PRIM) && v.mixed) {  // con2prim in FP32 from the rounded state
            const float E = narrow(q.x), r = narrow(q.y), ru = narrow(q.z), rv = narrow(q.w);
            const float u = ru / r, w = rv / r;
            const float p = narrow(gi.gamma1) * (E - 0.5f * r * (u * u + w * w));
            v.qpf[i] = make_float4(r, u, w, p);
            pr[0] = widen(r); pr[1] = widen(u); pr[2] = widen(w); pr[3] = widen(p);
            v.qp[i] = make_double4(pr[0], pr[1], pr[2], pr[3]);
            have = true;
            if (v.laminar || v.grad_type == UNS_GRAD_GGFC) v.qT[i] = (double)(p / (r * (float)gi.znd));
            if ((flags & BEGIN_POS) && (r <= 0.f || p <= 0.f)) set_err(v.err, UNS_ERR_NONPOSITIVE, i);
        } else if (flags & BEGIN_PRIM) {
            const PrimT<F64I> P = con2prim_t<F64I>(gi, q.x, q.y, q.z, q.w);
            v.qp[i] = make_double4(q.y, P.u.v, P.v.v, P.p.v);
            v.qT[i] = P.t.v;
            pr[0] = q.y; pr[1] = P.u.v; pr[2] = P.v.v; pr[3] = P.p.v;
            have = true;
            if ((flags & BEGIN_POS) && (P.rho <= F64I(0.0) || P.p <= F64I(0.0))) set_err(v.err, UNS_ERR_NONPOSITIVE, i);
        }
        if (flags & BEGIN_OLD) v.qold[i] = q;
    }
    if (flags & BEGIN_MINMAX) {
        if (live && i < v.ntot) {
            if (!have) {
                const double4 p = v.qp[i];
                pr[0] = p.x; pr[1] = p.y; pr[2] = p.z; pr[3] = p.w;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) { emx[j] = enc_ord(pr[j]); emn[j] = emx[j]; }
        }
        if (v.ninst && blockIdx.x * blockDim.x >= v.noc) {  // ghost blocks of packed cases: per-case lane groups
            const unsigned grp = __match_any_sync(0xffffffffu, live ? inst : -1);
            unsigned long long mx[4], mn[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) { mx[j] = grp_max_u64(grp, emx[j]); mn[j] = grp_min_u64(grp, emn[j]); }
            if (live && (int)(threadIdx.x & 31) == __ffs(grp) - 1)
                for (int j = 0; j < 4; ++j) {
                    atomicMax(&v.minmax[8 * inst + j], mx[j]);
                    atomicMin(&v.minmax[8 * inst + 4 + j], mn[j]);
                }
            return;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { emx[j] = grp_max_u64(0xffffffffu, emx[j]); emn[j] = grp_min_u64(0xffffffffu, emn[j]); }
        __shared__ unsigned long long smx[kBlock / 32][4], smn[kBlock / 32][4];
        int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l == 0)
            for (int j = 0; j < 4; ++j) { smx[w][j] = emx[j]; smn[w][j] = emn[j]; }
        __syncthreads();
        if (threadIdx.x < 4) {  // a block of one case (padded interior blocks of packed cases too)
            const int bi = block_inst(v);
            int j = threadIdx.x;
            unsigned long long a = smx[0][j], b = smn[0][j];
            for (int k = 1; k < kBlock / 32; ++k) { a = smx[k][j] > a ? smx[k][j] : a; b = smn[k][j] < b ? smn[k][j] : b; }
            atomicMax(&v.minmax[8 * bi + j], a);
            atomicMin(&v.minmax[8 * bi + 4 + j], b);
        }
    }
}

// avg_c2v vertex part (average.F90:11-29): pseudo-Laplacian weighted mean.
// FP64 form: 0.42 -> 0.18 ms at 4.2 M cells with the products and the five
// divisions on the integer pipe (106 FP64 instructions per vertex -> 36).
__global__ void __launch_bounds__(512) k_vertex_avg(CCView v) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.nop || stopped(v, vert_inst(v, i))) return;
    if (v.mixed) {  // FP32 from the FP32 primitives; FP64 copies only where an FP64 kernel reads them
        const bool dbl = v.laminar || v.grad_type == UNS_GRAD_GGFC;
        float wt = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
        double c4 = 0.0;
        auto add = [&](int c, float w, const float4& q) {
            wt = wt + w;
            c0 = c0 + q.x * w; c1 = c1 + q.y * w; c2 = c2 + q.z * w; c3 = c3 + q.w * w;
            if (dbl) c4 = c4 + v.qT[c] * (double)w;
        };
        int k = v.v2c_off[i];
        const int k1 = v.v2c_off[i + 1];
        for (; k + 3 < k1; k += 4) {  // four cells' gathers in flight together, sums in order
            int c[4];
            float w[4];
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) { c[u] = __ldg(&v.v2c[k + u]); w[u] = __ldg(&v.v2c_wtf[k + u]); }
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = v.qpf[c[u]];
#pragma unroll
            for (int u = 0; u < 4; ++u) add(c[u], w[u], q[u]);
        }
        for (; k < k1; ++k) {
            const int c = __ldg(&v.v2c[k]);
            add(c, __ldg(&v.v2c_wtf[k]), v.qpf[c]);
        }
        const float r = 1.f / wt;
        const float4 pp = make_float4(c0 * r, c1 * r, c2 * r, c3 * r);
        v.ppf[i] = pp;
        if (dbl) {
            v.pp[i] = make_double4(pp.x, pp.y, pp.z, pp.w);
            v.ppT[i] = c4 / (double)wt;
        }
        return;
    }
    F64I wt = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0, c4 = 0.0;
    for (int k = v.v2c_off[i]; k < v.v2c_off[i + 1]; ++k) {
        int c = __ldg(&v.v2c[k]);
        const F64I w = __ldg(&v.v2c_wt[k]);
        wt = wt + w;
        const double4 q = v.qp[c];
        c0 = c0 + F64I(q.x) * w;
        c1 = c1 + F64I(q.y) * w;
        c2 = c2 + F64I(q.z) * w;
        c3 = c3 + F64I(q.w) * w;
        c4 = c4 + F64I(v.qT[c]) * w;
    }
    v.pp[i] = make_double4((c0 / wt).v, (c1 / wt).v, (c2 / wt).v, (c3 / wt).v);
    v.ppT[i] = (c4 / wt).v;
}

// avg_c2v face part (average.F90:31-36) + spectral02 face radius
// (timestep.F90:77-104).  FP64 form: 0.62 -> 0.14 ms at 4.2 M cells (54 FP64
// instructions per face -> 8; now half HBM-bound, 106 B per face).
__global__ void __launch_bounds__(kBlock) k_face_prim_spec(CCView v) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= v.nof) return;
    const int inst = face_inst(v, f);
    if (stopped(v, inst)) return;
    const Gas& g = gas_of(v, inst);
    if (v.mixed) {  // FP32; the FP64 face radius stays (the LU-SGS prep reads it)
        const int2 p = v.fpt[f];
        const float4 a = v.ppf[p.x], b = v.ppf[p.y], na = v.fnaf[f];
        const float4 q = make_float4(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z), 0.5f * (a.w + b.w));
        v.fqf[f] = q;
        const float a0 = sqrtf((float)g.gamma * q.w / q.x);
        float ll = na.z * (fabsf(q.y * na.x + q.z * na.y) + a0);
        if (v.laminar) {
            ll = ll + (float)(g.vll * v.fmu[f]) / q.x;
            v.fq[f] = make_double4(q.x, q.y, q.z, q.w);
            v.fqT[f] = 0.5 * (v.ppT[p.x] + v.ppT[p.y]);
        }
        v.flaf[f] = ll;
        v.fla[f] = (double)ll;
        return;
    }
    int2 p = v.fpt[f];
    F64I a[4], b[4], q[4];
    f4get(v.pp[p.x], a);
    f4get(v.pp[p.y], b);
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = half(a[j] + b[j]);
    v.fq[f] = f4(q);
    v.fqT[f] = half(F64I(v.ppT[p.x]) + F64I(v.ppT[p.y])).v;
    const double2 n = v.fn[f];
    const F64I a0 = sqrt(F64I(g.gamma) * q[3] / q[0]);
    const F64I un = q[1] * n.x + q[2] * n.y;
    F64I ll = F64I(v.farea[f]) * (fabs(un) + a0);
    // the viscous term of an inviscid flow is 0 / q[0]: +0 unless q[0] is 0 or NaN
    if (v.laminar || !dpos(fabs(q[0]).v)) ll = ll + F64I(g.vll) * F64I(v.fmu[f]) / q[0];
    v.fla[f] = ll.v;
}

// Diamond-path face gradient (gradient.F90:183-261, gradtrixy :281-321).
__device__ __forceinline__ bool gradtri(const F64I* pr0, const F64I* pr1, const F64I* pr2, F64I x0, F64I y0,
                                        F64I x1, F64I y1, F64I x2, F64I y2, F64I gxo[5], F64I gyo[5], F64I& tarea) {
    const F64I xs[3] = {x0, x1, x2}, ys[3] = {y0, y1, y2};
    const F64I* prs[3] = {pr0, pr1, pr2};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int ip1 = (i == 2) ? 0 : i + 1;
        const F64I dx = half(xs[ip1] + xs[i]), dy = ys[ip1] - ys[i];
        tarea = i == 0 ? F64I(zero_plus((dx * dy).v)) : tarea + dx * dy;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int ip1 = (i == 2) ? 0 : i + 1;
        const F64I dx = ys[ip1] - ys[i], dy = -(xs[ip1] - xs[i]);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const F64I var = half(prs[i][k] + prs[ip1][k]);
            gxo[k] = i == 0 ? F64I(zero_plus((var * dx).v)) : gxo[k] + var * dx;
            gyo[k] = i == 0 ? F64I(zero_plus((var * dy).v)) : gyo[k] + var * dy;
        }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) { gxo[k] = gxo[k] / tarea; gyo[k] = gyo[k] / tarea; }
    return dpos(tarea.v);
}

// FP64 unit-bound as plain doubles (477 instructions per face, thirty
// divisions among them): 373 -> 143 us at 262 k cells.
__global__ void __launch_bounds__(kBlock) k_face_ggfc(CCView v) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= v.nof || stopped(v, face_inst(v, f))) return;
    int2 nb = v.fnb[f];
    int2 p = v.fpt[f];
    const double2 X1 = v.pxy[p.x], X2 = v.pxy[p.y], Ci = v.cen[nb.x], Co = v.cen[nb.y];
    F64I P1[5], P2[5], QI[5], QO[5];
    f4get(v.pp[p.x], P1); P1[4] = v.ppT[p.x];
    f4get(v.pp[p.y], P2); P2[4] = v.ppT[p.y];
    f4get(v.qp[nb.x], QI); QI[4] = v.qT[nb.x];
    f4get(v.qp[nb.y], QO); QO[4] = v.qT[nb.y];
    F64I g1x[5], g1y[5], g2x[5], g2y[5], a1, a2;
    const bool ok1 = gradtri(P1, QO, P2, X1.x, X1.y, Co.x, Co.y, X2.x, X2.y, g1x, g1y, a1);
    const bool ok2 = gradtri(P1, P2, QI, X1.x, X1.y, X2.x, X2.y, Ci.x, Ci.y, g2x, g2y, a2);
    if (!(ok1 && ok2)) set_err(v.err, UNS_ERR_MESH, f);
    const F64I s = a1 + a2;
    F64I gx[5], gy[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        gx[k] = (a1 * g1x[k] + a2 * g2x[k]) / s;
        gy[k] = (a1 * g1y[k] + a2 * g2y[k]) / s;
    }
    v.fgx[f] = f4(gx);
    v.fgy[f] = f4(gy);
    v.fgT[f] = make_double2(gx[4].v, gy[4].v);
    v.fasum[f] = s.v;
}

// Per-cell gather over the index-sorted face list: spectral radius + dt
// (timestep.F90:40-49, 101-103), the cell gradient (Gradient_GG
// gradient.F90:95-156, Gradient_GG_FC :159-323, Gradient_LSQR :2-93) and
// limiter_VKN1 (limiter.F90:146-279).  Face order is the reference's loop
// order (interior faces, then boundary faces).
// CG_DIAG: also the LU-SGS diagonal and its reciprocal (with CG_DT; only an
// LU-SGS step reads them).
enum { CG_DT = 1, CG_GRAD = 2, CG_LIM = 4, CG_DIAG = 8 };

// atomicMin of an order-encoded dt into its instance's slot with one atomic
// per converged group of lanes of one instance.  Same result as one atomic
// per lane (min is exact and order-free), without 32 same-address atomics
// per warp.
__device__ __forceinline__ void warp_atomic_min_u64(const CCView& v, int inst, unsigned long long e) {
    const unsigned mask = v.ninst ? __match_any_sync(__activemask(), inst) : __activemask();
    const unsigned long long m = grp_min_u64(mask, e);
    if ((int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicMin(&v.dtmin[inst], m);
}

// The FP64 unit bounded this kernel (520 instructions and 14 divisions per
// cell, 86 % busy; 4.25 ms at 4.2 M cells).  S = F64I leaves the sums alone
// there and takes 1.70 ms; its products' latency (138 cycles against 64) is in
// the way where an SM sub-partition has a warp or two, so small meshes take
// S = F64 (16 384 cells: 25-29 us against 33).  80 registers for three blocks
// per SM rather than two: 1.96 -> 1.93 ms; what is rare (a tie of two ratios, a
// boundary face's average, the native operations) is called, because predicated
// off it would hold the FP64 unit all the same: 1.93 -> 1.70 ms.
template <class S>
__global__ void __launch_bounds__(kBlock, std::is_same<S, F64I>::value ? 3 : 1) k_cell_grad(CCView v, int flags, double cfl_in) {
    // the limiter tolerances of the block's instance (blocks of cells are
    // instance-pure), formed once per block
    __shared__ double stol[4], stol2[4];
    if ((flags & CG_LIM) && threadIdx.x < 4) {
        const int b = block_inst(v), j = threadIdx.x;
        const double t = 0.05 * (dec_ord(v.minmax[8 * b + j]) - dec_ord(v.minmax[8 * b + 4 + j]));
        stol[j] = t;
        stol2[j] = t * t;
    }
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
    const S cvi = v.cv[i];
    if (flags & CG_DT) {
        S la = 0.0;
        for (int k = k0; k < k1; ++k) la = la + v.fla[v.cf[k] & FACE_MASK];
        v.la[i] = la.v;
        const S dt = S(cur_cfl(v, inst, cfl_in)) * cvi / la;
        v.dt[i] = dt.v;
        v.dcv[i] = (dt / cvi).v;
        if (flags & CG_DIAG) {
            const S diag = cvi / dt + S(0.5 * 1.5) * la;
            v.diag[i] = diag.v;
            v.diaginv[i] = (S(1.0) / diag).v;
        }
        warp_atomic_min_u64(v, inst, enc_ord(dt.v));
    }
    S gx[4], gy[4];
    if (flags & CG_GRAD) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { gx[j] = 0.0; gy[j] = 0.0; }
        S den = 1.0;
        if (v.grad_type == UNS_GRAD_GG) {
            for (int k = k0; k < k1; ++k) {
                int e = v.cf[k], f = e & FACE_MASK;
                double2 n = v.fn[f];
                const S area = v.farea[f];
                S q[4];
                f4get(v.fq[f], q);
                // + on the `in` side of an interior face, - on the other and on a boundary face
                const bool minus = f >= v.nfi || (e & SIDE_BIT);
                const S dx = S(flip64(n.x, minus)) * area, dy = S(flip64(n.y, minus)) * area;
#pragma unroll
                for (int j = 0; j < 4; ++j) { gx[j] = gx[j] + q[j] * dx; gy[j] = gy[j] + q[j] * dy; }
            }
            den = cvi;
        } else if (v.grad_type == UNS_GRAD_GGFC) {
            for (int k = k0; k < k1; ++k) {
                int f = v.cf[k] & FACE_MASK;
                const S s = v.fasum[f];
                S a[4], b[4];
                f4get(v.fgx[f], a);
                f4get(v.fgy[f], b);
#pragma unroll
                for (int j = 0; j < 4; ++j) { gx[j] = gx[j] + a[j] * s; gy[j] = gy[j] + b[j] * s; }
            }
            den = v.cov[i];
        } else {  // LSQR
            for (int k = k0; k < k1; ++k) {
                int e = v.cf[k], f = e & FACE_MASK;
                const double4 w = v.lsw[f];
                int2 nb = v.fnb[f];
                S qa[4], qb[4];
                f4get(v.qp[nb.x], qa);
                f4get(v.qp[nb.y], qb);
                const bool out = f < v.nfi && (e & SIDE_BIT);
                const S wx = flip64(out ? w.z : w.x, out), wy = flip64(out ? w.w : w.y, out);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const S var = qb[j] - qa[j];
                    gx[j] = gx[j] + var * wx;
                    gy[j] = gy[j] + var * wy;
                }
            }
        }
        if (v.grad_type != UNS_GRAD_LSQR) {
#pragma unroll
            for (int j = 0; j < 4; ++j) { gx[j] = gx[j] / den; gy[j] = gy[j] / den; }
        }
        v.gx[i] = f4(gx);
        v.gy[i] = f4(gy);
    } else {
        f4get(v.gx[i], gx);
        f4get(v.gy[i], gy);
    }
    if (flags & CG_LIM) {
        long long umax[4], umin[4];  // order keys
        S qi[4], ph[4];
        f4get(v.qp[i], qi);
        f4get(v.phi[i], ph);
#pragma unroll
        for (int j = 0; j < 4; ++j) { umax[j] = order_key(qi[j].v); umin[j] = umax[j]; }
        for (int k = k0; k < k1; ++k) {
            int e = v.cf[k], f = e & FACE_MASK;
            double u[4];
            if (f < v.nfi) {
                int2 nb = v.fnb[f];
                d4get(v.qp[(e & SIDE_BIT) ? nb.x : nb.y], u);
            } else {
                int2 p = v.fpt[f];
                double4 a = v.pp[p.x], b = v.pp[p.y];
                u[0] = mean_rare(a.x, b.x); u[1] = mean_rare(a.y, b.y); u[2] = mean_rare(a.z, b.z); u[3] = mean_rare(a.w, b.w);
            }
            // (of two zeros the keys prefer the positive, rmax / rmin the first:
            // the differences from the cell's value drop the sign)
#pragma unroll
            for (int j = 0; j < 4; ++j) extend(u[j], umin[j], umax[j]);
        }
        // phi = min(phi, phi0 of every face): the faces' ratios nr/dr are
        // compared exactly and only the smallest is divided (the minimum of
        // correctly rounded quotients is the rounded minimum), so one
        // division per variable instead of one per face and variable.
        S bn[4], bd[4];
        bool have[4] = {false, false, false, false};
        const double2 c = v.cen[i];
        for (int k = k0; k < k1; ++k) {
            int f = v.cf[k] & FACE_MASK;
            double2 fc = v.fcen[f];
            const S d0 = S(fc.x) - c.x, d1 = S(fc.y) - c.y;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const S D_L = gx[j] * d0 + gy[j] * d1;
                const bool pos = dpos(D_L.v);
                if (pos || dneg(D_L.v)) {
                    // vk_terms with 2 a b and 2 b b scaled after the product
                    // (the same bits unless the product is subnormal, which
                    // terms that ratio_ok accepts do not show)
                    const S a = S(from_key(pos ? umax[j] : umin[j])) - qi[j];
                    const S aa = a * a, ab = a * D_L, t2 = stol2[j];
                    const S nr = aa + twice(ab) + t2, dr = aa + twice(D_L * D_L) + ab + t2;
                    if (!ratio_ok(nr.v, dr.v)) {
                        ph[j] = rmin(ph[j], S(vk_limit_rare(a.v, D_L.v, stol[j])));
                    } else if (!have[j] || ratio_less(nr, dr, bn[j], bd[j])) {
                        bn[j] = nr; bd[j] = dr; have[j] = true;
                    }
                } else {
                    ph[j] = rmin(ph[j], S(1.0));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (have[j]) ph[j] = rmin(ph[j], bn[j] / bd[j]);
        v.phi[i] = f4(ph);
    }
}

// k_cell_grad in the mixed form: the same gathers, face orders and formulas
// with the gradient and the Venkatakrishnan limiter in FP32 on the FP32
// copies.  dt, la and diag come from the FP32 face radii.  The per-cell pack
// (primitives, gradient, phi) is the gradient and limiter state of record in
// this form (phi is a running minimum across iterations); k_unpack_f32
// writes it back to the FP64 arrays when a caller reads them or the handle
// leaves the form.
__global__ void __launch_bounds__(kBlock, 5) k_cell_grad_mixed(CCView v, int flags, double cfl_in) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
    if (flags & CG_DT) {
        float la = 0.f;
        for (int k = k0; k < k1; ++k) la = la + v.flaf[v.cf[k] & FACE_MASK];
        const float cvf = (float)v.cv[i];
        const float dt = (float)cur_cfl(v, inst, cfl_in) * cvf / la;
        v.la[i] = (double)la;
        v.dt[i] = (double)dt;
        v.dcv[i] = (double)(dt / cvf);
        if (flags & CG_DIAG) {
            v.diag[i] = (double)(cvf / dt + 0.75f * la);
            v.diaginv[i] = 1.0 / v.diag[i];
        }
        warp_atomic_min_u64(v, inst, enc_ord((double)dt));
    }
    if (!(flags & (CG_GRAD | CG_LIM))) return;
    const float4 q4 = v.qpf[i];
    const float qi[4] = {q4.x, q4.y, q4.z, q4.w};
    float gx[4], gy[4];
    if (flags & CG_GRAD) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { gx[j] = 0.f; gy[j] = 0.f; }
        if (v.grad_type == UNS_GRAD_GG) {
            for (int k = k0; k < k1; ++k) {
                int e = v.cf[k], f = e & FACE_MASK;
                const float4 na = v.fnaf[f];
                const float4 q = v.fqf[f];
                // outward from this cell: + for the `in` side of an interior face
                const float s = (f < v.nfi && !(e & SIDE_BIT)) ? 1.f : -1.f;
                const float dx = s * (na.x * na.z), dy = s * (na.y * na.z);
                gx[0] += q.x * dx; gx[1] += q.y * dx; gx[2] += q.z * dx; gx[3] += q.w * dx;
                gy[0] += q.x * dy; gy[1] += q.y * dy; gy[2] += q.z * dy; gy[3] += q.w * dy;
            }
            const float r = 1.f / (float)v.cv[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) { gx[j] *= r; gy[j] *= r; }
        } else if (v.grad_type == UNS_GRAD_GGFC) {
            for (int k = k0; k < k1; ++k) {
                int f = v.cf[k] & FACE_MASK;
                const float s = (float)v.fasum[f];
                const double4 a = v.fgx[f], b = v.fgy[f];
                gx[0] += (float)a.x * s; gx[1] += (float)a.y * s; gx[2] += (float)a.z * s; gx[3] += (float)a.w * s;
                gy[0] += (float)b.x * s; gy[1] += (float)b.y * s; gy[2] += (float)b.z * s; gy[3] += (float)b.w * s;
            }
            const float r = 1.f / (float)v.cov[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) { gx[j] *= r; gy[j] *= r; }
        } else {  // LSQR
            for (int k = k0; k < k1; ++k) {
                int e = v.cf[k], f = e & FACE_MASK;
                const float4 w = v.lswf[f];
                const int2 nb = v.fnb[f];
                const float4 a = v.qpf[nb.x], b = v.qpf[nb.y];
                const float d[4] = {b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w};
                if (f < v.nfi && (e & SIDE_BIT)) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { gx[j] -= d[j] * w.z; gy[j] -= d[j] * w.w; }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) { gx[j] += d[j] * w.x; gy[j] += d[j] * w.y; }
                }
            }
        }
    } else {  // limiter alone: the gradient of record
        const float4 a = v.packf[4 * (size_t)i + 1], b = v.packf[4 * (size_t)i + 2];
        gx[0] = a.x; gx[1] = a.y; gx[2] = a.z; gx[3] = a.w;
        gy[0] = b.x; gy[1] = b.y; gy[2] = b.z; gy[3] = b.w;
    }
    const float4 p0 = v.packf[4 * (size_t)i + 3];
    float ph[4] = {p0.x, p0.y, p0.z, p0.w};
    if (flags & CG_LIM) {
        float tol[4], umax[4], umin[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float hi = (float)dec_ord(v.minmax[8 * inst + j]), lo = (float)dec_ord(v.minmax[8 * inst + 4 + j]);
            tol[j] = 0.05f * (hi - lo);
            tol[j] = tol[j] * tol[j];
            umax[j] = qi[j];
            umin[j] = qi[j];
        }
        for (int k = k0; k < k1; ++k) {
            int e = v.cf[k], f = e & FACE_MASK;
            float4 u;
            if (f < v.nfi) {
                const int2 nb = v.fnb[f];
                u = v.qpf[(e & SIDE_BIT) ? nb.x : nb.y];
            } else {
                u = v.fqf[f];  // the face average of avg_c2v, as limiter.F90 uses on boundary faces
            }
            umax[0] = rmax(umax[0], u.x); umin[0] = rmin(umin[0], u.x);
            umax[1] = rmax(umax[1], u.y); umin[1] = rmin(umin[1], u.y);
            umax[2] = rmax(umax[2], u.z); umin[2] = rmin(umin[2], u.z);
            umax[3] = rmax(umax[3], u.w); umin[3] = rmin(umin[3], u.w);
        }
        for (int k = k0; k < k1; ++k) {
            int e = v.cf[k], f = e & FACE_MASK;
            const float4 gd = v.fgeof[f];
            const float d0 = (e & SIDE_BIT) ? gd.z : gd.x, d1 = (e & SIDE_BIT) ? gd.w : gd.y;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float D_L = gx[j] * d0 + gy[j] * d1;
                float phi0 = 1.f;
                if (D_L != 0.f) {  // limiter.F90:286-294 with a = (umax or umin) - qi, b = D_L
                    const float a = (D_L > 0.f ? umax[j] : umin[j]) - qi[j];
                    const float nr = a * a + 2.f * a * D_L + tol[j];
                    const float dr = a * a + 2.f * D_L * D_L + a * D_L + tol[j];
                    phi0 = __fdividef(nr, dr);
                }
                ph[j] = rmin(ph[j], phi0);
            }
        }
    }
    v.packf[4 * (size_t)i] = q4;
    v.packf[4 * (size_t)i + 1] = make_float4(gx[0], gx[1], gx[2], gx[3]);
    v.packf[4 * (size_t)i + 2] = make_float4(gy[0], gy[1], gy[2], gy[3]);
    v.packf[4 * (size_t)i + 3] = make_float4(ph[0], ph[1], ph[2], ph[3]);
}

// k_face_prim_spec + k_cell_grad_mixed for the Green-Gauss gradient of an
// inviscid flow in the mixed form, as one gather per cell.  Each of the
// cell's faces is described by a cell-side record (v.sideg / v.sidei, in the
// cell's face order): the unit normal signed outward as Gradient_GG counts it,
// the centre-to-midpoint offset of this side, the cell across the face (-1 on
// a boundary) and the face's end points.  The face average and spectral
// radius are formed from the end points' vertex values with the operations of
// k_face_prim_spec (the sign of the normal drops out of |u.n|), so the
// records stream in order and the only gathers are the vertex values and the
// neighbours' primitives.  dt, the gradient, the limiter and the pack are
// those of k_cell_grad_mixed, bit for bit.
__global__ void __launch_bounds__(kBlock, 4) k_cell_grad_side(CCView v, int flags, double cfl_in) {
    // the limiter tolerances of the block's instance (blocks of cells are
    // instance-pure), decoded once per block
    __shared__ float stol[4];
    if ((flags & CG_LIM) && threadIdx.x < 4) {
        const int b = block_inst(v), j = threadIdx.x;
        const float hi = (float)dec_ord(v.minmax[8 * b + j]), lo = (float)dec_ord(v.minmax[8 * b + 4 + j]);
        const float t = 0.05f * (hi - lo);
        stol[j] = t * t;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    const Gas& g = gas_of(v, inst);
    const float gam = (float)(g.gamma);
    const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
    const float4 q4 = v.qpf[i];
    const float qi[4] = {q4.x, q4.y, q4.z, q4.w};
    float gx[4] = {0.f, 0.f, 0.f, 0.f}, gy[4] = {0.f, 0.f, 0.f, 0.f};
    float umax[4] = {qi[0], qi[1], qi[2], qi[3]}, umin[4] = {qi[0], qi[1], qi[2], qi[3]};
    float la = 0.f;
    for (int k = k0; k < k1; ++k) {
        const float4 sg = v.sideg[k];
        const int4 si = v.sidei[k];
        const float area = __int_as_float(si.w);
        const float4 a = v.ppf[si.y], b = v.ppf[si.z];
        const float4 u = si.x >= 0 ? v.qpf[si.x] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 q = make_float4(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z), 0.5f * (a.w + b.w));
        const float a0 = sqrtf(gam * q.w / q.x);
        la = la + area * (fabsf(q.y * sg.x + q.z * sg.y) + a0);
        const float dx = sg.x * area, dy = sg.y * area;
        gx[0] += q.x * dx; gx[1] += q.y * dx; gx[2] += q.z * dx; gx[3] += q.w * dx;
        gy[0] += q.x * dy; gy[1] += q.y * dy; gy[2] += q.z * dy; gy[3] += q.w * dy;
        const float4 w = si.x >= 0 ? u : q;  // the face average on a boundary face, as limiter.F90 uses
        umax[0] = rmax(umax[0], w.x); umin[0] = rmin(umin[0], w.x);
        umax[1] = rmax(umax[1], w.y); umin[1] = rmin(umin[1], w.y);
        umax[2] = rmax(umax[2], w.z); umin[2] = rmin(umin[2], w.z);
        umax[3] = rmax(umax[3], w.w); umin[3] = rmin(umin[3], w.w);
    }
    const float cvf = (float)(v.cv[i]);
    if (flags & CG_DT) {
        const float dt = (float)(cur_cfl(v, inst, cfl_in)) * cvf / la;
        const double dtd = (double)(dt);
        v.la[i] = (double)(la);
        v.dt[i] = dtd;
        v.dcv[i] = (double)(dt / cvf);
        if (flags & CG_DIAG) {
            v.diag[i] = (double)(cvf / dt + 0.75f * la);
            v.diaginv[i] = 1.0 / v.diag[i];
        }
        warp_atomic_min_u64(v, inst, enc_ord(dtd));
    }
    {
        const float r = 1.f / cvf;
#pragma unroll
        for (int j = 0; j < 4; ++j) { gx[j] *= r; gy[j] *= r; }
    }
    const float4 p0 = v.packf[4 * (size_t)i + 3];
    float ph[4] = {p0.x, p0.y, p0.z, p0.w};
    if (flags & CG_LIM) {
        const float tol[4] = {stol[0], stol[1], stol[2], stol[3]};
        for (int k = k0; k < k1; ++k) {
            const float4 sg = v.sideg[k];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float D_L = gx[j] * sg.z + gy[j] * sg.w;
                float phi0 = 1.f;
                if (D_L != 0.f) {  // limiter.F90:286-294 with a = (umax or umin) - qi, b = D_L
                    const float a = (D_L > 0.f ? umax[j] : umin[j]) - qi[j];
                    const float nr = a * a + 2.f * a * D_L + tol[j];
                    const float dr = a * a + 2.f * D_L * D_L + a * D_L + tol[j];
                    phi0 = __fdividef(nr, dr);
                }
                ph[j] = rmin(ph[j], phi0);
            }
        }
    }
    v.packf[4 * (size_t)i] = q4;
    v.packf[4 * (size_t)i + 1] = make_float4(gx[0], gx[1], gx[2], gx[3]);
    v.packf[4 * (size_t)i + 2] = make_float4(gy[0], gy[1], gy[2], gy[3]);
    v.packf[4 * (size_t)i + 3] = make_float4(ph[0], ph[1], ph[2], ph[3]);
}

// Convective face flux (fvresidual.F90:27-171).  Boundary faces also write
// their ghost cell (farfield: Riemann state; wall: slip / no-slip mirror).
// R = double for the FP64 form, float for FP32 face arithmetic.
template <class R>
__device__ __forceinline__ bool flux_dispatch(const Gas& g, R nx, R ny, R area, V4<R>& ql, V4<R>& qr, V4<R>& F) {
    return face_flux<R>(g, nx, ny, area, ql, qr, F);
}

// Boundary face f of cell `in` (fvresidual.F90:27-101): the reconstructed
// state of the cell (the FP32 pack of record in the mixed form), the farfield
// or wall ghost from it and, for a wall, from the cell's conserved state cin;
// writes the ghost cell, the wall force and the flux, and returns the flux.
template <class R>
__device__ __forceinline__ double4 bnd_face_flux(const CCView& v, const Gas& g, int f, int in, const double cin4[4]) {
    const double2 n = v.fn[f];
    const double area = v.farea[f];
    const double2 fc = v.fcen[f];
    const double2 ci = v.cen[in];
    F64 qi[4], gxi[4], gyi[4], phi_i[4];
    if constexpr (std::is_same<R, float>::value) {
        const float4* A = v.packf + 4 * (size_t)in;
        const float4 a0 = A[0], a1 = A[1], a2 = A[2], a3 = A[3];
        qi[0] = a0.x; qi[1] = a0.y; qi[2] = a0.z; qi[3] = a0.w;
        gxi[0] = a1.x; gxi[1] = a1.y; gxi[2] = a1.z; gxi[3] = a1.w;
        gyi[0] = a2.x; gyi[1] = a2.y; gyi[2] = a2.z; gyi[3] = a2.w;
        phi_i[0] = a3.x; phi_i[1] = a3.y; phi_i[2] = a3.z; phi_i[3] = a3.w;
    } else {
        f4get(v.qp[in], qi);
        f4get(v.gx[in], gxi);
        f4get(v.gy[in], gyi);
        f4get(v.phi[in], phi_i);
    }
    const int bc = v.fbc[f];
    const F64 d0 = F64(fc.x) - ci.x, d1 = F64(fc.y) - ci.y;
    V4<F64> qcl;
#pragma unroll
    for (int j = 0; j < 4; ++j) qcl[j] = qi[j] + phi_i[j] * (gxi[j] * d0 + gyi[j] * d1);
    double4 Fd = make_double4(0.0, 0.0, 0.0, 0.0);
    if (bc == 2001 || bc == 1001) {
        const V4<F64> cin = {cin4[0], cin4[1], cin4[2], cin4[3]};
        CCBnd<F64> b = cc_boundary<F64, typename Arith<R>::type, F64>(g, bc, n.x, n.y, area, qcl, cin, g.u_inf, g.v_inf);
        if (!b.ok) set_err(v.err, UNS_ERR_NEG_SOUND_SPEED, f);
        Fd = make_double4(b.F[0].v, b.F[1].v, b.F[2].v, b.F[3].v);
        const int out = v.fnb[f].y;
        v.qc[out] = make_double4(b.gq[0].v, b.gq[1].v, b.gq[2].v, b.gq[3].v);
        v.qp[out] = make_double4(b.gp[0].v, b.gp[1].v, b.gp[2].v, b.gp[3].v);
        v.qT[out] = b.gT.v;
        v.qpf[out] = make_float4(narrow(b.gp[0].v), narrow(b.gp[1].v), narrow(b.gp[2].v), narrow(b.gp[3].v));
        if (bc == 1001) v.fwall[f - v.nfi] = make_double2(Fd.z, Fd.w);
    }
    if constexpr (std::is_same<R, float>::value)  // values of FP32 arithmetic
        v.fFf()[f] = make_float4(narrow(Fd.x), narrow(Fd.y), narrow(Fd.z), narrow(Fd.w));
    else
        v.fF[f] = Fd;
    return Fd;
}

// FP64 form, 4.2 M cells: 3.85 -> 1.67 ms.  It was bound by the FP64 unit
// (228 operations and 14 divisions and square roots per face); now its sums
// alone are there (100 instructions, 6.4 k cycles per warp) and its products,
// divisions, square roots and halvings on the integer pipe (3 400 instructions,
// 6.8 k cycles).  What remains above the longer of the two is instruction fetch
// (6 200 instructions per face, each run once per warp; ncu: 3.2 of 12 stall
// cycles per issue) and latency at six warps per sub-partition (80 registers;
// at 124 and four warps 1.79 ms).
// One thread per face; the first blocks take the boundary faces, whose FP64
// ghost arithmetic is the longest per thread, so that they run beside the
// interior faces instead of after them.
template <class R>
__global__ void __launch_bounds__(std::is_same<R, float>::value ? 512 : kBlock, std::is_same<R, float>::value ? 2 : 3) k_face_conv(CCView v) {
    const int bs = blockDim.x;
    const int nbb = (v.nbf + bs - 1) / bs;
    const bool bnd = (int)blockIdx.x < nbb;
    const int f = bnd ? v.nfi + blockIdx.x * bs + threadIdx.x : (blockIdx.x - nbb) * bs + threadIdx.x;
    if (f >= (bnd ? v.nof : v.nfi)) return;
    const int inst = face_inst(v, f);
    if (stopped(v, inst)) return;
    const Gas& g = gas_of(v, inst);
    const int2 nb = v.fnb[f];
    if (bnd) {
        double cin[4] = {0.0, 0.0, 0.0, 0.0};
        if (v.fbc[f] == 1001) d4get(v.qc[nb.x], cin);
        bnd_face_flux<R>(v, g, f, nb.x, cin);
        return;
    }
    if constexpr (std::is_same<R, float>::value) {  // interior face of the mixed form: FP32 packs and geometry only
        const float4* A = v.packf + 4 * (size_t)nb.x;
        const float4* B = v.packf + 4 * (size_t)nb.y;
        const float4 qa = A[0], ga = A[1], ha = A[2], pa = A[3];
        const float4 qb = B[0], gb = B[1], hb = B[2], pb = B[3];
        const float4 d = v.fgeof[f], na = v.fnaf[f];
        const float zhi = 1.f / 3.f, zlo = 1.f - 1.f / 3.f;
        const float qi[4] = {qa.x, qa.y, qa.z, qa.w}, qo[4] = {qb.x, qb.y, qb.z, qb.w};
        const float gxi[4] = {ga.x, ga.y, ga.z, ga.w}, gyi[4] = {ha.x, ha.y, ha.z, ha.w};
        const float gxo[4] = {gb.x, gb.y, gb.z, gb.w}, gyo[4] = {hb.x, hb.y, hb.z, hb.w};
        const float phi_i[4] = {pa.x, pa.y, pa.z, pa.w}, phi_o[4] = {pb.x, pb.y, pb.z, pb.w};
        V4<float> ql, qr, F;
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // recon (fvresidual.F90:235-247)
            const float beta = qo[j] - qi[j];
            ql[j] = qi[j] + 0.5f * phi_i[j] * (zhi * beta + zlo * (gxi[j] * d.x + gyi[j] * d.y));
            qr[j] = qo[j] + 0.5f * phi_o[j] * (zhi * -beta + zlo * (gxo[j] * d.z + gyo[j] * d.w));
        }
        bool ok = flux_dispatch<float>(g, na.x, na.y, na.z, ql, qr, F);
        if (!ok) set_err(v.err, UNS_ERR_NEG_SOUND_SPEED, f);
        v.fFf()[f] = make_float4(F[0], F[1], F[2], F[3]);
    } else {
        const int in = nb.x, out = nb.y;
        const double2 n = v.fn[f];
        const double area = v.farea[f];
        const double2 fc = v.fcen[f];
        const double2 ci = v.cen[in], co = v.cen[out];
        F64I qi[4], gxi[4], gyi[4], phi_i[4], qo[4], gxo[4], gyo[4], phi_o[4];
        f4get(v.qp[in], qi);
        f4get(v.gx[in], gxi);
        f4get(v.gy[in], gyi);
        f4get(v.phi[in], phi_i);
        f4get(v.qp[out], qo);
        f4get(v.gx[out], gxo);
        f4get(v.gy[out], gyo);
        f4get(v.phi[out], phi_o);
        const F64I zhi = 1.0 / 3.0, zlo = 1.0 - 1.0 / 3.0;
        const F64I dl0 = F64I(fc.x) - ci.x, dl1 = F64I(fc.y) - ci.y;
        const F64I dr0 = F64I(fc.x) - co.x, dr1 = F64I(fc.y) - co.y;
        V4<F64I> ql, qr, F;
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // recon (fvresidual.F90:235-247); the two sides' beta differ in sign alone
            const F64I zb = zhi * (qo[j] - qi[j]);
            F64I alfa = gxi[j] * dl0 + gyi[j] * dl1;
            ql[j] = qi[j] + half(phi_i[j]) * (zb + zlo * alfa);
            alfa = gxo[j] * dr0 + gyo[j] * dr1;
            qr[j] = qo[j] + half(phi_o[j]) * (zlo * alfa - zb);
        }
        bool ok = flux_dispatch<F64I>(g, n.x, n.y, area, ql, qr, F);
        if (!ok) set_err(v.err, UNS_ERR_NEG_SOUND_SPEED, f);
        v.fF[f] = make_double4(F[0].v, F[1].v, F[2].v, F[3].v);
    }
}

// Sutherland viscosity of an interior cell (viscous_flux.F90:20-22,127-141).
__device__ __forceinline__ void cell_mul(const CCView& v, int i) {
    if (i >= v.noc) return;
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    const Gas& g = gas_of(v, inst);
    double4 c = v.qc[i];
    const PrimT<F64I> P = con2prim_t<F64I>(g, c.x, c.y, c.z, c.w);
    const F64I s0 = F64I(g.T_infd) / g.SCONST;
    const F64I num = F64I(1.0) + s0, den = P.t + s0;
    // t^1.5 as t sqrt(t): two correctly rounded operations, each half a unit
    // in the last place of its own result, together below 1.3 of t^1.5's
    // (1.2845 at t = 0x1.945ff5c063268p+0; pow's bound is two), without pow's
    // 100 instructions on the FP64 unit (262 k cells: 73 -> 13 us).  What pow
    // makes of t <= 0 stays pow's.
    const F64I t15 = dpos(P.t.v) ? P.t * sqrt(P.t) : F64I(pow_rare(P.t.v, 1.5));
    v.mul[i] = ((num / den) * t15).v;
}
__global__ void __launch_bounds__(kBlock) k_cell_mul(CCView v) { cell_mul(v, blockIdx.x * blockDim.x + threadIdx.x); }

// The wall faces' convective fluxes and ghosts (all: every boundary face's),
// and beside them (with_mul) every cell's viscosity: the wall faces' long
// chains take the first one-warp blocks, the cells run under them (laminar
// 512x256: 31 + 13 -> 29 us).
template <class R>
__global__ void __launch_bounds__(32) k_wall_faces(CCView v, int with_mul, int all) {
    const int nwb = (v.nbf + 31) / 32;
    if ((int)blockIdx.x >= nwb) {
        if (with_mul) cell_mul(v, (blockIdx.x - nwb) * 32 + threadIdx.x);
        return;
    }
    const int f = v.nfi + blockIdx.x * 32 + threadIdx.x;
    if (f >= v.nof || (!all && v.fbc[f] != 1001)) return;
    const int inst = face_inst(v, f);
    if (stopped(v, inst)) return;
    const int in = v.fnb[f].x;
    double cin[4];
    d4get(v.qc[in], cin);
    bnd_face_flux<R>(v, gas_of(v, inst), f, in, cin);
}

// Laminar viscous face flux (viscous_flux.F90:30-76), stored as flux*area.
__global__ void __launch_bounds__(kBlock) k_face_visc(CCView v) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= v.nof) return;
    const int inst = face_inst(v, f);
    if (stopped(v, inst)) return;
    const Gas& g = gas_of(v, inst);
    int2 nb = v.fnb[f];
    double2 n = v.fn[f];
    double area = v.farea[f];
    typedef F64I S;
    const S mu = (nb.y < v.noc) ? half(S(v.mul[nb.x]) + v.mul[nb.y]) : S(v.mul[nb.x]);
    v.fmu[f] = mu.v;
    const double4 q = v.fq[f];
    const double4 a = v.fgx[f], b = v.fgy[f];
    const double2 t = v.fgT[f];
    const S uvel = q.y, vvel = q.z;
    const S ux = a.y, uy = b.y, vx = a.z, vy = b.z;
    const S two_third = 2.0 / 3.0;
    const S tauxx = two_third * (twice(ux) - vy);
    const S tauxy = uy + vx;
    const S tauyy = two_third * (twice(vy) - ux);
    const S factor = (S(g.gamma) - 1.0) * g.m_inf * g.m_inf * g.prandtl;
    const S qx = -(S(t.x) / factor), qy = -(S(t.y) / factor);
    const S mr = mu / g.rey;
    const S f1 = mr * ((uvel * tauxx + vvel * tauxy - qx) * n.x + (uvel * tauxy + vvel * tauyy - qy) * n.y);
    const S f3 = mr * (tauxx * n.x + tauxy * n.y);
    const S f4_ = mr * (tauxy * n.x + tauyy * n.y);
    const double V2 = (f3 * area).v, V3 = (f4_ * area).v;
    v.fV[f] = make_double4((f1 * area).v, 0.0, V2, V3);
    if (f >= v.nfi) v.fwallv[f - v.nfi] = (v.fbc[f] == 1001) ? make_double2(V2, V3) : make_double2(0.0, 0.0);
}

// A face's stored flux: FP64, or in the mixed form the FP32 values that its
// arithmetic gave (half the bytes of writing them as FP64, and the conversion
// on the integer pipe of the reader instead of the FP64 unit of the writer).
__device__ __forceinline__ double4 widen4(const float4& F) { return make_double4(widen(F.x), widen(F.y), widen(F.z), widen(F.w)); }
template <class R>
__device__ __forceinline__ double4 stored_flux(const CCView& v, int f) {
    if constexpr (std::is_same<R, float>::value) return widen4(v.fFf()[f]);
    else return v.fF[f];
}

// Residual gather in the reference's accumulation order, optionally fused
// with one RK3 stage (main.F90:92-101) and the block partials of the norm.
// FP64 form, 4.2 M cells: 0.48 -> 0.20 ms (60 FP64 instructions per cell -> 25:
// products on the integer pipe, the sum's first term and stage 1's weights 0
// and 1 dropped); k_begin 0.32 -> 0.13 ms alike.
__device__ __forceinline__ void add4(double r[4], const double4& a) { r[0] = r[0] + a.x; r[1] = r[1] + a.y; r[2] = r[2] + a.z; r[3] = r[3] + a.w; }

// The same on F64 or F64I, the sign by a flip of the operand's sign bit.
template <class S>
__device__ __forceinline__ void signed_add4(S r[4], const double4& a, bool minus) {
    r[0] = r[0] + S(flip64(a.x, minus));
    r[1] = r[1] + S(flip64(a.y, minus));
    r[2] = r[2] + S(flip64(a.z, minus));
    r[3] = r[3] + S(flip64(a.w, minus));
}
// The face fluxes of a cell in the reference's order, boundary faces first;
// the sum's first term (0.0 + F) costs no FP64 instruction.
template <class S>
__device__ __forceinline__ void gather_res(const CCView& v, int k0, int k1, S r[4]) {
    bool first = true;
    auto take = [&](const double4& F, bool minus) {
        if (first) {
            r[0] = zero_plus(flip64(F.x, minus));
            r[1] = zero_plus(flip64(F.y, minus));
            r[2] = zero_plus(flip64(F.z, minus));
            r[3] = zero_plus(flip64(F.w, minus));
            first = false;
        } else {
            signed_add4(r, F, minus);
        }
    };
    r[0] = r[1] = r[2] = r[3] = 0.0;
    for (int k = k0; k < k1; ++k) {
        int f = v.cf[k] & FACE_MASK;
        if (f >= v.nfi) take(v.fF[f], false);
    }
    for (int k = k0; k < k1; ++k) {
        int e = v.cf[k], f = e & FACE_MASK;
        if (f < v.nfi) take(v.fF[f], (e & SIDE_BIT) != 0);
    }
}

__global__ void __launch_bounds__(kBlock) k_cell_res(CCView v, int irk, int partial) {
    if (stopped(v, block_inst(v))) return;  // blocks of cells are instance-pure
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0;
    if (i < v.noc && cell_inst(v, i) >= 0) {
        const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
        F64I r[4];
        gather_res(v, k0, k1, r);
        if (v.laminar) {
            for (int k = k0; k < k1; ++k) {
                int e = v.cf[k], f = e & FACE_MASK;
                signed_add4(r, v.fV[f], !(f < v.nfi && (e & SIDE_BIT)));
            }
        }
        v.res[i] = f4(r);
        if (irk > 0) {
            const F64I dtbyarea = v.dcv[i];  // dt / cv, formed once per time step
            F64I o[4], c[4], q[4];
            f4get(v.qc[i], c);
#pragma unroll
            for (int j = 0; j < 4; ++j) q[j] = c[j] - dtbyarea * r[j];
            if (irk > 1) {  // stage 1: a = 0, b = 1
                const F64I a = rk3_a(irk), b = rk3_b(irk);
                f4get(v.qold[i], o);
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = a * o[j] + b * q[j];
            }
            v.qc[i] = f4(q);
        }
        if (partial) rr = (r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3]).v;
    }
    if (partial) {
        __shared__ double s[kBlock / 32];
        rr = warp_sum(rr);
        if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = rr;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int k = 0; k < kBlock / 32; ++k) t = t + s[k];
            v.partial[blockIdx.x] = t;
        }
    }
}

// The residual gather of the mixed form: FP64 accumulation of the face
// fluxes in the cell's face order (the first face initialises the sum), the
// RK stage with fused multiply-adds, and the FP64 norm partial reduced with
// one FP64 add per cell before the warp stage (FP64 issue, not bytes, bounds
// this kernel on GB300).  walls_done: the mixed form's one-pass step, where
// k_wall_rk3 has already advanced the wall cells through all three
// stages; they only contribute their residual to the norm here.
// The fluxes are read as the FP32 values they are, 16 bytes a face instead of
// 32, and widened here.  4.2 M cells: 153 -> 144 us, of which the 17 FP64
// instructions per cell hold the unit 117 and the memory traffic takes 90; with
// fewer than seven blocks per SM it is slower (six: 162, five: 177).
__global__ void __launch_bounds__(kBlock, 8) k_cell_res_mixed(CCView v, int irk, int partial, int walls_done) {
    if (stopped(v, block_inst(v))) return;  // blocks of cells are instance-pure
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0;
    if (i < v.noc && cell_inst(v, i) >= 0) {
        double r[4] = {0.0, 0.0, 0.0, 0.0};
        if (walls_done && ((__ldg(v.bcell + (i >> 5)) >> (i & 31)) & 1u)) {
            d4get(v.res[i], r);  // a wall cell: its last-stage residual (k_wall_rk3)
        } else {
            const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
            const float4* fF = v.fFf();
            auto add = [&](int k, int e, float4 F) {
                const bool minus = (e & FACE_MASK) < v.nfi && (e & SIDE_BIT);
                const unsigned m = minus ? 0x80000000u : 0u;
                if (k == k0) {
                    const double4 D = widen4(F);
                    r[0] = flip64(D.x, minus); r[1] = flip64(D.y, minus); r[2] = flip64(D.z, minus); r[3] = flip64(D.w, minus);
                } else {
                    F.x = __uint_as_float(__float_as_uint(F.x) ^ m); F.y = __uint_as_float(__float_as_uint(F.y) ^ m);
                    F.z = __uint_as_float(__float_as_uint(F.z) ^ m); F.w = __uint_as_float(__float_as_uint(F.w) ^ m);
                    const double4 D = widen4(F);
                    r[0] = add64(r[0], D.x); r[1] = add64(r[1], D.y); r[2] = add64(r[2], D.z); r[3] = add64(r[3], D.w);
                }
            };
            if (k1 - k0 == 3) {  // a triangle: the three fluxes' gathers in flight together, summed in order
                const int e0 = v.cf[k0], e1 = v.cf[k0 + 1], e2 = v.cf[k0 + 2];
                const float4 F0 = fF[e0 & FACE_MASK], F1 = fF[e1 & FACE_MASK], F2 = fF[e2 & FACE_MASK];
                add(k0, e0, F0);
                add(k0 + 1, e1, F1);
                add(k0 + 2, e2, F2);
            } else {
                for (int k = k0; k < k1; ++k) {
                    const int e = v.cf[k];
                    add(k, e, fF[e & FACE_MASK]);
                }
            }
            if (v.laminar) {
                for (int k = k0; k < k1; ++k) {
                    const int e = v.cf[k], f = e & FACE_MASK;
                    const double4 V = v.fV[f];
                    const double s = (f < v.nfi && (e & SIDE_BIT)) ? 1.0 : -1.0;
                    r[0] = __fma_rn(s, V.x, r[0]); r[1] = __fma_rn(s, V.y, r[1]); r[2] = __fma_rn(s, V.z, r[2]); r[3] = __fma_rn(s, V.w, r[3]);
                }
            }
            v.res[i] = d4(r);
            if (irk > 0) {
                const double D = v.dcv[i];
                double c[4], q[4];
                d4get(v.qc[i], c);
#pragma unroll
                for (int j = 0; j < 4; ++j) q[j] = __fma_rn(-D, r[j], c[j]);
                if (irk > 1) {
                    const double a = rk3_a(irk), b = rk3_b(irk);
                    double o[4];
                    d4get(v.qold[i], o);
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[j] = __fma_rn(a, o[j], mul64(b, q[j]));
                }
                v.qc[i] = d4(q);
            }
        }
        if (partial) rr = __fma_rn(r[3], r[3], __fma_rn(r[2], r[2], __fma_rn(r[1], r[1], mul64(r[0], r[0]))));
    }
    if (partial) {
        __shared__ double sh[kBlock];
        sh[threadIdx.x] = rr;
        __syncthreads();
        if (threadIdx.x < 32) {
            double t = sh[threadIdx.x];
            for (int k = threadIdx.x + 32; k < kBlock; k += 32) t = add64(t, sh[k]);
            t = warp_sum(t);
            if (threadIdx.x == 0) v.partial[blockIdx.x] = t;
        }
    }
}

// The RK stages of an inviscid step in one pass over the cells.  Stage 2's and
// 3's interior and farfield face fluxes equal the first stage's: their
// inputs -- the cells' primitives, gradient and limiter -- are formed once
// per time step (main.F90:62-84) and the farfield ghost is built from them
// alone; only a wall ghost reads the stage's conserved state (slip_wall /
// NoSlip_wall, boundCond.F90:19-81).  So a cell without a wall face keeps the
// first stage's residual in both stages, and a wall cell's residual changes
// only through its own wall faces, whose fluxes its thread recomputes from
// the cell's stage state.  Each stage update and the last stage's norm
// partial are evaluated as in the stage-by-stage sequence (k_cell_res for the
// FP64 form, k_cell_res_mixed for the mixed form), so states, residuals,
// ghosts and norms are the same bit for bit.
template <bool kMixed>
__device__ __forceinline__ void rk_update(int irk, double D, const double o[4], const double r[4], double q[4]) {
    const double a = rk3_a(irk), b = rk3_b(irk);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (kMixed) q[j] = __fma_rn(a, o[j], mul64(b, __fma_rn(-D, r[j], q[j])));
        else if (irk == 2) q[j] = (F64I(a) * F64I(o[j]) + quarter(F64I(q[j]) - F64I(D) * F64I(r[j]))).v;  // b = 1/4
        else q[j] = (F64I(a) * F64I(o[j]) + F64I(b) * (F64I(q[j]) - F64I(D) * F64I(r[j]))).v;
    }
}
__device__ __forceinline__ double norm2(const double r[4]) {
    return (F64I(r[0]) * F64I(r[0]) + F64I(r[1]) * F64I(r[1]) + F64I(r[2]) * F64I(r[2]) + F64I(r[3]) * F64I(r[3])).v;
}

// The residual of wall cell i at stage state q: its wall faces' fluxes
// recomputed (ghosts, wall force and fF written), the other faces' stored;
// with recompute false every face's stored flux (the first stage's sum).
template <class R>
__device__ __forceinline__ void wall_cell_res(const CCView& v, const Gas& g, int i, const double q[4], double r[4],
                                              bool recompute = true) {
    const int k0 = v.cf_off[i], k1 = v.cf_off[i + 1];
    auto flux = [&](int f) -> double4 {
        return (recompute && f >= v.nfi && v.fbc[f] == 1001) ? bnd_face_flux<R>(v, g, f, i, q) : stored_flux<R>(v, f);
    };
    if constexpr (std::is_same<R, float>::value) {  // k_cell_res_mixed's order
        for (int k = k0; k < k1; ++k) {
            const int e = v.cf[k], f = e & FACE_MASK;
            const double4 F = flux(f);
            const double s = (f < v.nfi && (e & SIDE_BIT)) ? -1.0 : 1.0;
            if (k == k0) { r[0] = s * F.x; r[1] = s * F.y; r[2] = s * F.z; r[3] = s * F.w; }
            else { r[0] = __fma_rn(s, F.x, r[0]); r[1] = __fma_rn(s, F.y, r[1]); r[2] = __fma_rn(s, F.z, r[2]); r[3] = __fma_rn(s, F.w, r[3]); }
        }
    } else {  // k_cell_res's order: boundary faces first
        F64 t[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k = k0; k < k1; ++k) {
            const int f = v.cf[k] & FACE_MASK;
            if (f >= v.nfi) signed_add4(t, flux(f), false);
        }
        for (int k = k0; k < k1; ++k) {
            const int e = v.cf[k], f = e & FACE_MASK;
            if (f < v.nfi) signed_add4(t, v.fF[f], (e & SIDE_BIT) != 0);
        }
        r[0] = t[0].v; r[1] = t[1].v; r[2] = t[2].v; r[3] = t[3].v;
    }
}

// The three stages of wall cell i (instance inst), from the stored face fluxes
// (k_face_conv's) in the first and its own wall faces' recomputed ones in the
// other two.
template <class R>
__device__ __forceinline__ void wall_cell_rk3(const CCView& v, int i, int inst) {
    constexpr bool kMixed = std::is_same<R, float>::value;
    double r[4], q[4], o[4];
    d4get(v.qc[i], q);
    d4get(v.qold[i], o);
    const double D = v.dcv[i];
    wall_cell_res<R>(v, gas_of(v, inst), i, q, r, false);
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = kMixed ? __fma_rn(-D, r[j], q[j]) : (F64(q[j]) - F64(D) * F64(r[j])).v;
#pragma unroll 1  // one copy of the long body
    for (int irk = 2; irk <= 3; ++irk) {
        wall_cell_res<R>(v, gas_of(v, inst), i, q, r);
        rk_update<kMixed>(irk, D, o, r, q);
    }
    v.res[i] = d4(r);
    v.qc[i] = d4(q);
}

// The wall cells (v.wcell), one per thread in one-warp blocks so that their
// long FP64 chains spread over the SMs; before k_cell_rk3 or k_cell_res_mixed,
// which advance the other cells, or beside the first (enqueue_rk3).
template <class R>
__global__ void __launch_bounds__(32) k_wall_rk3(CCView v) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= v.nwcell) return;
    const int i = v.wcell[t];
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    wall_cell_rk3<R>(v, i, inst);
}

// The residual of every wall cell (v.wcell) from the stored face fluxes, in
// the residual gather's order (uns_cc_fvresidual's cached form).
template <class R>
__global__ void __launch_bounds__(32) k_wall_res(CCView v) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= v.nwcell) return;
    const int i = v.wcell[t];
    const int inst = cell_inst(v, i);
    if (inst < 0 || stopped(v, inst)) return;
    const double q[4] = {0.0, 0.0, 0.0, 0.0};
    double r[4];
    wall_cell_res<R>(v, gas_of(v, inst), i, q, r, false);
    v.res[i] = d4(r);
}

// Every other cell's three stages and the norm in the FP64 form; the wall cells
// contribute the last-stage residual that k_wall_rk3 stored.  A stage's state
// is the next one's in registers, and the state that began the step is the one
// read (k_begin copied it to qold), so a cell reads its state once and its
// fluxes once: 4.2 M cells 316 us against 150 for the first stage with the
// residual and 204 for the other two, which read residual and both states
// again; 16 384 cells 12.6 us against 10.0 + 4.8 and a launch.
__global__ void __launch_bounds__(kBlock) k_cell_rk3(CCView v) {
    if (stopped(v, block_inst(v))) return;  // blocks of cells are instance-pure
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int inst = i < v.noc ? cell_inst(v, i) : -1;
    double rr = 0.0;
    if (inst >= 0) {
        double r[4] = {0.0, 0.0, 0.0, 0.0};
        if ((__ldg(v.bcell + (i >> 5)) >> (i & 31)) & 1u) {
            if (!v.wpart) d4get(v.res[i], r);  // else k_wall_parts, when both kernels are done
        } else {
            F64I R[4];
            gather_res(v, v.cf_off[i], v.cf_off[i + 1], R);
            v.res[i] = f4(R);
            double o[4], q[4];
            d4get(v.qc[i], o);
            const double D = v.dcv[i];  // dt / cv, formed once per time step
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                r[j] = R[j].v;
                q[j] = (F64I(o[j]) - F64I(D) * R[j]).v;  // stage 1: a = 0, b = 1
            }
            rk_update<false>(2, D, o, r, q);
            rk_update<false>(3, D, o, r, q);
            v.qc[i] = d4(q);
        }
        rr = norm2(r);
    }
    if (v.wpart) {  // one partial per warp (v.ninst == 0)
        rr = warp_sum(rr);
        if ((threadIdx.x & 31) == 0) v.partial[i >> 5] = rr;
    } else {  // k_cell_res's
        __shared__ double s[kBlock / 32];
        rr = warp_sum(rr);
        if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = rr;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int k = 0; k < kBlock / 32; ++k) t = t + s[k];
            v.partial[blockIdx.x] = t;
        }
    }
}

// The norm's per-warp partials of the blocks of cells that hold wall cells
// (v.wblk), from the stored last-stage residuals of all their cells, once
// k_wall_rk3 and the k_cell_rk3 that ran beside it are both done.
__global__ void __launch_bounds__(kBlock) k_wall_parts(CCView v) {
    if (stopped(v)) return;
    const int i = v.wblk[blockIdx.x] * kBlock + threadIdx.x;
    double rr = 0.0;
    if (i < v.noc) {
        double r[4];
        d4get(v.res[i], r);
        rr = norm2(r);
    }
    rr = warp_sum(rr);
    if ((threadIdx.x & 31) == 0) v.partial[i >> 5] = rr;
}

// One Jacobi sweep of cirs (ImpResiSmoothening.F90:27-44).
__global__ void __launch_bounds__(kBlock) k_cirs(CCView v, const double4* src, double4* dst, double eps) {
    if (stopped(v)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k = v.cf_off[i]; k < v.cf_off[i + 1]; ++k) {
        int e = v.cf[k], f = e & FACE_MASK;
        if (f >= v.nfi) continue;
        int2 nb = v.fnb[f];
        add4(s, src[(e & SIDE_BIT) ? nb.x : nb.y]);
    }
    double den = 1.0 / (1.0 + eps * (double)v.nc2c[i]);
    double o[4];
    d4get(v.res0[i], o);
    double r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = (s[j] * eps + o[j]) * den;
    dst[i] = d4(r);
}

__global__ void __launch_bounds__(kBlock) k_rk_stage(CCView v, int irk) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    double a = rk3_a(irk), b = rk3_b(irk);
    double dtbyarea = v.dt[i] / v.cv[i];
    double o[4], c[4], r[4], q[4];
    d4get(v.qold[i], o);
    d4get(v.qc[i], c);
    d4get(v.res[i], r);
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = a * o[j] + b * (c[j] - dtbyarea * r[j]);
    v.qc[i] = d4(q);
}

__global__ void __launch_bounds__(kBlock) k_res_partial(CCView v) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0;
    if (i < v.noc) {
        double4 r = v.res[i];
        rr = r.x * r.x + r.y * r.y + r.z * r.z + r.w * r.w;
    }
    __shared__ double s[kBlock / 32];
    rr = warp_sum(rr);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = rr;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < kBlock / 32; ++k) t = t + s[k];
        v.partial[blockIdx.x] = t;
    }
}

// Deterministic final sum of the block partials; in the graph path it also
// records the history, the first-iteration normalisation and the stop flag
// (solution.F90:159-166, main.F90:57).
// Block partial k: stored, or the sum of its eight warp partials in warp
// order (v.wpart), the warps past the last cell counting zero as they do in
// a block's own sum.
__device__ __forceinline__ double block_partial(const CCView& v, int k) {
    if (!v.wpart) return v.partial[k];
    const int nw = (v.noc + 31) >> 5;
    double t = 0.0;
#pragma unroll
    for (int u = 0; u < kBlock / 32; ++u) t = t + (8 * k + u < nw ? v.partial[8 * k + u] : 0.0);
    return t;
}

__global__ void __launch_bounds__(kBlock) k_res_final(CCView v, int nparts, double* out) {
    const int inst = blockIdx.x;  // one block per instance
    if (stopped(v, inst)) return;
    const int k0 = v.ninst ? v.boff[inst] : 0;
    const int n = v.ninst ? v.boff[inst + 1] - k0 : nparts;
    __shared__ double s[kBlock];
    double t = 0.0;
    // eight partials loaded together, then added in the loop's order
    int k = threadIdx.x;
    for (; k + 7 * kBlock < n; k += 8 * kBlock) {
        double p[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) p[u] = block_partial(v, k0 + k + u * kBlock);
#pragma unroll
        for (int u = 0; u < 8; ++u) t = t + p[u];
    }
    for (; k < n; k += kBlock) t = t + block_partial(v, k0 + k);
    s[threadIdx.x] = t;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) s[threadIdx.x] = s[threadIdx.x] + s[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const int nc = v.ninst ? v.ncell[inst] : v.noc;
        double fres = sqrt(s[0] / (double)nc / 4.0);
        if (out) out[inst] = fres;
        if (!isfinite(fres)) set_err(v.err, UNS_ERR_NAN, inst);
        if (v.iter) {
            int it = v.iter[inst];
            v.fres_hist[(size_t)inst * v.cfl_stride + it] = fres;
            if (it == 0 && v.first_iter) v.fres1[inst] = fres;
            double f1 = v.fres1[inst];
            double nf = (f1 >= 2.220446049250313e-16) ? fres / f1 : fres;
            const double mr = v.ninst ? v.minres[inst] : v.min_res;
            if (!(nf > mr) || v.err->code != 0) {
                v.done[inst] = 1;
                if (v.err->code != 0) v.err->iter = it;
            }
            v.iter[inst] = it + 1;
            // reset the encoded reductions for the next iteration
            for (int j = 0; j < 4; ++j) { v.minmax[8 * inst + j] = 0ULL; v.minmax[8 * inst + 4 + j] = ~0ULL; }
            v.dtmin[inst] = ~0ULL;
        }
    }
}

__global__ void k_reset_minmax(CCView v) {
    const int n = v.ninst ? v.ninst : 1;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        if (stopped(v, k)) continue;
        for (int j = 0; j < 4; ++j) { v.minmax[8 * k + j] = 0ULL; v.minmax[8 * k + 4 + j] = ~0ULL; }
        v.dtmin[k] = ~0ULL;
    }
}

// Sequential wall-force sums in face order (fvresidual.F90:99-100 then
// viscous_flux.F90:73-74).
__global__ void k_forces(CCView v, double* out) {
    double fx = 0.0, fy = 0.0;
#pragma unroll 8
    for (int k = 0; k < v.nbf; ++k)  // unrolled: loads in flight together, sums in order
        if (v.fbc[v.nfi + k] == 1001) { fx = fx + v.fwall[k].x; fy = fy + v.fwall[k].y; }
    if (v.laminar)
#pragma unroll 8
        for (int k = 0; k < v.nbf; ++k)
            if (v.fbc[v.nfi + k] == 1001) { fx = fx - v.fwallv[k].x; fy = fy - v.fwallv[k].y; }
    out[0] = fx;
    out[1] = fy;
}

__global__ void k_check_pos(CCView v) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc || cell_inst(v, i) < 0) return;
    double4 p = v.qp[i];
    if (p.x <= 0.0 || p.w <= 0.0) set_err(v.err, UNS_ERR_NONPOSITIVE, i);
}

__global__ void k_initialize(CCView v, double4 qinf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.ntot) {
        const int inst = cell_inst(v, i);
        v.qc[i] = (v.ninst && inst >= 0) ? v.qinfs[inst] : qinf;
        v.qp[i] = make_double4(0.0, 0.0, 0.0, 0.0); v.qT[i] = 0.0;
        v.qpf[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (i < v.noc) {
        v.phi[i] = make_double4(1.0, 1.0, 1.0, 1.0);
        v.packf[4 * (size_t)i + 3] = make_float4(1.f, 1.f, 1.f, 1.f);
    }
}

// Rebuilds every FP32 copy from the FP64 state, so a handle switched to the
// mixed form between calls starts from consistent copies.
__global__ void k_mirror_f32(CCView v) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.ntot) {
        double4 q = v.qp[i];
        float4 qf = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
        v.qpf[i] = qf;
        if (i < v.noc) {
            double4 a = v.gx[i], b = v.gy[i], c = v.phi[i];
            v.packf[4 * (size_t)i] = qf;
            v.packf[4 * (size_t)i + 1] = make_float4((float)a.x, (float)a.y, (float)a.z, (float)a.w);
            v.packf[4 * (size_t)i + 2] = make_float4((float)b.x, (float)b.y, (float)b.z, (float)b.w);
            v.packf[4 * (size_t)i + 3] = make_float4((float)c.x, (float)c.y, (float)c.z, (float)c.w);
        }
    }
    if (i < v.nof) {
        double4 q = v.fq[i];
        v.fqf[i] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
        v.flaf[i] = (float)v.fla[i];
    }
    if (i < v.nop) {
        double4 q = v.pp[i];
        v.ppf[i] = make_float4((float)q.x, (float)q.y, (float)q.z, (float)q.w);
    }
}

// The gradient and phi of record of the mixed form (the per-cell pack)
// written back to the FP64 arrays.
__global__ void k_unpack_f32(CCView v) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.noc) return;
    const float4* A = v.packf + 4 * (size_t)i;
    const float4 a = A[1], b = A[2], c = A[3];
    v.gx[i] = make_double4(a.x, a.y, a.z, a.w);
    v.gy[i] = make_double4(b.x, b.y, b.z, b.w);
    v.phi[i] = make_double4(c.x, c.y, c.z, c.w);
}

// normal_flux pieces (lusgs.F90:328-359): the flux of a state along (nx, ny).
__device__ __forceinline__ void nflux_prims(const PrimT<F64I>& w, F64I nx, F64I ny, F64I o[4]) {
    const F64I et = w.e * w.rho;
    const F64I un = w.u * nx + w.v * ny;
    o[0] = (et + w.p) * un;
    o[1] = w.rho * un;
    o[2] = o[1] * w.u + w.p * nx;
    o[3] = o[1] * w.v + w.p * ny;
}

// Per LU-SGS call: everything a sweep item needs from a face that does not
// change during the sweeps, contiguous in schedule order:
//   rec[3r]   normal_flux of qold(nb) along the cell's outward normal
//             (lusgs.F90:328-346, the flux1 part)
//   rec[3r+1] (nx, ny, area, omega * la) with the cell's outward normal
//   rec[3r+2] (qold(nb).rho, 0, nb as integer bits, 0)
__global__ void __launch_bounds__(kBlock) k_cc_sweep_prep(CCView v) {
    if (stopped(v)) return;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nrec) return;
    const int c = v.rec_face[r], nb = v.rec_nb[r];
    const double2 n = v.fn[c];
    const bool flip = v.rec_flip[r] != 0;
    const double nx = flip64(n.x, flip), ny = flip64(n.y, flip);
    const double4 q = v.qold[nb];
    const PrimT<F64I> P = con2prim_t<F64I>(v.g, q.x, q.y, q.z, q.w);
    F64I o[4];
    nflux_prims(P, nx, ny, o);
    v.rec[3 * (size_t)r] = f4(o);
    v.rec[3 * (size_t)r + 1] = make_double4(nx, ny, v.farea[c], (F64I(kOmega) * v.fla[c]).v);
    v.rec[3 * (size_t)r + 2] = make_double4(q.y, 0.0, __longlong_as_double((long long)nb), 0.0);
}

// Mixed-precision sweeps (delta form): per record, in FP32, the neighbour's
// old state and primitives and the face geometry (the cell's outward normal):
//   [rho, rho*u, rho*v, E] [u, v, p, u.n] [nx, ny, area, omega*la] [1, nb, 0, 0]
__global__ void __launch_bounds__(kBlock) k_cc_sweep_prep_mixed(CCView v) {
    if (stopped(v)) return;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nrec) return;
    const int c = v.rec_face[r], nb = v.rec_nb[r];
    const double2 n = v.fn[c];
    const bool flip = v.rec_flip[r] != 0;
    const double nx = flip64(n.x, flip), ny = flip64(n.y, flip);
    const double4 q = v.qold[nb];
    const PrimT<F64I> P = con2prim_t<F64I>(v.g, q.x, q.y, q.z, q.w);
    float4* rf = reinterpret_cast<float4*>(v.rec) + 4 * (size_t)r;
    rf[0] = make_float4((float)q.y, (float)q.z, (float)q.w, (float)q.x);
    rf[1] = make_float4((float)P.u, (float)P.v, (float)P.p, (float)(P.u * nx + P.v * ny));
    rf[2] = make_float4((float)nx, (float)ny, (float)v.farea[c], (float)(F64I(kOmega) * v.fla[c]));
    rf[3] = make_float4(1.f, __int_as_float(nb), 0.f, 0.f);
}

SweepArgs sweep_args(const CCView& v, bool mixed) {
    SweepArgs a;
    a.n = v.noc; a.sched = v.sched; a.rec = v.rec; a.rec_src = v.rec_src;
    a.diag = mixed ? v.diaginv : v.diag;
    a.qold = v.qold; a.res = v.res; a.qc = v.qc;
    a.out = v.srec; a.outf = reinterpret_cast<float4*>(v.srec);
    a.outd = reinterpret_cast<double4*>(v.srec + 2 * (size_t)v.noc);
    a.err = v.err; a.wait_cycles = v.wait_cycles; a.ring_cycles = ring_wait_limit(v.wait_cycles); a.skip_code = v.skip_code;
    a.gm1 = v.g.gamma - 1.0;
    return a;
}

// The sweeps (uns_sweep.cuh) over the interior cells.  kPerSM: blocks that an
// SM must have room for.  The FP64 sweep takes 91 registers where it has them
// (one block), and 80 where sweeps of several handles are to share the SMs
// (two; 3 to 5 % longer alone).  The FP32 one takes 76 either way.
template <int kPerSM>
__global__ void __launch_bounds__(kSweepBlock, kPerSM) k_lusgs(SweepArgs a, const int* done, const int* __restrict__ woff) {
    if (done && *((volatile const int*)done) != 0) return;
    sweep_block<true, false>(a, woff);
}
__global__ void __launch_bounds__(kSweepBlock, 1) k_lusgs_mixed(SweepArgs a, const int* done, const int* __restrict__ woff) {
    if (done && *((volatile const int*)done) != 0) return;
    sweep_block<true, true>(a, woff);
}

}  // namespace

// ====================================================================== handle

namespace {

// The handle's report (h->v.err leads it), after all that the stream holds.
int read_report(uns_cc_handle* h, DevReport* r) {
    UNS_CUDA(cudaMemcpyAsync(r, h->v.err, sizeof(DevReport), cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

// The device error e, if it is one: its message set, the device's cleared.
int take_dev_err(uns_cc_handle* h, const DevErr& e) {
    if (e.code != 0) {
        const char* what = e.code == UNS_ERR_NEG_SOUND_SPEED ? "Roe scheme: sonic speed is negative at face "
                           : e.code == UNS_ERR_NONPOSITIVE  ? "Density/pressure is negative at cell "
                           : e.code == UNS_ERR_MESH         ? "ggfc,gradtrixy: -ve area at face "
                           : e.code == UNS_ERR_TIMEOUT      ? "bounded device wait timed out in block "
                                                            : "device error at ";
        set_last_error(std::string(what) + std::to_string(e.index));
        int code = e.code;
        DevErr z = {0, 0, 0, 0};
        h->ghosts_set = true;  // a boundary face that raised it raises it again in the next call
        UNS_CUDA(cudaMemcpyAsync(h->v.err, &z, sizeof(DevErr), cudaMemcpyHostToDevice, h->stream));
        UNS_CUDA(cudaStreamSynchronize(h->stream));
        return code;
    }
    return UNS_OK;
}

int check_dev_err(uns_cc_handle* h) {
    DevReport r;
    const int rc = read_report(h, &r);
    return rc ? rc : take_dev_err(h, r.err);
}

void launch_cfg(int n, dim3& g, dim3& b) { b = dim3(kBlock); g = dim3(std::max(1, nblocks(n))); }

#define LAUNCH(kern, n, ...)                                                         \
    do {                                                                             \
        dim3 g_, b_;                                                                 \
        launch_cfg((n), g_, b_);                                                     \
        kern<<<g_, b_, 0, h->stream>>>(__VA_ARGS__);                                 \
        UNS_CUDA(cudaGetLastError());                                                \
    } while (0)

int enqueue_minmax(uns_cc_handle* h, CCView& v) {
    k_reset_minmax<<<1, 32, 0, h->stream>>>(v);
    UNS_CUDA(cudaGetLastError());
    LAUNCH(k_begin, v.ntot, v, (int)BEGIN_MINMAX);
    return UNS_OK;
}

// k_face_conv's grid: the boundary faces' blocks, then the interior faces'.
#define LAUNCH_FACE_CONV(R, v)                                                                     \
    do {                                                                                           \
        const int bs_ = face_bs<R>(h, (v));                                                        \
        const int nb_ = std::max(1, ((v).nbf + bs_ - 1) / bs_ + ((v).nfi + bs_ - 1) / bs_);        \
        k_face_conv<R><<<nb_, bs_, 0, h->stream>>>(v);                                             \
        UNS_CUDA(cudaGetLastError());                                                              \
    } while (0)

// Block size of a per-element kernel whose threads are independent (no
// block-level reduction): kBlock, halved down to one warp while the launch
// would have fewer than two blocks per SM, so that a small mesh spreads its
// FP64 work over every SM sub-partition instead of stacking warps on a few
// SMs (meshes above about 2 x 256 x SMs elements keep kBlock).  The
// per-element arithmetic, and so every result, is the same at any width.
inline int spread_bs(const uns_cc_handle* h, int n) {
    int bs = kBlock;
    while (bs > 32 && (n + bs - 1) / bs < 2 * h->nsm) bs >>= 1;
    return bs;
}

// Block size of k_face_conv: blk_face in the mixed form and where a caller or
// the autotuner has set one.  The FP64 form's code is longer than the
// instruction cache, and the warps of a large block run through it together:
// 256 threads on large meshes (4.2 M cells: 1.67 ms, 1.95 at 64 and 128; 262 k
// cells: 146 us, 156 at 64), 64 where that leaves fewer than four blocks per SM
// and the last of them idle (102 k cells: 74 us, 76 at 256; 16 k: 33, 39).
template <class R>
inline int face_bs(const uns_cc_handle* h, const CCView& v) {
    if (std::is_same<R, float>::value) return v.blk_face;
    if (h->blk_face_set) return std::min(v.blk_face, kBlock);
    int bs = kBlock;
    while (bs > 64 && nblocks(v.nof, bs) < 4 * h->nsm) bs >>= 1;
    return bs;
}

// A launch over n items with block size bs.
#define LAUNCH_BS(kern, n, bs, ...)                                                                \
    do {                                                                                           \
        const int bs_ = (bs);                                                                      \
        kern<<<std::max(1, (int)(((n) + bs_ - 1) / bs_)), bs_, 0, h->stream>>>(__VA_ARGS__);       \
        UNS_CUDA(cudaGetLastError());                                                              \
    } while (0)

#define LAUNCH_SPREAD(kern, n, ...) LAUNCH_BS(kern, (n), spread_bs(h, (n)), __VA_ARGS__)

// k_cell_grad by the size of the launch; LAUNCH_CELL_GRAD: or its FP32 form for
// a handle in the mixed form.
#define LAUNCH_FP64_GRAD(v, flags, cfl)                                                          \
    do {                                                                                       \
        if (spread_bs(h, (v).noc) < kBlock) LAUNCH_SPREAD(k_cell_grad<F64>, (v).noc, (v), (int)(flags), (cfl)); \
        else LAUNCH_SPREAD(k_cell_grad<F64I>, (v).noc, (v), (int)(flags), (cfl));              \
    } while (0)
#define LAUNCH_CELL_GRAD(v, flags, cfl)                                                 \
    do {                                                                               \
        if ((v).mixed) LAUNCH(k_cell_grad_mixed, (v).noc, (v), (int)(flags), (cfl));   \
        else LAUNCH_FP64_GRAD(v, flags, cfl);                                          \
    } while (0)

int enqueue_gradient(uns_cc_handle* h, CCView& v, int extra_flags, double cfl, bool do_reduce) {
    if (v.grad_type == UNS_GRAD_GGFC) LAUNCH(k_face_ggfc, v.nof, v);
    int flags = CG_GRAD | extra_flags | (v.ilimit ? CG_LIM : 0);
    if (v.ilimit && do_reduce) { int rc = enqueue_minmax(h, v); if (rc) return rc; }
    LAUNCH_CELL_GRAD(v, flags, cfl);
    return UNS_OK;
}

double epsirs_of(const uns_cc_handle* h, double cfl) {
    double r = cfl / h->P.cfl_max;
    return std::max(0.25 * (r * r - 1.0), 0.0);
}

// Whether the main loop's RK3 step runs its three stages as one pass over the
// cells (k_cell_rk3): an inviscid flow without a smoothing sweep (a viscous
// stage recomputes the cell gradient and viscosity from the stage's state; a
// smoothing sweep replaces the residual that the pass reuses).
bool rk3_in_one_pass(const uns_cc_handle* h, const CCView& v, double cfl) {
    const double eps = v.irs ? epsirs_of(h, cfl) : 0.0;
    return h->P.time_mode == UNS_TIME_RK3 && !v.laminar && !(v.irs && eps > 0.0);
}

// Whether the step forms the face averages and radii inside the cell
// gradient pass (k_cell_grad_side): the mixed form with the Green-Gauss
// gradient of an inviscid flow under RK3 (the LU-SGS prep reads the FP64 face
// radii that k_face_prim_spec writes).
bool grad_by_sides(const uns_cc_handle* h, const CCView& v) {
    return v.mixed && v.sideg != nullptr && h->P.time_mode == UNS_TIME_RK3;
}

// The wall faces' convective fluxes and ghosts, with_mul the cells' viscosity
// too.  (A farfield face's flux and ghost follow from the reconstructed state;
// all: they are formed again all the same.)
int enqueue_wall_faces(uns_cc_handle* h, CCView& v, bool with_mul, bool all = false) {
    const int nb = (v.nbf + 31) / 32 + (with_mul ? (v.noc + 31) / 32 : 0);
    if (nb == 0) return UNS_OK;
    if (v.mixed) k_wall_faces<float><<<nb, 32, 0, h->stream>>>(v, with_mul, all);
    else k_wall_faces<double><<<nb, 32, 0, h->stream>>>(v, with_mul, all);
    UNS_CUDA(cudaGetLastError());
    return UNS_OK;
}

// uns_cc_fvresidual when only the wall faces' fluxes can have changed since
// the last call that computed every face (same primitives, gradient and
// limiter; the reference main loop's RK stages 2 and 3): those fluxes and the
// wall cells' residuals; every other cell keeps the residual it has.  The
// other boundary faces give what they gave, which their ghost rows still hold
// unless set_state wrote them (ghosts_set): then they run too.
int enqueue_wall_res(uns_cc_handle* h, CCView& v) {
    int rc = enqueue_wall_faces(h, v, false, h->ghosts_set);
    if (rc) return rc;
    if (v.nbf > 0 && v.nwcell > 0) {
        const int nb = (v.nwcell + 31) / 32;
        if (v.mixed) k_wall_res<float><<<nb, 32, 0, h->stream>>>(v);
        else k_wall_res<double><<<nb, 32, 0, h->stream>>>(v);
        UNS_CUDA(cudaGetLastError());
    }
    return UNS_OK;
}

// Whether k_cell_rk3 of this handle runs spread over the SMs with
// per-warp norm partials: one case (no packed instances) on a small mesh.
inline bool rk3_warp_partials(const uns_cc_handle* h, const CCView& v) {
    return v.ninst == 0 && spread_bs(h, v.noc) < kBlock;
}

// k_res_final's view after the FP64 one-pass RK stages.
inline CCView final_view(const uns_cc_handle* h, const CCView& v) {
    CCView w = v;
    w.wpart = rk3_warp_partials(h, v) ? 1 : 0;
    return w;
}

// The wall cells' three stages.
int enqueue_wall_rk(uns_cc_handle* h, CCView& v, cudaStream_t stream) {
    if (v.nwcell == 0) return UNS_OK;
    const int nb = (v.nwcell + 31) / 32;
    if (v.mixed) k_wall_rk3<float><<<nb, 32, 0, stream>>>(v);
    else k_wall_rk3<double><<<nb, 32, 0, stream>>>(v);
    UNS_CUDA(cudaGetLastError());
    return UNS_OK;
}

// The other cells' three stages and the norm's partials, but for those of the
// wall cells' blocks where the pass is spread (enqueue_wall_parts).
int enqueue_cell_rk(uns_cc_handle* h, CCView& v) {
    if (v.mixed) {
        LAUNCH(k_cell_res_mixed, v.noc, v, 1, 1, 1);
    } else if (rk3_warp_partials(h, v)) {
        CCView w = v;
        w.wpart = 1;
        LAUNCH_SPREAD(k_cell_rk3, v.noc, w);
    } else {
        LAUNCH(k_cell_rk3, v.noc, v);
    }
    return UNS_OK;
}

// Those partials, after both kernels.
int enqueue_wall_parts(uns_cc_handle* h, CCView& v) {
    if (v.mixed || v.nwcell == 0 || !rk3_warp_partials(h, v)) return UNS_OK;
    k_wall_parts<<<v.nwblk, kBlock, 0, h->stream>>>(v);
    UNS_CUDA(cudaGetLastError());
    return UNS_OK;
}

// Both.  The wall cells' chain (a thread per cell, 27-40 us at any size) runs on
// a stream of its own beside the other cells' where these leave it room, on the
// meshes that spread their launches: 16 384 cells 114 -> 109 us per iteration.
// On larger ones they fill the chip, the chain gets its turn behind them and the
// partials' launch comes on top (a mixed packed study: 503 -> 510 us).
int enqueue_rk3(uns_cc_handle* h, CCView& v) {
    const bool beside = v.nwcell > 0 && !v.mixed && rk3_warp_partials(h, v);
    if (!beside) {
        const int rc = enqueue_wall_rk(h, v, h->stream);
        return rc ? rc : enqueue_cell_rk(h, v);
    }
    UNS_CUDA(cudaEventRecord(h->fork, h->stream));
    UNS_CUDA(cudaStreamWaitEvent(h->side, h->fork, 0));
    int rc = enqueue_wall_rk(h, v, h->side);
    if (!rc) rc = enqueue_cell_rk(h, v);
    // joined whichever of the two launches failed, so that no capture is left open
    cudaError_t e = cudaEventRecord(h->join, h->side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(h->stream, h->join, 0);
    if (rc) return rc;
    UNS_CUDA(e);
    return enqueue_wall_parts(h, v);
}

// fvresidual as a kernel sequence; irk > 0 fuses that RK stage into the
// residual gather (only when no smoothing sweep sits in between).
// walls_only: the other faces' convective fluxes of the step's first stage
// still hold (same primitives, gradient and limiter).
int enqueue_fvresidual(uns_cc_handle* h, CCView& v, double cfl, int irk, int partial, bool* fused, bool walls_only = false) {
    if (walls_only) {
        int rc = enqueue_wall_faces(h, v, v.laminar != 0);
        if (rc) return rc;
    } else if (h->P.precision == UNS_PREC_MIXED) LAUNCH_FACE_CONV(float, v);
    else LAUNCH_FACE_CONV(double, v);
    if (v.laminar) {
        if (!walls_only) LAUNCH(k_cell_mul, v.noc, v);
        if (v.grad_type != UNS_GRAD_GGFC) {
            CCView w = v;
            w.grad_type = UNS_GRAD_GGFC;
            int rc = enqueue_gradient(h, w, 0, cfl, true);
            if (rc) return rc;
        }
        LAUNCH(k_face_visc, v.nof, v);
    }
    double eps = v.irs ? epsirs_of(h, cfl) : 0.0;
    // With eps == 0 both smoothing sweeps reproduce the residual exactly
    // ((0*x + r) * 1 == r for finite x), so they are launched only for eps > 0.
    bool smooth = v.irs && eps > 0.0;
    *fused = !smooth && irk > 0;
    if (v.mixed) LAUNCH(k_cell_res_mixed, v.noc, v, *fused ? irk : 0, (partial && !smooth) ? 1 : 0, 0);
    else if ((partial && !smooth) || v.ninst) LAUNCH(k_cell_res, v.noc, v, *fused ? irk : 0, (partial && !smooth) ? 1 : 0);
    else LAUNCH_SPREAD(k_cell_res, v.noc, v, *fused ? irk : 0, 0);
    if (smooth) {
        UNS_CUDA(cudaMemcpyAsync(v.res0, v.res, sizeof(double4) * v.noc, cudaMemcpyDeviceToDevice, h->stream));
        LAUNCH(k_cirs, v.noc, v, (const double4*)v.res0, v.restmp, eps);
        LAUNCH(k_cirs, v.noc, v, (const double4*)v.restmp, v.res, eps);
        if (partial) LAUNCH(k_res_partial, v.noc, v);
    }
    return UNS_OK;
}

int enqueue_lusgs(uns_cc_handle* h, CCView& v) {
    const bool mixed = h->P.precision != UNS_PREC_FP64;  // FP32 sweep arithmetic
    if (v.nrec > 0) {
        if (mixed) LAUNCH(k_cc_sweep_prep_mixed, v.nrec, v);
        else LAUNCH(k_cc_sweep_prep, v.nrec, v);
    }
    // re-arm the records
    const long long n2 = 2LL * v.noc;
    if (mixed) {
        k_fill_unset_f<<<std::min<long long>(nblocks(n2), 4096), kBlock, 0, h->stream>>>((float4*)v.srec, n2);
        k_fill_unset<<<std::min<long long>(nblocks(2 * n2), 4096), kBlock, 0, h->stream>>>(v.srec + n2, 2 * n2);
    } else {
        k_fill_unset<<<std::min<long long>(nblocks(5 * n2), 4096), kBlock, 0, h->stream>>>(v.srec, 5 * n2);
    }
    UNS_CUDA(cudaGetLastError());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(h->sweep_blocks);
    cfg.blockDim = dim3(kSweepBlock);
    cfg.dynamicSmemBytes = mixed ? sweep_smem_bytes<true>() : sweep_smem_bytes<false>();
    cfg.stream = h->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const SweepArgs a = sweep_args(v, mixed);
    auto kern = mixed ? k_lusgs_mixed : h->share_sms ? k_lusgs<2> : k_lusgs<1>;
    UNS_CUDA(cudaLaunchKernelEx(&cfg, kern, a, (const int*)v.done, (const int*)h->woff));
    return UNS_OK;
}

// The main-loop body (main.F90:60-115) as one kernel sequence.
int enqueue_iteration(uns_cc_handle* h, CCView& v, double cfl_for_eps) {
    int rc;
    k_reset_minmax<<<1, 32, 0, h->stream>>>(v);
    UNS_CUDA(cudaGetLastError());
    int bflags = BEGIN_PRIM | BEGIN_OLD | BEGIN_POS | (v.ilimit ? BEGIN_MINMAX : 0);
    LAUNCH(k_begin, v.ntot, v, bflags);
    LAUNCH_BS(k_vertex_avg, v.nop, v.blk_vert, v);
    const int gflags = CG_DT | CG_GRAD | (v.ilimit ? CG_LIM : 0) | (h->P.time_mode == UNS_TIME_RK3 ? 0 : CG_DIAG);
    if (grad_by_sides(h, v)) {
        LAUNCH_BS(k_cell_grad_side, v.noc, v.blk_grad, v, gflags, 0.0);
    } else {
        LAUNCH_SPREAD(k_face_prim_spec, v.nof, v);
        if (v.grad_type == UNS_GRAD_GGFC) LAUNCH(k_face_ggfc, v.nof, v);
        LAUNCH_CELL_GRAD(v, gflags, 0.0);
    }
    if (rk3_in_one_pass(h, v, cfl_for_eps)) {
        // The wall cells through all three stages, then every other cell and the
        // norm.  A cell without a wall face has the same residual r in all three
        // stages, and then the RK3 stages (main.F90:92-101, a = 0, 3/4, 1/3;
        // b = 1, 1/4, 2/3) give, with D = dt/cv,
        //   q1 = qold - D r,  q2 = 3/4 qold + 1/4 (q1 - D r) = qold - D r / 2,
        //   q3 = 1/3 qold + 2/3 (q2 - D r) = qold - D r = q1
        // in exact arithmetic; the mixed form keeps the FP64 q1 (it differs from
        // the three rounded stage updates in the last bits, far below the FP32
        // face arithmetic).  The FP64 form evaluates every stage's update in the
        // reference's operation order (k_cell_rk3).
        if (v.mixed) LAUNCH_FACE_CONV(float, v);
        else LAUNCH_FACE_CONV(double, v);
        if ((rc = enqueue_rk3(h, v))) return rc;
        if (!v.mixed) {
            k_res_final<<<std::max(1, v.ninst), kBlock, 0, h->stream>>>(final_view(h, v), h->nparts, nullptr);
            UNS_CUDA(cudaGetLastError());
            return UNS_OK;
        }
    } else if (h->P.time_mode == UNS_TIME_RK3) {
        // A viscous stage with the GG-FC gradient, and a smoothing sweep, keep
        // the primitives, gradient and limiter that the interior and farfield
        // fluxes read (above): stages 2 and 3 recompute the wall faces alone
        // (laminar 512x256: three times 157 us of fluxes and viscosities ->
        // 157 + 2 x 29).
        // With another gradient a viscous stage replaces the cell gradient.
        const bool keep = !v.laminar || v.grad_type == UNS_GRAD_GGFC;
        for (int irk = 1; irk <= 3; ++irk) {
            bool fused = false;
            if ((rc = enqueue_fvresidual(h, v, cfl_for_eps, irk, irk == 3, &fused, keep && irk > 1))) return rc;
            if (!fused) LAUNCH(k_rk_stage, v.noc, v, irk);
        }
    } else {
        bool fused = false;
        if ((rc = enqueue_fvresidual(h, v, cfl_for_eps, 0, 1, &fused))) return rc;
        if ((rc = enqueue_lusgs(h, v))) return rc;
    }
    k_res_final<<<std::max(1, v.ninst), kBlock, 0, h->stream>>>(v, h->nparts, nullptr);
    UNS_CUDA(cudaGetLastError());
    return UNS_OK;
}

}  // namespace

namespace uns {

int cc_check_dev_err(uns_cc_handle* h) { return check_dev_err(h); }

// The RK3 main-loop body of enqueue_iteration / enqueue_fvresidual with the
// limiter frozen (the view's ilimit cleared, so phi keeps its values) and a
// fixed CFL, calling `hook` where the adjoint records its linearisation
// points.  Residual smoothing is not part of it (the caller checks that its
// eps is 0).
int cc_record_iteration(uns_cc_handle* h, double cfl, CCRecHook hook, void* ctx) {
    CCView v = h->v;
    v.ilimit = 0;
    v.cfl_sched = nullptr;
    v.iter = nullptr;
    v.done = nullptr;
    int rc;
    LAUNCH(k_begin, v.ntot, v, (int)(BEGIN_PRIM | BEGIN_OLD | BEGIN_POS));
    LAUNCH_BS(k_vertex_avg, v.nop, v.blk_vert, v);
    LAUNCH_SPREAD(k_face_prim_spec, v.nof, v);
    if (v.grad_type == UNS_GRAD_GGFC) LAUNCH(k_face_ggfc, v.nof, v);
    LAUNCH_FP64_GRAD(v, CG_DT | CG_GRAD, cfl);
    if ((rc = hook(h, REC_AFTER_START, 0, ctx))) return rc;
    for (int irk = 1; irk <= 3; ++irk) {
        if ((rc = hook(h, REC_BEFORE_FACE_CONV, irk, ctx))) return rc;
        LAUNCH_FACE_CONV(double, v);
        if (v.laminar) {
            if ((rc = hook(h, REC_BEFORE_CELL_MUL, irk, ctx))) return rc;
            LAUNCH(k_cell_mul, v.noc, v);
            if (v.grad_type != UNS_GRAD_GGFC) {
                CCView w = v;
                w.grad_type = UNS_GRAD_GGFC;
                LAUNCH(k_face_ggfc, w.nof, w);
                LAUNCH_FP64_GRAD(w, CG_GRAD, cfl);
            }
            LAUNCH(k_face_visc, v.nof, v);
            if ((rc = hook(h, REC_AFTER_FACE_VISC, irk, ctx))) return rc;
        }
        LAUNCH(k_cell_res, v.noc, v, irk, 0);
    }
    return check_dev_err(h);
}

}  // namespace uns

// Gas constants of one case: math + initialize (CCFVM/solution.F90:4-84),
// and its freestream conserved state.
static Gas make_gas(const uns_params* p, double4* qinf) {
    Gas g;
    g.gamma = 1.4;
    g.gamma1 = g.gamma - 1.0;
    double pi = 4.0 * std::atan(1.0);
    double aoa = p->aoa_deg * pi / 180.0;
    double q1 = 1.0, q2 = std::cos(aoa) * 1.0, q3 = std::sin(aoa) * 1.0;
    g.p_inf = 1.0 / (g.gamma * p->m_inf * p->m_inf);
    double q0 = g.p_inf / (g.gamma - 1.0) + 0.5;
    g.r_inf = q1;
    g.a_inf = std::sqrt(g.gamma * g.p_inf / g.r_inf);
    g.u_inf = q2 / q1;
    g.v_inf = q3 / q1;
    g.m_inf = p->m_inf;
    g.znd = 1.0 / (g.gamma * p->m_inf * p->m_inf);
    g.T_infd = 300.0;
    g.SCONST = 110.4;
    g.t_wall = p->t_wall / g.T_infd;
    g.rey = p->rey;
    g.prandtl = 0.72;
    g.vll = (p->flow_type != UNS_FLOW_INVISCID) ? 2.0 * g.gamma / (g.prandtl * p->rey * 0.25) : 0.0;
    g.mref = std::max((double)0.32f, 0.5 * p->m_inf);
    g.flux = p->flux_type;
    g.flow = p->flow_type;
    g.iwall = p->iwall;
    *qinf = make_double4(q0, q1, q2, q3);
    return g;
}

static int create_impl(const uns_cc_mesh* m, const uns_params* p, bool lusgs_schedule, uns_cc_handle** out);
static int grow_schedule(uns_cc_handle* h, int cap);
static int iterate_graph(uns_cc_handle* h, int niter, const double* cfl, int first_iter, double* fres_raw, int* done_iters);

// ====================================================================== C-ABI
extern "C" {

int uns_cc_create(const uns_cc_mesh* m, const uns_params* p, uns_cc_handle** out) {
    return create_impl(m, p, true, out);
}

}  // extern "C"

static int create_impl(const uns_cc_mesh* m, const uns_params* p, bool lusgs_schedule, uns_cc_handle** out) {
    if (!m || !p || !out) { set_last_error("uns_cc_create: null argument"); return UNS_ERR_ARG; }
    *out = nullptr;
    if (m->nop <= 0 || m->noc <= 0 || m->nfi < 0 || m->nbf < 0) { set_last_error("uns_cc_create: bad sizes"); return UNS_ERR_ARG; }
    if (p->flux_type < 0 || p->flux_type > 3 || p->grad_type < 0 || p->grad_type > 2 || p->flow_type < 0 ||
        p->flow_type > 1 || p->time_mode < 0 || p->time_mode > 1 || !(p->m_inf > 0.0) ||
        p->precision < UNS_PREC_FP64 || p->precision > UNS_PREC_MIXED_SWEEP) {
        set_last_error("uns_cc_create: bad parameters");
        return UNS_ERR_ARG;
    }
    const int nop = m->nop, noc = m->noc, nfi = m->nfi, nbf = m->nbf, nof = nfi + nbf, ntot = noc + nbf;
    // Validate indices on the host before anything reaches the device.
    for (int f = 0; f < nof; ++f) {
        bool ok = m->fin[f] >= 0 && m->fin[f] < noc && m->fp1[f] >= 0 && m->fp1[f] < nop && m->fp2[f] >= 0 && m->fp2[f] < nop;
        ok = ok && (f < nfi ? (m->fout[f] >= 0 && m->fout[f] < noc) : (m->fout[f] == noc + (f - nfi)));
        if (!ok) { set_last_error("uns_cc_create: face " + std::to_string(f) + " has an out-of-range index"); return UNS_ERR_MESH; }
    }
    for (int i = 0; i < nop; ++i)
        if (m->v2c_off[i] > m->v2c_off[i + 1]) { set_last_error("uns_cc_create: bad v2c"); return UNS_ERR_MESH; }
    for (int k = 0; k < m->v2c_off[nop]; ++k)
        if (m->v2c[k] < 0 || m->v2c[k] >= ntot) { set_last_error("uns_cc_create: v2c index out of range"); return UNS_ERR_MESH; }
    for (int i = 0; i < noc; ++i)
        for (int k = m->c2f_off[i]; k < m->c2f_off[i + 1]; ++k)
            if (m->c2f[k] < 0 || m->c2f[k] >= nof) { set_last_error("uns_cc_create: c2f index out of range"); return UNS_ERR_MESH; }

    uns_cc_handle* h = new uns_cc_handle();
    h->P = *p;
    int rc = UNS_OK;
    auto fail = [&](int code) { uns_cc_destroy(h); return code; };
    int lowest = 0, highest = 0;
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaDeviceGetStreamPriorityRange(&lowest, &highest) != cudaSuccess ||
        cudaStreamCreateWithPriority(&h->side, cudaStreamNonBlocking, highest) != cudaSuccess ||
        cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming) != cudaSuccess) {
        set_last_error("uns_cc_create: cudaStreamCreate failed (no usable GPU?)");
        return fail(UNS_ERR_CUDA);  // with the streams and events that were created
    }
    {
        int dev = 0, nsm = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            nsm > 0)
            h->nsm = nsm;
    }
    Gas& g = h->g;
    g = make_gas(p, &h->qinf);

    // Host-side derived connectivity.
    std::vector<double2> pxy(nop), cen(ntot), fn(nof), fcen(nof);
    std::vector<int2> fnb(nof), fpt(nof);
    for (int i = 0; i < nop; ++i) pxy[i] = make_double2(m->px[i], m->py[i]);
    for (int i = 0; i < ntot; ++i) cen[i] = make_double2(m->cx[i], m->cy[i]);
    for (int f = 0; f < nof; ++f) {
        fnb[f] = make_int2(m->fin[f], m->fout[f]);
        fpt[f] = make_int2(m->fp1[f], m->fp2[f]);
        fn[f] = make_double2(m->fnx[f], m->fny[f]);
        fcen[f] = make_double2(m->fcx[f], m->fcy[f]);
    }
    std::vector<int> cnt(noc + 1, 0);
    for (int f = 0; f < nof; ++f) { cnt[m->fin[f] + 1]++; if (m->fout[f] < noc) cnt[m->fout[f] + 1]++; }
    for (int i = 0; i < noc; ++i) cnt[i + 1] += cnt[i];
    std::vector<int> cf(cnt[noc]), pos(cnt.begin(), cnt.end() - 1);
    for (int f = 0; f < nof; ++f) {  // ascending face index per cell
        cf[pos[m->fin[f]]++] = f;
        if (m->fout[f] < noc) cf[pos[m->fout[f]]++] = f | SIDE_BIT;
    }
    // LSQ weights (gradient.F90:27-44, 72-78), host-side in the reference's
    // expression order (-ffp-contract=off translation unit).
    std::vector<double4> lsw(nof);
    for (int f = 0; f < nof; ++f) {
        int in = m->fin[f], o = m->fout[f];
        double xc = m->cx[in], yc = m->cy[in], xn = m->cx[o], yn = m->cy[o];
        double dx = xn - xc, dy = yn - yc;
        double r11 = m->r11[in], r12 = m->r12[in], r22 = m->r22[in];
        double alfa1 = dx / r11 / r11;
        double alfa2 = f < nfi ? (dy - dx * r12 / r11) / (r22 * r22) : (dy - dx * r12 / r11) / r22 / r22;
        double wx0 = alfa1 - alfa2 * r12 / r11, wy0 = alfa2, wx1 = 0.0, wy1 = 0.0;
        if (f < nfi) {
            dx = xc - xn; dy = yc - yn;
            r11 = m->r11[o]; r12 = m->r12[o]; r22 = m->r22[o];
            alfa1 = dx / r11 / r11;
            alfa2 = (dy - dx * r12 / r11) / (r22 * r22);
            wx1 = alfa1 - alfa2 * r12 / r11; wy1 = alfa2;
        }
        lsw[f] = make_double4(wx0, wy0, wx1, wy1);
    }
    h->lsq_r.resize((size_t)noc * 3);
    for (int i = 0; i < noc; ++i) { h->lsq_r[3 * i] = m->r11[i]; h->lsq_r[3 * i + 1] = m->r12[i]; h->lsq_r[3 * i + 2] = m->r22[i]; }
    h->fnb_host = fnb;
    // FP32 geometry of the mixed form, rounded once from the FP64 values.
    std::vector<float4> fgeof(nof), fnaf(nof), lswf(nof);
    for (int f = 0; f < nof; ++f) {
        int in = m->fin[f], o = m->fout[f];
        double xl = m->fcx[f] - m->cx[in], yl = m->fcy[f] - m->cy[in];
        double xr = f < nfi ? m->fcx[f] - m->cx[o] : 0.0, yr = f < nfi ? m->fcy[f] - m->cy[o] : 0.0;
        fgeof[f] = make_float4((float)xl, (float)yl, (float)xr, (float)yr);
        fnaf[f] = make_float4((float)m->fnx[f], (float)m->fny[f], (float)m->farea[f], 0.f);
        lswf[f] = make_float4((float)lsw[f].x, (float)lsw[f].y, (float)lsw[f].z, (float)lsw[f].w);
    }
    std::vector<int> rc2f_off(m->c2f_off, m->c2f_off + noc + 1);
    std::vector<int> rc2f(m->c2f, m->c2f + rc2f_off[noc]);

    CCView& v = h->v;
    std::memset(&v, 0, sizeof(v));
    v.nop = nop; v.noc = noc; v.nfi = nfi; v.nbf = nbf; v.nof = nof; v.ntot = ntot;
    v.g = g;
    v.grad_type = p->grad_type; v.ilimit = p->ilimit; v.irs = p->irs;
    v.laminar = p->flow_type == UNS_FLOW_LAMINAR;
    v.cfl_max = p->cfl_max; v.min_res = p->min_res;
    v.mixed = p->precision == UNS_PREC_MIXED;
    // Block sizes of the kernels without block-level reductions, from a
    // measured sweep of 64-512 on the 4.2 M-cell mixed step and the 256-case
    // batch (faces 64, vertices 256, cell gradient 128); UNS_CC_BLOCK_FACE /
    // _VERTEX (64..512) and UNS_CC_BLOCK_GRAD (64..256: a divisor of the
    // 256-cell instance-pure blocks) override them for tuning runs.
    auto block_env = [](const char* name, int def, int hi) {
        const char* e = std::getenv(name);
        const int b = e ? std::atoi(e) : def;
        return (b == 64 || b == 128 || b == 256 || b == 512) && b <= hi ? b : def;
    };
    h->blk_face_set = std::getenv("UNS_CC_BLOCK_FACE") != nullptr;
    v.blk_face = block_env("UNS_CC_BLOCK_FACE", 64, 512);
    v.blk_vert = block_env("UNS_CC_BLOCK_VERTEX", kBlock, 512);
    v.blk_grad = block_env("UNS_CC_BLOCK_GRAD", 128, kBlock);
#define UP(field, vec) if ((rc = h->upload(*(std::remove_const<std::remove_pointer<decltype(v.field)>::type>::type**)&v.field, vec.data(), vec.size()))) return fail(rc)
#define AL(field, n) if ((rc = h->alloc(v.field, (n)))) return fail(rc)
    UP(pxy, pxy); UP(cen, cen);
    { std::vector<double> t(m->cv, m->cv + noc); UP(cv, t); }
    { std::vector<double> t(m->cov, m->cov + noc); UP(cov, t); }
    UP(fnb, fnb); UP(fpt, fpt); UP(fn, fn); UP(fcen, fcen);
    { std::vector<double> t(m->farea, m->farea + nof); UP(farea, t); }
    { std::vector<int> t(m->fbc, m->fbc + nof); UP(fbc, t); }
    UP(lsw, lsw);
    { std::vector<int> t(m->nc2c, m->nc2c + noc); UP(nc2c, t); }
    UP(cf_off, cnt); UP(cf, cf);
    if (p->grad_type == UNS_GRAD_GG && p->flow_type != UNS_FLOW_LAMINAR) {  // cell-side records (k_cell_grad_side)
        std::vector<float4> sg(cf.size());
        std::vector<int4> si(cf.size());
        for (size_t k = 0; k < cf.size(); ++k) {
            const int e = cf[k], f = e & FACE_MASK;
            const bool out_side = f < nfi && (e & SIDE_BIT);
            const float s = (f < nfi && !(e & SIDE_BIT)) ? 1.f : -1.f;  // Gradient_GG's sign (boundary: -1)
            const float4 na = fnaf[f], gd = fgeof[f];
            sg[k] = make_float4(s * na.x, s * na.y, out_side ? gd.z : gd.x, out_side ? gd.w : gd.y);
            const int nbr = f < nfi ? (out_side ? m->fin[f] : m->fout[f]) : -1;
            int area_bits;
            std::memcpy(&area_bits, &na.z, sizeof(int));
            si[k] = make_int4(nbr, m->fp1[f], m->fp2[f], area_bits);
        }
        UP(sideg, sg); UP(sidei, si);
    }
    {  // wall cells: a bit per cell and their list
        std::vector<unsigned> t((noc + 31) / 32, 0u);
        std::vector<int> wc;
        for (int f = nfi; f < nof; ++f) {
            const int c = m->fin[f];
            if (m->fbc[f] == 1001 && c >= 0 && c < noc) t[c >> 5] |= 1u << (c & 31);
        }
        for (int c = 0; c < noc; ++c)
            if ((t[c >> 5] >> (c & 31)) & 1u) wc.push_back(c);
        std::vector<int> wb;
        for (int c : wc)
            if (wb.empty() || wb.back() != c / kBlock) wb.push_back(c / kBlock);
        UP(bcell, t); UP(wcell, wc); UP(wblk, wb);
        v.nwcell = (int)wc.size();
        v.nwblk = (int)wb.size();
    }
    UP(rc2f_off, rc2f_off); UP(rc2f, rc2f);
    { std::vector<int> t(m->v2c_off, m->v2c_off + nop + 1); UP(v2c_off, t); }
    { std::vector<int> t(m->v2c, m->v2c + m->v2c_off[nop]); UP(v2c, t); }
    { std::vector<double> t(m->v2c_wt, m->v2c_wt + m->v2c_off[nop]); UP(v2c_wt, t); }
    AL(qc, ntot); AL(qp, ntot); AL(qT, ntot); AL(qold, noc); AL(res, noc); AL(res0, noc); AL(restmp, noc);
    AL(gx, noc); AL(gy, noc); AL(phi, noc); AL(dt, noc); AL(la, noc); AL(mul, ntot);
    AL(pp, nop); AL(ppT, nop); AL(fq, nof); AL(fqT, nof); AL(fla, nof); AL(fmu, nof);
    AL(fF, nof); AL(fV, nof); AL(fgx, nof); AL(fgy, nof); AL(fgT, nof); AL(fasum, nof);
    AL(fwall, nbf); AL(fwallv, nbf);
    AL(diag, noc); AL(diaginv, noc);
    UP(fgeof, fgeof); UP(fnaf, fnaf); UP(lswf, lswf);
    AL(qpf, ntot); AL(fqf, nof); AL(flaf, nof); AL(packf, 4 * (size_t)noc); AL(ppf, nop); AL(dcv, noc);
    { std::vector<float> t(m->v2c_wt, m->v2c_wt + m->v2c_off[nop]); UP(v2c_wtf, t); }
    AL(minmax, 8); AL(dtmin, 1);
    h->v.wait_cycles = kWaitCycles;
    h->v.skip_code = -1;
    h->nparts = nblocks(noc);
    AL(partial, 8 * (size_t)h->nparts);  // per-warp partials of a small mesh's spread RK pass
    DevReport* report = nullptr;
    if ((rc = h->alloc(report, 1))) return fail(rc);
    v.err = &report->err;
    h->d_scalar = report->scalar;
    if ((rc = h->alloc(h->d_iter, 1))) return fail(rc);
    if ((rc = h->alloc(h->d_done, 1))) return fail(rc);
    if ((rc = h->alloc(h->d_fres1, 1))) return fail(rc);
    // LU-SGS warp schedule on the reference c2f lists.
    if (lusgs_schedule) {
        int maxdeg = 0;
        for (int i = 0; i < noc; ++i) maxdeg = std::max(maxdeg, m->c2f_off[i + 1] - m->c2f_off[i]);
        if (maxdeg > 32) { set_last_error("uns_cc_create: a cell has more than 32 faces"); return fail(UNS_ERR_MESH); }
        if (noc >= (1 << 30)) { set_last_error("uns_cc_create: too many cells"); return fail(UNS_ERR_MESH); }
        int dev = 0, nsm = 0, per = 0;
        if (sweep_allow_smem<false>(k_lusgs<1>) != cudaSuccess || sweep_allow_smem<false>(k_lusgs<2>) != cudaSuccess ||
            sweep_allow_smem<true>(k_lusgs_mixed) != cudaSuccess ||
            cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_lusgs<1>, kSweepBlock, sweep_smem_bytes<false>()) != cudaSuccess || per < 1) {
            set_last_error("uns_cc_create: cannot size the cooperative LU-SGS launch");
            return fail(UNS_ERR_CUDA);
        }
        const int blocks = nsm * std::min(per, kSweepBlocksPerSM);
        // the cell across each c2f face (ghosts >= noc), and whether the face
        // normal points into the cell
        auto other = [&](int i, int f, int* flip) {
            if (m->fout[f] == i) { *flip = 1; return m->fin[f]; }
            *flip = 0;
            return m->fout[f];
        };
        std::vector<int> nbr(m->c2f_off[noc]);
        std::vector<signed char> flip(m->c2f_off[noc]);
        for (int i = 0; i < noc; ++i)
            for (int k = m->c2f_off[i]; k < m->c2f_off[i + 1]; ++k) {
                int fl;
                nbr[k] = other(i, m->c2f[k], &fl);
                flip[k] = (signed char)fl;
            }
        WarpSchedule ws = list_schedule(noc, m->c2f_off, nbr.data(), blocks * kSweepPairs);
        if (!ws.indexable()) { set_last_error("uns_cc_create: too many cells"); return fail(UNS_ERR_MESH); }
        h->sweep_blocks = ws.blocks();
        std::vector<int4> sched(ws.items.size());
        std::vector<int> rf, rn, rl;
        rf.reserve(2 * (size_t)nfi); rn.reserve(2 * (size_t)nfi); rl.reserve(2 * (size_t)nfi);
        for (size_t pos = 0; pos < ws.items.size(); ++pos) {
            const int it = ws.items[pos] >> 1, pass = ws.items[pos] & 1;
            const int first = (int)rf.size();
            ask_ahead(ws, pos, m->c2f_off, nbr.data(), m->c2f, flip.data());
            for (int k = m->c2f_off[it]; k < m->c2f_off[it + 1]; ++k) {
                const int nb = nbr[k];
                const bool take = nb >= 0 && nb < noc && (pass == 0 ? nb < it : nb > it);
                if (!take) continue;
                rf.push_back(m->c2f[k]); rn.push_back(nb); rl.push_back(flip[k]);
            }
            sched[pos] = make_int4(it, pass, first, (int)rf.size() - first);
        }
        v.nrec = (int)rf.size();
        if ((rc = h->upload(h->woff, ws.off.data(), ws.off.size()))) return fail(rc);
        UP(sched, sched); UP(rec_face, rf); UP(rec_nb, rn); UP(rec_flip, rl); UP(rec_src, ws.src);
        AL(rec, 3 * rf.size());
        AL(srec, 10 * (size_t)noc);
    }
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) { set_last_error("uns_cc_create: upload failed"); return fail(UNS_ERR_CUDA); }
    rc = uns_cc_initialize(h);
    if (rc) return fail(rc);
    *out = h;
    return UNS_OK;
#undef UP
#undef AL
}

extern "C" {

int uns_cc_destroy(uns_cc_handle* h) {
    if (!h) return UNS_OK;
    if (h->stream) cudaStreamSynchronize(h->stream);
    cc_adj_free(h);
    if (h->graph) cudaGraphExecDestroy(h->graph);
    for (void* p : h->allocs) cudaFree(p);
    if (h->d_cfl) cudaFree(h->d_cfl);
    if (h->d_hist) cudaFree(h->d_hist);
    if (h->fork) cudaEventDestroy(h->fork);
    if (h->join) cudaEventDestroy(h->join);
    if (h->side) cudaStreamDestroy(h->side);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return UNS_OK;
}

int uns_cc_initialize(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView v = h->v;
    k_initialize<<<nblocks(v.ntot), kBlock, 0, h->stream>>>(v, h->qinf);
    UNS_CUDA(cudaGetLastError());
    UNS_CUDA(cudaMemsetAsync(v.mul, 0, sizeof(double) * v.ntot, h->stream));
    UNS_CUDA(cudaMemsetAsync(v.fmu, 0, sizeof(double) * v.nof, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

int uns_cc_set_state(uns_cc_handle* h, const double* qc) {
    if (!h || !qc) return UNS_ERR_ARG;
    h->ghosts_set = true;
    UNS_CUDA(cudaMemcpyAsync(h->v.qc, qc, sizeof(double4) * h->v.ntot, cudaMemcpyHostToDevice, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

int uns_cc_get_state(uns_cc_handle* h, double* qc) {
    if (!h || !qc) return UNS_ERR_ARG;
    UNS_CUDA(cudaMemcpyAsync(qc, h->v.qc, sizeof(double4) * h->v.ntot, cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

int uns_cc_get_field(uns_cc_handle* h, int field, double* out) {
    if (!h || !out) return UNS_ERR_ARG;
    const CCView& v = h->v;
    if (v.mixed && (field == UNS_CC_GRAD || field == UNS_CC_PHI)) LAUNCH(k_unpack_f32, v.noc, v);
    // the graph step of this form forms the face radii inside k_cell_grad_side
    if (v.mixed && v.sideg && field == UNS_CC_FLA) LAUNCH_SPREAD(k_face_prim_spec, v.nof, v);
    auto d2h = [&](void* dst, const void* src, size_t bytes) {
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, h->stream);
    };
    auto interleave = [&](const double4* a, const double* b, int n, int stride5) -> int {
        std::vector<double4> A(n);
        std::vector<double> B(n);
        UNS_CUDA(d2h(A.data(), a, sizeof(double4) * n));
        UNS_CUDA(d2h(B.data(), b, sizeof(double) * n));
        UNS_CUDA(cudaStreamSynchronize(h->stream));
        for (int i = 0; i < n; ++i) {
            double* o = out + (size_t)i * stride5;
            o[0] = A[i].x; o[1] = A[i].y; o[2] = A[i].z; o[3] = A[i].w; o[4] = B[i];
        }
        return UNS_OK;
    };
    switch (field) {
        case UNS_CC_QC: UNS_CUDA(d2h(out, v.qc, sizeof(double4) * v.ntot)); break;
        case UNS_CC_QP: return interleave(v.qp, v.qT, v.ntot, 5);
        case UNS_CC_QOLD: UNS_CUDA(d2h(out, v.qold, sizeof(double4) * v.noc)); break;
        case UNS_CC_RES: UNS_CUDA(d2h(out, v.res, sizeof(double4) * v.noc)); break;
        case UNS_CC_PHI: UNS_CUDA(d2h(out, v.phi, sizeof(double4) * v.noc)); break;
        case UNS_CC_DT: UNS_CUDA(d2h(out, v.dt, sizeof(double) * v.noc)); break;
        case UNS_CC_LA: UNS_CUDA(d2h(out, v.la, sizeof(double) * v.noc)); break;
        case UNS_CC_FLA: UNS_CUDA(d2h(out, v.fla, sizeof(double) * v.nof)); break;
        case UNS_CC_FMU: UNS_CUDA(d2h(out, v.fmu, sizeof(double) * v.nof)); break;
        case UNS_CC_MUL: UNS_CUDA(d2h(out, v.mul, sizeof(double) * v.noc)); break;
        case UNS_CC_PTPRIM: return interleave(v.pp, v.ppT, v.nop, 5);
        case UNS_CC_FQP: return interleave(v.fq, v.fqT, v.nof, 5);
        case UNS_CC_FWALL: {
            std::vector<double2> A(v.nbf), B(v.nbf);
            UNS_CUDA(d2h(A.data(), v.fwall, sizeof(double2) * v.nbf));
            UNS_CUDA(d2h(B.data(), v.fwallv, sizeof(double2) * v.nbf));
            UNS_CUDA(cudaStreamSynchronize(h->stream));
            for (int b = 0; b < v.nbf; ++b) {
                out[4 * (size_t)b] = A[b].x; out[4 * (size_t)b + 1] = A[b].y;
                out[4 * (size_t)b + 2] = v.laminar ? B[b].x : 0.0; out[4 * (size_t)b + 3] = v.laminar ? B[b].y : 0.0;
            }
            return UNS_OK;
        }
        case UNS_CC_GRAD: {
            std::vector<double4> X(v.noc), Y(v.noc);
            UNS_CUDA(d2h(X.data(), v.gx, sizeof(double4) * v.noc));
            UNS_CUDA(d2h(Y.data(), v.gy, sizeof(double4) * v.noc));
            UNS_CUDA(cudaStreamSynchronize(h->stream));
            for (int i = 0; i < v.noc; ++i) {
                double a[4] = {X[i].x, X[i].y, X[i].z, X[i].w}, b[4] = {Y[i].x, Y[i].y, Y[i].z, Y[i].w};
                for (int j = 0; j < 4; ++j) { out[(size_t)i * 8 + 2 * j] = a[j]; out[(size_t)i * 8 + 2 * j + 1] = b[j]; }
            }
            return UNS_OK;
        }
        case UNS_CC_FGRAD: {
            std::vector<double4> X(v.nof), Y(v.nof);
            std::vector<double2> T(v.nof);
            UNS_CUDA(d2h(X.data(), v.fgx, sizeof(double4) * v.nof));
            UNS_CUDA(d2h(Y.data(), v.fgy, sizeof(double4) * v.nof));
            UNS_CUDA(d2h(T.data(), v.fgT, sizeof(double2) * v.nof));
            UNS_CUDA(cudaStreamSynchronize(h->stream));
            for (int f = 0; f < v.nof; ++f) {
                double a[5] = {X[f].x, X[f].y, X[f].z, X[f].w, T[f].x}, b[5] = {Y[f].x, Y[f].y, Y[f].z, Y[f].w, T[f].y};
                for (int j = 0; j < 5; ++j) { out[(size_t)f * 10 + 2 * j] = a[j]; out[(size_t)f * 10 + 2 * j + 1] = b[j]; }
            }
            return UNS_OK;
        }
        default: set_last_error("uns_cc_get_field: unknown field"); return UNS_ERR_ARG;
    }
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

int uns_cc_set_field(uns_cc_handle* h, int field, const double* in) {
    if (!h || !in) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView& v = h->v;
    switch (field) {
        case UNS_CC_QC:
            UNS_CUDA(cudaMemcpyAsync(v.qc, in, sizeof(double4) * v.ntot, cudaMemcpyHostToDevice, h->stream));
            break;
        case UNS_CC_QP: {
            std::vector<double4> A(v.ntot);
            std::vector<double> B(v.ntot);
            std::vector<float4> F(v.ntot);
            for (int i = 0; i < v.ntot; ++i) {
                const double* o = in + (size_t)i * 5;
                A[i] = make_double4(o[0], o[1], o[2], o[3]);
                B[i] = o[4];
                F[i] = make_float4((float)o[0], (float)o[1], (float)o[2], (float)o[3]);
            }
            UNS_CUDA(cudaMemcpyAsync(v.qp, A.data(), sizeof(double4) * v.ntot, cudaMemcpyHostToDevice, h->stream));
            UNS_CUDA(cudaMemcpyAsync(v.qT, B.data(), sizeof(double) * v.ntot, cudaMemcpyHostToDevice, h->stream));
            UNS_CUDA(cudaMemcpyAsync(v.qpf, F.data(), sizeof(float4) * v.ntot, cudaMemcpyHostToDevice, h->stream));
            UNS_CUDA(cudaStreamSynchronize(h->stream));
            return UNS_OK;
        }
        case UNS_CC_PHI:
            if (v.mixed) LAUNCH(k_unpack_f32, v.noc, v);
            UNS_CUDA(cudaMemcpyAsync(v.phi, in, sizeof(double4) * v.noc, cudaMemcpyHostToDevice, h->stream));
            if (v.mixed) LAUNCH(k_mirror_f32, std::max(std::max(v.ntot, v.nof), v.nop), v);
            break;
        default: set_last_error("uns_cc_set_field: field cannot be set"); return UNS_ERR_ARG;
    }
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    return UNS_OK;
}

int uns_cc_con2prim(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView v = h->v;
    LAUNCH(k_begin, v.noc, v, (int)BEGIN_PRIM);
    return UNS_OK;
}

int uns_cc_avg_c2v(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView v = h->v;
    LAUNCH_BS(k_vertex_avg, v.nop, v.blk_vert, v);
    LAUNCH_SPREAD(k_face_prim_spec, v.nof, v);
    return UNS_OK;
}

int uns_cc_time_step(uns_cc_handle* h, double cfl, double* dtglobal) {
    if (!h) return UNS_ERR_ARG;
    CCView v = h->v;
    h->cfl_cur = cfl;  // cirs of this iteration uses the same CFL
    k_reset_minmax<<<1, 32, 0, h->stream>>>(v);
    UNS_CUDA(cudaGetLastError());
    LAUNCH_CELL_GRAD(v, CG_DT | CG_DIAG, cfl);
    if (dtglobal) {
        unsigned long long e = 0;
        UNS_CUDA(cudaMemcpyAsync(&e, v.dtmin, 8, cudaMemcpyDeviceToHost, h->stream));
        UNS_CUDA(cudaStreamSynchronize(h->stream));
        *dtglobal = std::min(1.0e20, dec_ord(e));
    }
    return UNS_OK;
}

int uns_cc_save_old(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    CCView v = h->v;
    LAUNCH(k_begin, v.noc, v, (int)BEGIN_OLD);
    return UNS_OK;
}

int uns_cc_gradient(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView v = h->v;
    return enqueue_gradient(h, v, 0, 0.0, true);
}

int uns_cc_limit(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    ++h->flux_gen;
    CCView v = h->v;
    int rc = enqueue_minmax(h, v);
    if (rc) return rc;
    LAUNCH_CELL_GRAD(v, CG_LIM, 0.0);
    return UNS_OK;
}

int uns_cc_fvresidual(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    CCView v = h->v;
    bool fused = false;
    // Since the last call that computed every face, only the conserved state
    // has changed (rk_stage, set_state): the interior and farfield fluxes read
    // the primitives, gradient and limiter alone, so only the wall faces and
    // their cells' residuals are recomputed, and after set_state every
    // boundary face and ghost row (bit-identical to a full call).
    // Viscous fluxes read the state, and a smoothing sweep replaces the stored
    // residual: those calls compute everything.
    const bool smooth = v.irs && epsirs_of(h, h->cfl_cur) > 0.0;
    const bool walls = !v.laminar && !smooth && h->res_gen == h->flux_gen;
    const int rc = walls ? enqueue_wall_res(h, v) : enqueue_fvresidual(h, v, h->cfl_cur, 0, 0, &fused);
    if (!rc) { h->res_gen = h->flux_gen; h->ghosts_set = false; }
    return rc;
}

int uns_cc_rk_stage(uns_cc_handle* h, int irk) {
    if (!h || irk < 1 || irk > 3) return UNS_ERR_ARG;
    CCView v = h->v;
    LAUNCH(k_rk_stage, v.noc, v, irk);
    return UNS_OK;
}

int uns_cc_lusgs(uns_cc_handle* h) {
    if (!h) return UNS_ERR_ARG;
    if (!h->v.srec) {  // packed cases are explicit: no sweep schedule, no records
        set_last_error("uns_cc_lusgs: the handle has no sweep schedule (packed cases)");
        return UNS_ERR_ARG;
    }
    int rc = uns_cc_fvresidual(h);
    if (rc) return rc;
    CCView v = h->v;
    return enqueue_lusgs(h, v);
}

int uns_cc_check_positivity(uns_cc_handle* h, int* bad) {
    if (!h) return UNS_ERR_ARG;
    CCView v = h->v;
    // An error that is there already is reported in place of the check's (the
    // first error stays, set_err).
    UNS_CUDA(cudaMemcpyAsync(v.err + 1, v.err, sizeof(DevErr), cudaMemcpyDeviceToDevice, h->stream));
    LAUNCH(k_check_pos, v.noc, v);
    DevReport r;
    const int rc = read_report(h, &r);
    if (rc) { if (bad) *bad = -1; return rc; }
    if (bad) *bad = r.before.code == 0 && r.err.code == UNS_ERR_NONPOSITIVE ? r.err.index : -1;
    return take_dev_err(h, r.err);
}

int uns_cc_residue(uns_cc_handle* h, double* fres) {
    if (!h || !fres) return UNS_ERR_ARG;
    CCView v = h->v;
    LAUNCH(k_res_partial, v.noc, v);
    k_res_final<<<1, kBlock, 0, h->stream>>>(v, h->nparts, h->d_scalar);
    UNS_CUDA(cudaGetLastError());
    DevReport r;
    const int rc = read_report(h, &r);
    if (rc) return rc;
    *fres = r.scalar[0];
    return take_dev_err(h, r.err);
}

int uns_cc_forces(uns_cc_handle* h, double* fx, double* fy) {
    if (!h || !fx || !fy) return UNS_ERR_ARG;
    k_forces<<<1, 1, 0, h->stream>>>(h->v, h->d_scalar);
    UNS_CUDA(cudaGetLastError());
    double r[2];
    UNS_CUDA(cudaMemcpyAsync(r, h->d_scalar, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    *fx = r[0];
    *fy = r[1];
    return UNS_OK;
}

// One main-loop iteration of a handle captured as a graph, wired to the
// handle's device-side CFL schedule, iteration counter, history and stop flag.
static int capture_iteration(uns_cc_handle* h, int first_iter, cudaGraph_t* out) {
    CCView v = h->v;
    v.cfl_sched = h->d_cfl;
    v.cfl_stride = h->cfl_cap;
    v.iter = h->d_iter;
    v.done = h->d_done;
    v.fres_hist = h->d_hist;
    v.fres1 = h->d_fres1;
    v.first_iter = first_iter ? 1 : 0;
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    UNS_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue_iteration(h, v, 0.0);
    cudaError_t ce = cudaStreamEndCapture(h->stream, out);
    if (rc) return rc;
    if (ce != cudaSuccess) { set_last_error(std::string("graph capture: ") + cudaGetErrorString(ce)); return UNS_ERR_CUDA; }
    return UNS_OK;
}

int uns_cc_iterate(uns_cc_handle* h, int niter, const double* cfl, int first_iter, double* fres_raw, int* done_iters) {
    if (!h || niter < 0 || (niter > 0 && (!cfl || !fres_raw))) return UNS_ERR_ARG;
    if (h->v.ninst) { set_last_error("uns_cc_iterate: a packed handle iterates with uns_cc_packed_iterate"); return UNS_ERR_ARG; }
    if (done_iters) *done_iters = 0;
    if (niter == 0) return UNS_OK;
    if (niter > h->cfl_cap) {
        int rc = grow_schedule(h, niter);
        if (rc) return rc;
    }
    // The smoothing sweeps are launched only while their coefficient is
    // non-zero; the schedule must agree on that for the whole chunk.
    bool any_smooth = false, all_smooth = true;
    for (int k = 0; k < niter; ++k) {
        bool s = h->P.irs && epsirs_of(h, cfl[k]) > 0.0;
        any_smooth = any_smooth || s;
        all_smooth = all_smooth && s;
    }
    if (any_smooth) {
        // Residual smoothing with a CFL above CFLmax changes the sweep
        // weights per iteration: run the chunk through the per-call path.
        double f1 = 0.0;
        int done = 0;
        for (int k = 0; k < niter; ++k) {
            int rc;
            if ((rc = uns_cc_con2prim(h)) || (rc = uns_cc_avg_c2v(h)) || (rc = uns_cc_time_step(h, cfl[k], nullptr)) ||
                (rc = uns_cc_save_old(h)) || (rc = uns_cc_gradient(h)))
                return rc;
            if (h->P.time_mode == UNS_TIME_RK3) {
                for (int irk = 1; irk <= 3; ++irk)
                    if ((rc = uns_cc_fvresidual(h)) || (rc = uns_cc_rk_stage(h, irk))) return rc;
            } else if ((rc = uns_cc_lusgs(h))) return rc;
            int bad;
            if ((rc = uns_cc_check_positivity(h, &bad))) return rc;
            if ((rc = uns_cc_residue(h, &fres_raw[k]))) return rc;
            ++done;
            if (first_iter && k == 0) f1 = fres_raw[0];
            double nf = (f1 >= 2.220446049250313e-16) ? fres_raw[k] / f1 : fres_raw[k];
            if (!(nf > h->P.min_res)) break;
        }
        if (done_iters) *done_iters = done;
        return UNS_OK;
    }
    (void)all_smooth;
    return iterate_graph(h, niter, cfl, first_iter, fres_raw, done_iters);
}

}  // extern "C"

// Device CFL schedule and residual history with room for cap iterations per
// instance; the captured iteration bakes in their addresses and stride.
static int grow_schedule(uns_cc_handle* h, int cap) {
    const size_t n = (size_t)std::max(1, h->v.ninst);
    if (h->d_cfl) cudaFree(h->d_cfl);
    if (h->d_hist) cudaFree(h->d_hist);
    h->d_cfl = nullptr; h->d_hist = nullptr;
    UNS_CUDA(cudaMalloc(&h->d_cfl, sizeof(double) * n * cap));
    UNS_CUDA(cudaMalloc(&h->d_hist, sizeof(double) * n * cap));
    h->cfl_cap = cap;
    ++h->gen;
    if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    return UNS_OK;
}

// The graph-replayed iterations of every instance: cfl and fres_raw are
// [instances][niter], done_iters [instances].
static int iterate_graph(uns_cc_handle* h, int niter, const double* cfl, int first_iter, double* fres_raw, int* done_iters) {
    ++h->flux_gen;
    const int n = std::max(1, h->v.ninst);
    if (niter > h->cfl_cap) {
        int rc = grow_schedule(h, niter);
        if (rc) return rc;
    }
    const size_t pitch = sizeof(double) * h->cfl_cap, row = sizeof(double) * niter;
    UNS_CUDA(cudaMemcpy2DAsync(h->d_cfl, pitch, cfl, row, row, n, cudaMemcpyHostToDevice, h->stream));
    UNS_CUDA(cudaMemsetAsync(h->d_iter, 0, sizeof(int) * n, h->stream));
    UNS_CUDA(cudaMemsetAsync(h->d_done, 0, sizeof(int) * n, h->stream));
    UNS_CUDA(cudaMemsetAsync(h->d_hist, 0, pitch * n, h->stream));
    if (!h->graph || h->graph_first != (first_iter ? 1 : 0)) {
        if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
        cudaGraph_t graph;
        int rc = capture_iteration(h, first_iter, &graph);
        if (rc) return rc;
        cudaError_t ce = cudaGraphInstantiate(&h->graph, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) { set_last_error(std::string("graph instantiate: ") + cudaGetErrorString(ce)); return UNS_ERR_CUDA; }
        h->graph_first = first_iter ? 1 : 0;
    }
    for (int k = 0; k < niter; ++k) UNS_CUDA(cudaGraphLaunch(h->graph, h->stream));
    UNS_CUDA(cudaMemcpy2DAsync(fres_raw, row, h->d_hist, pitch, row, n, cudaMemcpyDeviceToHost, h->stream));
    std::vector<int> it(n, 0);
    UNS_CUDA(cudaMemcpyAsync(it.data(), h->d_iter, sizeof(int) * n, cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    if (done_iters) std::copy(it.begin(), it.end(), done_iters);
    return check_dev_err(h);
}

extern "C" {

int uns_cc_set_wait_limit(uns_cc_handle* h, long long cycles) {
    if (!h || cycles <= 0) return UNS_ERR_ARG;
    h->v.wait_cycles = cycles;
    ++h->gen;
    if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    return UNS_OK;
}

int uns_cc_debug_unpublish(uns_cc_handle* h, int cell, int pass) {
    if (!h || cell < -1 || cell >= h->v.noc || pass < 0 || pass > 1) return UNS_ERR_ARG;
    h->v.skip_code = cell < 0 ? -1 : (cell << 1) | pass;
    ++h->gen;
    if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    return UNS_OK;
}

int uns_cc_set_precision(uns_cc_handle* h, int precision) {
    if (!h || precision < UNS_PREC_FP64 || precision > UNS_PREC_MIXED_SWEEP) return UNS_ERR_ARG;
    ++h->flux_gen;
    if (h->P.precision != precision) {
        UNS_CUDA(cudaStreamSynchronize(h->stream));
        h->P.precision = precision;
        CCView& v = h->v;
        const int was_mixed = v.mixed;
        v.mixed = precision == UNS_PREC_MIXED;
        if (v.mixed && !was_mixed) LAUNCH(k_mirror_f32, std::max(std::max(v.ntot, v.nof), v.nop), v);
        if (was_mixed && !v.mixed) LAUNCH(k_unpack_f32, v.noc, v);
        ++h->gen;
        if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    }
    return UNS_OK;
}

// ---------------------------------------------------------------- batches
// Independent instances advanced together: one CUDA graph whose parallel
// branches are the instances' captured iterations, so one launch advances
// every instance by one iteration and small meshes share the GPU.  Each
// instance keeps its own device state, CFL schedule, history and stop flag;
// an instance that has converged skips its kernels on the device.
struct uns_cc_batch {
    std::vector<uns_cc_handle*> hs;
    std::vector<int> gens;  // each handle's `gen` when the graph was built
    cudaStream_t stream = nullptr;
    cudaGraphExec_t exec = nullptr;
    int first = -1;
};

int uns_cc_batch_create(uns_cc_handle* const* handles, int n, uns_cc_batch** out) {
    if (!handles || n <= 0 || !out) { set_last_error("uns_cc_batch_create: bad arguments"); return UNS_ERR_ARG; }
    *out = nullptr;
    std::vector<uns_cc_handle*> hs(handles, handles + n);
    std::vector<uns_cc_handle*> sorted = hs;
    std::sort(sorted.begin(), sorted.end());
    if (!sorted[0] || std::adjacent_find(sorted.begin(), sorted.end()) != sorted.end()) {
        set_last_error("uns_cc_batch_create: null or repeated handle");
        return UNS_ERR_ARG;
    }
    auto* b = new uns_cc_batch();
    b->hs = hs;
    b->gens.assign(n, -1);
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete b;
        set_last_error("uns_cc_batch_create: cudaStreamCreate failed");
        return UNS_ERR_CUDA;
    }
    *out = b;
    return UNS_OK;
}

void* uns_cc_batch_stream(uns_cc_batch* b) { return b ? (void*)b->stream : nullptr; }

int uns_cc_batch_destroy(uns_cc_batch* b) {
    if (!b) return UNS_OK;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return UNS_OK;
}

int uns_cc_batch_iterate(uns_cc_batch* b, int niter, const double* cfl, int first_iter, double* fres_raw,
                         int* done_iters) {
    if (!b || niter < 0 || (niter > 0 && (!cfl || !fres_raw || !done_iters))) return UNS_ERR_ARG;
    const int n = (int)b->hs.size();
    if (niter == 0) {
        for (int i = 0; i < n; ++i) done_iters[i] = 0;
        return UNS_OK;
    }
    for (int i = 0; i < n; ++i) {
        uns_cc_handle* h = b->hs[i];
        ++h->flux_gen;
        for (int k = 0; k < niter; ++k)
            if (h->P.irs && epsirs_of(h, cfl[(size_t)i * niter + k]) > 0.0) {
                set_last_error("uns_cc_batch_iterate: residual smoothing above CFLmax is not batched");
                return UNS_ERR_ARG;
            }
        if (niter > h->cfl_cap) {
            UNS_CUDA(cudaStreamSynchronize(h->stream));
            if (h->d_cfl) cudaFree(h->d_cfl);
            if (h->d_hist) cudaFree(h->d_hist);
            h->d_cfl = nullptr; h->d_hist = nullptr;
            UNS_CUDA(cudaMalloc(&h->d_cfl, sizeof(double) * niter));
            UNS_CUDA(cudaMalloc(&h->d_hist, sizeof(double) * niter));
            h->cfl_cap = niter;
            ++h->gen;
            if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
        }
        UNS_CUDA(cudaStreamSynchronize(h->stream));
    }
    bool rebuild = !b->exec || b->first != (first_iter ? 1 : 0);
    for (int i = 0; i < n && !rebuild; ++i) rebuild = b->gens[i] != b->hs[i]->gen;
    if (rebuild) {
        if (b->exec) { cudaGraphExecDestroy(b->exec); b->exec = nullptr; }
        // Sweeps that do not fit beside each other, one block per SM, take the
        // form of which an SM holds two (102 400 cells each: two handles 3.17
        // -> 2.02 ms per iteration, three 4.72 -> 3.29, eight 12.6 -> 7.6).
        int sweeps = 0, blocks = 0;
        for (const uns_cc_handle* h : b->hs)
            if (h->P.time_mode == UNS_TIME_LUSGS) { ++sweeps; blocks += h->sweep_blocks; }
        const bool share = sweeps > 1 && blocks > b->hs[0]->nsm;
        cudaGraph_t parent;
        UNS_CUDA(cudaGraphCreate(&parent, 0));
        for (int i = 0; i < n; ++i) {
            cudaGraph_t child;
            b->hs[i]->share_sms = share;
            int rc = capture_iteration(b->hs[i], first_iter, &child);
            b->hs[i]->share_sms = false;
            if (rc) { cudaGraphDestroy(parent); return rc; }
            cudaGraphNode_t node;
            cudaError_t ce = cudaGraphAddChildGraphNode(&node, parent, nullptr, 0, child);
            cudaGraphDestroy(child);
            if (ce != cudaSuccess) {
                cudaGraphDestroy(parent);
                set_last_error(std::string("batch graph: ") + cudaGetErrorString(ce));
                return UNS_ERR_CUDA;
            }
            b->gens[i] = b->hs[i]->gen;
        }
        cudaError_t ce = cudaGraphInstantiate(&b->exec, parent, 0);
        cudaGraphDestroy(parent);
        if (ce != cudaSuccess) { set_last_error(std::string("batch graph instantiate: ") + cudaGetErrorString(ce)); return UNS_ERR_CUDA; }
        b->first = first_iter ? 1 : 0;
    }
    for (int i = 0; i < n; ++i) {
        uns_cc_handle* h = b->hs[i];
        UNS_CUDA(cudaMemcpyAsync(h->d_cfl, cfl + (size_t)i * niter, sizeof(double) * niter, cudaMemcpyHostToDevice, b->stream));
        UNS_CUDA(cudaMemsetAsync(h->d_iter, 0, sizeof(int), b->stream));
        UNS_CUDA(cudaMemsetAsync(h->d_done, 0, sizeof(int), b->stream));
        UNS_CUDA(cudaMemsetAsync(h->d_hist, 0, sizeof(double) * niter, b->stream));
    }
    for (int k = 0; k < niter; ++k) UNS_CUDA(cudaGraphLaunch(b->exec, b->stream));
    for (int i = 0; i < n; ++i) {
        uns_cc_handle* h = b->hs[i];
        UNS_CUDA(cudaMemcpyAsync(fres_raw + (size_t)i * niter, h->d_hist, sizeof(double) * niter, cudaMemcpyDeviceToHost,
                                 b->stream));
        UNS_CUDA(cudaMemcpyAsync(done_iters + i, h->d_iter, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
    }
    UNS_CUDA(cudaStreamSynchronize(b->stream));
    for (int i = 0; i < n; ++i) {
        int rc = check_dev_err(b->hs[i]);
        if (rc) return rc;
    }
    return UNS_OK;
}

void* uns_cc_stream(uns_cc_handle* h) { return h ? (void*)h->stream : nullptr; }

// Launch-geometry autotuner: times k_face_conv, k_vertex_avg and (in the
// mixed Green-Gauss step) k_cell_grad_side at each candidate block size on
// the handle's own mesh and state, keeps the fastest, and re-captures the
// step with them.  The timed launches read the handle's arrays and write
// scratch copies only, so the solution, the running limiter and the device
// counters are untouched.
int uns_cc_autotune(uns_cc_handle* h, int reps, int* blocks) {
    if (!h || reps < 1) return UNS_ERR_ARG;
    ++h->flux_gen;
    const CCView& v = h->v;
    std::vector<void*> bufs;
    auto scratch = [&](size_t bytes) -> void* {
        void* q = nullptr;
        if (cudaMalloc(&q, std::max<size_t>(bytes, 16)) != cudaSuccess) return nullptr;
        bufs.push_back(q);
        return q;
    };
    auto release = [&]() { for (void* q : bufs) cudaFree(q); bufs.clear(); };
    CCView t = v;  // inputs as the handle has them, outputs redirected
    t.cfl_sched = nullptr; t.iter = nullptr; t.done = nullptr;
    bool ok = (t.fF = (double4*)scratch(sizeof(double4) * v.nof)) && (t.qc = (double4*)scratch(sizeof(double4) * v.ntot)) &&
              (t.qp = (double4*)scratch(sizeof(double4) * v.ntot)) && (t.qT = (double*)scratch(sizeof(double) * v.ntot)) &&
              (t.qpf = (float4*)scratch(sizeof(float4) * v.ntot)) && (t.fwall = (double2*)scratch(sizeof(double2) * v.nbf)) &&
              (t.err = (DevErr*)scratch(sizeof(DevErr))) && (t.ppf = (float4*)scratch(sizeof(float4) * v.nop)) &&
              (t.pp = (double4*)scratch(sizeof(double4) * v.nop)) && (t.ppT = (double*)scratch(sizeof(double) * v.nop)) &&
              (t.la = (double*)scratch(sizeof(double) * v.noc)) && (t.dt = (double*)scratch(sizeof(double) * v.noc)) &&
              (t.dcv = (double*)scratch(sizeof(double) * v.noc)) && (t.packf = (float4*)scratch(sizeof(float4) * 4 * (size_t)v.noc)) &&
              (t.dtmin = (unsigned long long*)scratch(sizeof(unsigned long long) * std::max(1, v.ninst))) &&
              (t.minmax = (unsigned long long*)scratch(sizeof(unsigned long long) * 8 * std::max(1, v.ninst)));
    if (!ok) { release(); set_last_error("uns_cc_autotune: no device memory for the scratch outputs"); return UNS_ERR_CUDA; }
    int rc = UNS_OK;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    auto cuda = [&](cudaError_t e) { if (e != cudaSuccess && rc == UNS_OK) { rc = UNS_ERR_CUDA; set_last_error(std::string("uns_cc_autotune: ") + cudaGetErrorString(e)); } };
    cuda(cudaMemcpyAsync(t.qc, v.qc, sizeof(double4) * v.ntot, cudaMemcpyDeviceToDevice, h->stream));
    cuda(cudaMemcpyAsync(t.qp, v.qp, sizeof(double4) * v.ntot, cudaMemcpyDeviceToDevice, h->stream));
    cuda(cudaMemcpyAsync(t.qT, v.qT, sizeof(double) * v.ntot, cudaMemcpyDeviceToDevice, h->stream));
    cuda(cudaMemcpyAsync(t.qpf, v.qpf, sizeof(float4) * v.ntot, cudaMemcpyDeviceToDevice, h->stream));
    cuda(cudaMemcpyAsync(t.packf, v.packf, sizeof(float4) * 4 * (size_t)v.noc, cudaMemcpyDeviceToDevice, h->stream));
    cuda(cudaMemsetAsync(t.err, 0, sizeof(DevErr), h->stream));
    {  // a limiter range of [0, 1] for every case
        auto enc = [](double x) {  // enc_ord on the host
            unsigned long long b;
            std::memcpy(&b, &x, sizeof(b));
            return (b & 0x8000000000000000ULL) ? ~b : (b | 0x8000000000000000ULL);
        };
        std::vector<unsigned long long> mm(8 * (size_t)std::max(1, v.ninst));
        for (size_t k = 0; k < mm.size(); ++k) mm[k] = enc((k % 8) < 4 ? 1.0 : 0.0);
        cuda(cudaMemcpyAsync(t.minmax, mm.data(), sizeof(unsigned long long) * mm.size(), cudaMemcpyHostToDevice, h->stream));
        cuda(cudaStreamSynchronize(h->stream));
    }
    cuda(cudaEventCreate(&e0));
    cuda(cudaEventCreate(&e1));
    const bool sides = grad_by_sides(h, v);
    auto time_it = [&](auto&& launch) -> float {
        launch();  // warm-up
        cuda(cudaEventRecord(e0, h->stream));
        for (int r = 0; r < reps; ++r) launch();
        cuda(cudaEventRecord(e1, h->stream));
        cuda(cudaEventSynchronize(e1));
        float ms = 0.f;
        cuda(cudaEventElapsedTime(&ms, e0, e1));
        cuda(cudaGetLastError());
        return ms;
    };
    auto pick = [&](std::initializer_list<int> cand, auto&& launch_with) -> int {
        int best = 0;
        float tbest = 0.f;
        for (int bs : cand) {
            const float ms = time_it([&]() { launch_with(bs); });
            if (rc) return 0;
            if (!best || ms < tbest) { best = bs; tbest = ms; }
        }
        return best;
    };
    int bf = 0, bv = 0, bg = 0;
    if (rc == UNS_OK && v.nof > 0)
        bf = pick({64, 128, 256, v.mixed ? 512 : 256}, [&](int bs) {
            const int nb = std::max(1, (v.nbf + bs - 1) / bs + (v.nfi + bs - 1) / bs);
            if (v.mixed) k_face_conv<float><<<nb, bs, 0, h->stream>>>(t);
            else k_face_conv<double><<<nb, bs, 0, h->stream>>>(t);
        });
    if (rc == UNS_OK && v.nop > 0)
        bv = pick({64, 128, 256, 512}, [&](int bs) { k_vertex_avg<<<(v.nop + bs - 1) / bs, bs, 0, h->stream>>>(t); });
    if (rc == UNS_OK && sides && v.noc > 0)
        bg = pick({64, 128, 256}, [&](int bs) {
            k_cell_grad_side<<<(v.noc + bs - 1) / bs, bs, 0, h->stream>>>(t, CG_DT | CG_GRAD | (v.ilimit ? CG_LIM : 0), 0.5);
        });
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamSynchronize(h->stream);
    release();
    if (rc) return rc;
    if (bf) { h->v.blk_face = bf; h->blk_face_set = true; }
    if (bv) h->v.blk_vert = bv;
    if (bg) h->v.blk_grad = bg;
    if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    ++h->gen;  // the captured step changes
    if (blocks) { blocks[0] = h->v.blk_face; blocks[1] = h->v.blk_vert; blocks[2] = h->v.blk_grad; }
    return check_dev_err(h);
}

// cell_rk23 is the wall cells' three stages (k_wall_rk3); where they run,
// cell_res is the other cells' pass (k_cell_rk3 or k_cell_res_mixed).
int uns_cc_profile(uns_cc_handle* h, double cfl, int reps, double* ms, const char** names, int nphase) {
    static const char* kNames[] = {"begin", "vertex_avg", "face_prim_spec", "face_ggfc", "cell_grad", "face_conv",
                                   "viscous", "cell_res", "cirs", "lusgs_sweeps", "residue", "cell_rk23"};
    const int NP = 12;
    if (!h || reps < 1 || !ms) return UNS_ERR_ARG;
    ++h->flux_gen;
    std::vector<double> acc(NP, 0.0);
    cudaEvent_t e0, e1;
    UNS_CUDA(cudaEventCreate(&e0));
    UNS_CUDA(cudaEventCreate(&e1));
    CCView v = h->v;
    int rc = UNS_OK;
    auto timed = [&](int phase, auto&& launch) -> int {
        UNS_CUDA(cudaEventRecord(e0, h->stream));
        int r = launch();
        if (r) return r;
        UNS_CUDA(cudaEventRecord(e1, h->stream));
        UNS_CUDA(cudaEventSynchronize(e1));
        float t = 0.f;
        UNS_CUDA(cudaEventElapsedTime(&t, e0, e1));
        acc[phase] += t;
        return UNS_OK;
    };
    const bool rk3 = h->P.time_mode == UNS_TIME_RK3;
    const double eps = v.irs ? epsirs_of(h, cfl) : 0.0;
    const bool smooth = v.irs && eps > 0.0;
    for (int r = 0; r < reps && !rc; ++r) {
        rc = timed(0, [&]() -> int {
            k_reset_minmax<<<1, 32, 0, h->stream>>>(v);
            UNS_CUDA(cudaGetLastError());
            LAUNCH(k_begin, v.ntot, v, BEGIN_PRIM | BEGIN_OLD | BEGIN_POS | (v.ilimit ? BEGIN_MINMAX : 0));
            return UNS_OK;
        });
        if (!rc) rc = timed(1, [&]() -> int { LAUNCH_BS(k_vertex_avg, v.nop, v.blk_vert, v); return UNS_OK; });
        const bool sides = grad_by_sides(h, v);
        if (!rc && !sides) rc = timed(2, [&]() -> int { LAUNCH_SPREAD(k_face_prim_spec, v.nof, v); return UNS_OK; });
        if (!rc && v.grad_type == UNS_GRAD_GGFC) rc = timed(3, [&]() -> int { LAUNCH(k_face_ggfc, v.nof, v); return UNS_OK; });
        if (!rc) rc = timed(4, [&]() -> int {
            const int gflags = CG_DT | CG_GRAD | (v.ilimit ? CG_LIM : 0) | (rk3 ? 0 : CG_DIAG);
            if (sides) LAUNCH_BS(k_cell_grad_side, v.noc, v.blk_grad, v, gflags, cfl);
            else LAUNCH_CELL_GRAD(v, gflags, cfl);
            return UNS_OK;
        });
        const bool one_pass = rk3_in_one_pass(h, v, cfl);
        for (int irk = 1; irk <= (rk3 && !one_pass ? 3 : 1) && !rc; ++irk) {
            rc = timed(5, [&]() -> int {
                if (irk > 1 && (!v.laminar || v.grad_type == UNS_GRAD_GGFC)) return enqueue_wall_faces(h, v, false);
                if (h->P.precision == UNS_PREC_MIXED) LAUNCH_FACE_CONV(float, v);
                else LAUNCH_FACE_CONV(double, v);
                return UNS_OK;
            });
            if (!rc && v.laminar) rc = timed(6, [&]() -> int {
                LAUNCH(k_cell_mul, v.noc, v);
                if (v.grad_type != UNS_GRAD_GGFC) {
                    CCView w = v;
                    w.grad_type = UNS_GRAD_GGFC;
                    int r2 = enqueue_gradient(h, w, 0, cfl, true);
                    if (r2) return r2;
                }
                LAUNCH(k_face_visc, v.nof, v);
                return UNS_OK;
            });
            int fuse = (rk3 && !smooth) ? irk : 0;
            if (!rc && one_pass) rc = timed(11, [&]() -> int { return enqueue_wall_rk(h, v, h->stream); });
            if (!rc) rc = timed(7, [&]() -> int {
                if (one_pass) {
                    const int rc1 = enqueue_cell_rk(h, v);
                    return rc1 ? rc1 : enqueue_wall_parts(h, v);
                }
                if (v.mixed) LAUNCH(k_cell_res_mixed, v.noc, v, fuse, smooth ? 0 : 1, 0);
                else if (!smooth || v.ninst) LAUNCH(k_cell_res, v.noc, v, fuse, smooth ? 0 : 1);
                else LAUNCH_SPREAD(k_cell_res, v.noc, v, fuse, 0);  // as the iteration launches it
                return UNS_OK;
            });
            if (!rc && smooth) rc = timed(8, [&]() -> int {
                UNS_CUDA(cudaMemcpyAsync(v.res0, v.res, sizeof(double4) * v.noc, cudaMemcpyDeviceToDevice, h->stream));
                LAUNCH(k_cirs, v.noc, v, (const double4*)v.res0, v.restmp, eps);
                LAUNCH(k_cirs, v.noc, v, (const double4*)v.restmp, v.res, eps);
                LAUNCH(k_res_partial, v.noc, v);
                if (rk3) LAUNCH(k_rk_stage, v.noc, v, irk);
                return UNS_OK;
            });
        }
        if (!rc && !rk3) rc = timed(9, [&]() -> int { return enqueue_lusgs(h, v); });
        if (!rc) rc = timed(10, [&]() -> int {
            k_res_final<<<1, kBlock, 0, h->stream>>>(one_pass && !v.mixed ? final_view(h, v) : v, h->nparts, h->d_scalar);
            UNS_CUDA(cudaGetLastError());
            return UNS_OK;
        });
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    for (int k = 0; k < nphase; ++k) {
        ms[k] = k < NP ? acc[k] / reps : 0.0;
        if (names) names[k] = k < NP ? kNames[k] : "";
    }
    return check_dev_err(h);
}

}  // extern "C"

// ------------------------------------------------------------ packed cases
// Many independent CCFVM cases in ONE index space: the meshes are
// concatenated (points, then interior cells padded per case to a multiple of
// the block size, interior faces, boundary faces and their ghosts in case
// order), every element records its case, and the per-case constants and
// loop control become arrays.  One launch of each kernel then advances every
// case; each case's arithmetic, face orders and norm blocks are the ones it
// has alone, so it evolves bit-identically to a handle of its own.
extern "C" {

int uns_cc_create_packed(const uns_cc_mesh* meshes, const uns_params* params, int n, uns_cc_handle** out) {
    if (!meshes || !params || !out || n < 1) { set_last_error("uns_cc_create_packed: bad argument"); return UNS_ERR_ARG; }
    *out = nullptr;
    const uns_params& p0 = params[0];
    for (int i = 0; i < n; ++i) {
        const uns_params& p = params[i];
        if (p.time_mode != UNS_TIME_RK3 || p.irs != 0 || p.grad_type != p0.grad_type || p.ilimit != p0.ilimit ||
            p.flow_type != p0.flow_type || p.precision != p0.precision || p.limiter_type != p0.limiter_type) {
            set_last_error("uns_cc_create_packed: cases must share RK3 without smoothing, gradient, limiter, flow "
                           "type and precision (case " + std::to_string(i) + ")");
            return UNS_ERR_ARG;
        }
        const uns_cc_mesh& m = meshes[i];
        if (m.nop <= 0 || m.noc <= 0 || m.nfi < 0 || m.nbf < 0) { set_last_error("uns_cc_create_packed: bad sizes"); return UNS_ERR_ARG; }
    }
    std::vector<long long> C(n + 1, 0), F(n + 1, 0), B(n + 1, 0), P(n + 1, 0);
    for (int i = 0; i < n; ++i) {
        const uns_cc_mesh& m = meshes[i];
        C[i + 1] = C[i] + padded_cells(m.noc);
        F[i + 1] = F[i] + m.nfi;
        B[i + 1] = B[i] + m.nbf;
        P[i + 1] = P[i] + m.nop;
    }
    if (C[n] + B[n] >= (1LL << 30) || F[n] + B[n] >= (1LL << 30)) { set_last_error("uns_cc_create_packed: too large"); return UNS_ERR_ARG; }
    const int NOC = (int)C[n], NFI = (int)F[n], NBF = (int)B[n], NOP = (int)P[n], NOF = NFI + NBF, NTOT = NOC + NBF;
    std::vector<double> px(NOP), py(NOP), cx(NTOT, 0.0), cy(NTOT, 0.0), cv(NOC, 1.0), cov(NOC, 1.0);
    std::vector<double> r11(NOC, 1.0), r12(NOC, 0.0), r22(NOC, 1.0);
    std::vector<int> nc2c(NOC, 0), fp1(NOF), fp2(NOF), fin(NOF), fout(NOF), fbc(NOF);
    std::vector<double> fnx(NOF), fny(NOF), farea(NOF), fcx(NOF), fcy(NOF);
    std::vector<int> c2f_off(NOC + 1, 0), c2f, v2c_off(NOP + 1, 0), v2c;
    std::vector<double> v2c_wt;
    std::vector<int> cinst(NTOT, -1), finst(NOF), pinst(NOP);
    for (int i = 0; i < n; ++i) {
        const uns_cc_mesh& m = meshes[i];
        const int noc = m.noc, nfi = m.nfi, nof = m.nfi + m.nbf;
        auto cell = [&](int c) { return c < noc ? (int)C[i] + c : NOC + (int)B[i] + (c - noc); };
        auto face = [&](int f) { return f < nfi ? (int)F[i] + f : NFI + (int)B[i] + (f - nfi); };
        for (int k = 0; k < m.nop; ++k) { px[P[i] + k] = m.px[k]; py[P[i] + k] = m.py[k]; pinst[P[i] + k] = i; }
        for (int c = 0; c < noc + m.nbf; ++c) { cx[cell(c)] = m.cx[c]; cy[cell(c)] = m.cy[c]; cinst[cell(c)] = i; }
        for (int c = 0; c < noc; ++c) {
            const int g = (int)C[i] + c;
            cv[g] = m.cv[c]; cov[g] = m.cov[c]; r11[g] = m.r11[c]; r12[g] = m.r12[c]; r22[g] = m.r22[c]; nc2c[g] = m.nc2c[c];
        }
        for (int f = 0; f < nof; ++f) {
            const int g = face(f);
            if (m.fin[f] < 0 || m.fin[f] >= noc || m.fp1[f] < 0 || m.fp1[f] >= m.nop || m.fp2[f] < 0 || m.fp2[f] >= m.nop ||
                (f < nfi ? (m.fout[f] < 0 || m.fout[f] >= noc) : (m.fout[f] != noc + (f - nfi)))) {
                set_last_error("uns_cc_create_packed: case " + std::to_string(i) + " face " + std::to_string(f) +
                               " has an out-of-range index");
                return UNS_ERR_MESH;
            }
            fp1[g] = (int)P[i] + m.fp1[f]; fp2[g] = (int)P[i] + m.fp2[f];
            fin[g] = cell(m.fin[f]); fout[g] = cell(m.fout[f]); fbc[g] = m.fbc[f];
            fnx[g] = m.fnx[f]; fny[g] = m.fny[f]; farea[g] = m.farea[f]; fcx[g] = m.fcx[f]; fcy[g] = m.fcy[f];
            finst[g] = i;
        }
    }
    // cell -> faces (reference c2f order) and vertex -> cells, in global order
    for (int i = 0; i < n; ++i) {
        const uns_cc_mesh& m = meshes[i];
        const int noc = m.noc, nfi = m.nfi, ntot = noc + m.nbf;
        auto face = [&](int f) { return f < nfi ? (int)F[i] + f : NFI + (int)B[i] + (f - nfi); };
        auto cell = [&](int c) { return c < noc ? (int)C[i] + c : NOC + (int)B[i] + (c - noc); };
        for (int c = 0; c < (int)(C[i + 1] - C[i]); ++c) {
            const int g = (int)C[i] + c;
            if (c < noc)
                for (int k = m.c2f_off[c]; k < m.c2f_off[c + 1]; ++k) {
                    if (m.c2f[k] < 0 || m.c2f[k] >= m.nfi + m.nbf) { set_last_error("uns_cc_create_packed: c2f index out of range"); return UNS_ERR_MESH; }
                    c2f.push_back(face(m.c2f[k]));
                }
            c2f_off[g + 1] = (int)c2f.size();
        }
        for (int k = 0; k < m.nop; ++k) {
            const int g = (int)P[i] + k;
            for (int e = m.v2c_off[k]; e < m.v2c_off[k + 1]; ++e) {
                if (m.v2c[e] < 0 || m.v2c[e] >= ntot) { set_last_error("uns_cc_create_packed: v2c index out of range"); return UNS_ERR_MESH; }
                v2c.push_back(cell(m.v2c[e]));
                v2c_wt.push_back(m.v2c_wt[e]);
            }
            v2c_off[g + 1] = (int)v2c.size();
        }
    }
    uns_cc_mesh pm;
    pm.nop = NOP; pm.noc = NOC; pm.nfi = NFI; pm.nbf = NBF;
    pm.px = px.data(); pm.py = py.data(); pm.cx = cx.data(); pm.cy = cy.data(); pm.cv = cv.data(); pm.cov = cov.data();
    pm.fp1 = fp1.data(); pm.fp2 = fp2.data(); pm.fin = fin.data(); pm.fout = fout.data(); pm.fbc = fbc.data();
    pm.fnx = fnx.data(); pm.fny = fny.data(); pm.farea = farea.data(); pm.fcx = fcx.data(); pm.fcy = fcy.data();
    pm.r11 = r11.data(); pm.r12 = r12.data(); pm.r22 = r22.data(); pm.nc2c = nc2c.data();
    pm.c2f_off = c2f_off.data(); pm.c2f = c2f.data(); pm.v2c_off = v2c_off.data(); pm.v2c = v2c.data(); pm.v2c_wt = v2c_wt.data();
    uns_cc_handle* h = nullptr;
    int rc = create_impl(&pm, &p0, false, &h);
    if (rc) return rc;
    auto fail = [&](int code) { uns_cc_destroy(h); return code; };
    // per-case constants and loop control
    std::vector<Gas> gas(n);
    std::vector<double4> qinfs(n);
    std::vector<int> boff(n + 1), ncell(n);
    std::vector<double> minres(n);
    for (int i = 0; i < n; ++i) {
        gas[i] = make_gas(&params[i], &qinfs[i]);
        boff[i] = (int)(C[i] / kBlock);
        ncell[i] = meshes[i].noc;
        minres[i] = params[i].min_res;
    }
    boff[n] = (int)(C[n] / kBlock);
    CCView& v = h->v;
#define UPP(field, vec) if ((rc = h->upload(*(std::remove_const<std::remove_pointer<decltype(v.field)>::type>::type**)&v.field, vec.data(), vec.size()))) return fail(rc)
    UPP(cinst, cinst); UPP(finst, finst); UPP(pinst, pinst); UPP(gas, gas); UPP(qinfs, qinfs);
    UPP(boff, boff); UPP(ncell, ncell); UPP(minres, minres);
#undef UPP
    if ((rc = h->alloc(v.minmax, 8 * (size_t)n)) || (rc = h->alloc(v.dtmin, (size_t)n)) || (rc = h->alloc(h->d_iter, (size_t)n)) ||
        (rc = h->alloc(h->d_done, (size_t)n)) || (rc = h->alloc(h->d_fres1, (size_t)n)))
        return fail(rc);
    v.ninst = n;
    if (cudaStreamSynchronize(h->stream) != cudaSuccess) { set_last_error("uns_cc_create_packed: upload failed"); return fail(UNS_ERR_CUDA); }
    if ((rc = uns_cc_initialize(h))) return fail(rc);
    *out = h;
    return UNS_OK;
}

int uns_cc_packed_layout(uns_cc_handle* h, int* cell_off, int* ghost_off) {
    if (!h || !h->v.ninst || !cell_off || !ghost_off) { set_last_error("uns_cc_packed_layout: not a packed handle"); return UNS_ERR_ARG; }
    const int n = h->v.ninst;
    std::vector<int> b(n + 1), nc(n);
    UNS_CUDA(cudaMemcpyAsync(b.data(), h->v.boff, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaMemcpyAsync(nc.data(), h->v.ncell, sizeof(int) * n, cudaMemcpyDeviceToHost, h->stream));
    std::vector<int> fi(h->v.nof);
    UNS_CUDA(cudaMemcpyAsync(fi.data(), h->v.finst, sizeof(int) * h->v.nof, cudaMemcpyDeviceToHost, h->stream));
    UNS_CUDA(cudaStreamSynchronize(h->stream));
    for (int i = 0; i <= n; ++i) cell_off[i] = b[i] * kBlock;
    // ghosts follow the boundary faces, which are in case order
    int k = 0;
    for (int i = 0; i < n; ++i) {
        ghost_off[i] = k;
        while (k < h->v.nbf && fi[h->v.nfi + k] == i) ++k;
    }
    ghost_off[n] = k;
    return UNS_OK;
}

int uns_cc_packed_iterate(uns_cc_handle* h, int niter, const double* cfl, int first_iter, double* fres_raw, int* done_iters) {
    if (!h || !h->v.ninst || niter < 1 || !cfl || !fres_raw) { set_last_error("uns_cc_packed_iterate: bad argument"); return UNS_ERR_ARG; }
    return iterate_graph(h, niter, cfl, first_iter, fres_raw, done_iters);
}

}  // extern "C"
