// uns_sweep.cuh -- the LU-SGS sweeps of both solvers (CCFVM/lusgs.F90:245-318,
// NCFVM/lusgs.f90:48-124) as one cooperative launch.
//
// A sweep is a chain of items (entity, pass), each a few dozen dependent FP64
// operations on values that other warps have just published.  Each sweep warp
// has its own list of items (uns_sched.hpp) and, on the same SM
// sub-partition, two helpers that walk the list with it:
//   the feeder loads an item's inputs ahead of time,
//   the poller reads its neighbours' records until they are published,
// both into a ring in shared memory laid out per lane; the sweep warp takes an
// entry, does the arithmetic and publishes.  Its only global accesses are the
// stores.  One warp doing all three took twice the time of the arithmetic: the
// results of loads and of FP64 instructions share the warp's few scoreboards,
// so an addition's result waits for a load in flight (NCFVM 1024x512: 9.56 ms;
// 7.00 with one helper for loads and polls; 6.54 with two).
//
// An entry passes from the feeder to the poller through the mbarrier `full`
// (the inputs are there, the neighbours' fields that must be polled hold
// kUnset), from the poller to the sweep warp through the count `ready` (a load
// of shared memory is all that a sweep warp spends where the entry is there;
// an mbarrier wait took 200 cycles of each item) and back to the feeder
// through the mbarrier `empty`.  Every wait is bounded; a warp that gives up
// raises `abort`, on which its partners return.
//
// Lanes of an item: lane = 4 * slot + k, slot = the taken face or edge (up to
// 8 per entry), k = the variable.  An FP64 instruction holds the sub-partition's
// unit 64-76 cycles whatever the number of active lanes, so the four flux
// components of up to eight faces are one pass, the per-variable sums and
// divisions run in lanes 0..3 and the three divisions of con2prim in lanes 0,
// 2 and 3 at once; the warp exchanges lane values through shared memory.
#pragma once
#include "uns_common.cuh"
#include "uns_fp64.cuh"
#include "uns_sched.hpp"

#include <type_traits>

namespace uns {

constexpr int kSweepPairs = 4;                   // sweep warps per block: one per SM sub-partition
static_assert(kSweepPairs == kSchedGroup, "WarpSchedule::src names a warp of a block");
constexpr int kSweepBlock = 3 * 32 * kSweepPairs;  // sweep warps, feeders, pollers
// One sweep block per SM, so that concurrently active items never share an FP64 unit.
constexpr int kSweepBlocksPerSM = 1;
constexpr int kSweepStages = 3;
constexpr double kOmega = 1.5;                   // CCFVM/lusgs.F90:229, NCFVM/lusgs.f90:26

// What the sweeps read and write.
struct SweepArgs {
    int n;                 // entities
    const int4* sched;     // (entity, pass, first record, records) per list position
    const int* rec_src;    // per record: its producer in this block (WarpSchedule::src), or -1
    const double4* rec;    // inputs per record (k_*_sweep_prep): 3 x double4, or 4 x float4 in the mixed form
    const double* diag;    // the diagonal, or its reciprocal in the mixed form
    const double4* qold;
    const double4* res;
    double4* qc;
    double2* out;          // FP64 records [pass * n + entity][5]: u v, p e*rho, rho dq0, dq1 dq2, dq3 -
    float4* outf;          // mixed records [pass * n + entity]: dq in FP32
    double4* outd;         //   and in FP64 (the entity's own backward step)
    DevErr* err;
    long long wait_cycles; // bound of a wait for a record
    long long ring_cycles; // and of a wait for a partner (ring_wait_limit)
    int skip_code;         // test hook: the item (entity << 1 | pass) that publishes nothing, or -1
    double gm1;
};

// One sweep warp's ring: NF 8-byte fields per lane and stage, and the item.
template <int NF>
struct __align__(16) SweepRing {
    unsigned long long full[kSweepStages], empty[kSweepStages];
    double f[kSweepStages][NF][32];
    int4 item[kSweepStages];
    int ready;  // entries that the sweep warp may read
    int abort;
    int pad[2];
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

template <int NF>
__device__ __forceinline__ void ring_init(SweepRing<NF>& R) {
    for (int s = 0; s < kSweepStages; ++s) {
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(smem_addr(&R.full[s])) : "memory");
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(smem_addr(&R.empty[s])) : "memory");
    }
    R.ready = 0;
    R.abort = 0;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.release.cta.shared.b64 _, [%0];" : : "r"(smem_addr(b)) : "memory");
}

__device__ __forceinline__ int ld_acquire(const int* p) {
    int x;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(x) : "r"(smem_addr(p)) : "memory");
    return x;
}
__device__ __forceinline__ void st_release(int* p, int x) {
    asm volatile("st.release.cta.shared.s32 [%0], %1;" : : "r"(smem_addr(p)), "r"(x) : "memory");
}
// A wait inside the ring (all lanes) outlasts the poller's own for a record;
// it ends early when a partner has aborted.  False: the caller returns.
struct RingWait {
    const int* abort;
    DevErr* err;
    long long limit, t0;
    __device__ __forceinline__ RingWait(const int* a, const SweepArgs& s)
        : abort(a), err(s.err), limit(s.ring_cycles), t0(0) {}
    __device__ __forceinline__ bool go_on(int spins) {
        if (spins == 0) t0 = clock64();
        if ((spins & 15) != 15) return true;
        if (*(const volatile int*)abort) return false;
        if (clock64() - t0 <= limit) return true;
        set_err(err, UNS_ERR_TIMEOUT, -1);
        *(volatile int*)const_cast<int*>(abort) = 1;
        return false;
    }
};

__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity, RingWait w) {
    const unsigned a = smem_addr(b);
    for (int spins = 0;; ++spins) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cta.shared.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
        if (!w.go_on(spins)) return false;
    }
}

// The sweep warp's wait (all lanes) for the ring's entry of that number.
__device__ __forceinline__ bool entry_wait(const int* ready, int entry, RingWait w) {
    for (int spins = 0; ld_acquire(ready) < entry; ++spins)
        if (!w.go_on(spins)) return false;
    return true;
}

// The last kBox records of a sweep warp, for the warps of its block: a record
// that a neighbouring warp needs is read here a few hundred cycles after its
// item ends, against 1 500-2 900 through L2 (store, poll, the two dies).
// seq[slot] is the list index of the record in the slot, ~index from the start
// of the item that will write it; a reader checks it before and after, and
// where the slot has moved on, or is about to (the item that takes it over may
// wait for the reader's), it takes the global record, published long before.
constexpr int kBox = 16;
template <int NP>
struct __align__(16) SweepBox {
    double2 rec[kBox][NP];
    int seq[kBox];
};
template <int NP>
__device__ __forceinline__ void box_init(SweepBox<NP>& b) {
    for (int i = 0; i < kBox; ++i) b.seq[i] = ~0;
}
// Marks the slot of list index idx as being written (lane 0, early in the item).
template <int NP>
__device__ __forceinline__ void box_open(SweepBox<NP>& b, int idx) {
    *(volatile int*)&b.seq[idx % kBox] = ~idx;
    __threadfence_block();
}

// Where a record comes from, in the upper word of an entry's code field: bits
// 0..30 one more than WarpSchedule::src, 0 for another
// block's; bit 31 the orientation's sign.
__device__ __forceinline__ int src_of(long long code) { return (int)((unsigned long long)code >> 32 & 0x7fffffffu) - 1; }

// Position in the ring: stage and the parity of its next phase.
struct RingPos {
    int stage = 0;
    unsigned phase = 0;
    __device__ __forceinline__ void next() {
        if (++stage == kSweepStages) { stage = 0; phase ^= 1; }
    }
};

__device__ __forceinline__ double ld_relaxed(const double* p) {
    double x;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(x) : "l"(p) : "memory");
    return x;
}
__device__ __forceinline__ double ld_field(const double* p) { return *(const volatile double*)p; }
__device__ __forceinline__ void st_field(double* p, double x) { *(volatile double*)p = x; }
__device__ __forceinline__ double unset() { return __longlong_as_double((long long)kUnset); }
__device__ __forceinline__ double pack2(float a, float b) { return dmake(__float_as_uint(b), __float_as_uint(a)); }
__device__ __forceinline__ float low_f(double x) { return __uint_as_float(dlo(x)); }
__device__ __forceinline__ float high_f(double x) { return __uint_as_float(dhi(x)); }

// The bounded wait of a poller; abort ends it too.
__device__ __forceinline__ bool poller_go_on(int spins, long long& t0, const SweepArgs& a, int* abort) {
    if ((spins & 63) == 63 && *(volatile int*)abort) return false;
    return poll_continue(spins, t0, a.err, a.wait_cycles);
}

// ---------------------------------------------------------------- FP64 form
// Fields of an entry: the slot's record, f1 its component k; the neighbour's
// record (u, v, p, e*rho, rho, component k of dq); twice the entity's diagonal,
// its qold and twice its res (pass 0) or its forward dq (pass 1), variable k;
// and the neighbour's code (entity << 1 | pass, -1 in an idle slot) with the
// sign of the record's orientation in the upper word.
enum { SF_F1, SF_NX, SF_NY, SF_DS, SF_OL, SF_U, SF_V, SF_P, SF_ET, SF_RHO, SF_DQ, SF_D2, SF_O, SF_R, SF_CODE, SF_N };
typedef SweepRing<SF_N> RingD;
typedef SweepBox<5> BoxD;  // the record's five 16-byte pieces

__device__ __forceinline__ void sweep_feed(const SweepArgs& a, RingD& R, int kbeg, int kend, int lane) {
    const int slot = lane >> 2, k = lane & 3;
    RingPos pos;
    int last = -1;  // the list's previous item: its values come from the sweep warp's registers
    int4 S = a.sched[kbeg];
    for (int kk = kbeg; kk < kend; ++kk) {
        const int4 Sn = kk + 1 < kend ? a.sched[kk + 1] : make_int4(0, 0, 0, 0);
        const int it = S.x, pass = S.y, ntake = S.w;
        int base = 0;
        do {
            const bool take = base + slot < ntake;
            double4 b = make_double4(0.0, 0.0, 0.0, 0.0), c = b;
            double f1 = 0.0, D = 1.0, o = 1.0, r = 0.0;
            int src = -1;
            if (take) {
                src = a.rec_src[S.z + base + slot];
                const double4* p = a.rec + 3 * (size_t)(S.z + base + slot);
                f1 = reinterpret_cast<const double*>(p)[k];
                b = p[1];
                c = p[2];
            }
            if (base == 0 && lane < 4) {
                D = a.diag[it];
                o = reinterpret_cast<const double*>(&a.qold[it])[lane];
                if (pass == 0) r = reinterpret_cast<const double*>(&a.res[it])[lane];
            }
            const int code = take ? ((int)__double_as_longlong(c.z) << 1) | pass : -1;
            const bool nb = take && code != last, own = base == 0 && lane < 4 && pass == 1 && (it << 1) != last;
            if (!mbar_wait(&R.empty[pos.stage], pos.phase ^ 1, RingWait(&R.abort, a))) return;
            double(*f)[32] = R.f[pos.stage];
            f[SF_F1][lane] = f1;
            f[SF_NX][lane] = b.x; f[SF_NY][lane] = b.y; f[SF_DS][lane] = b.z; f[SF_OL][lane] = b.w;
            f[SF_CODE][lane] = dmake((dhi(c.y) & 0x80000000u) | (unsigned)(src + 1), (unsigned)code);
            const double none = nb ? unset() : 0.0;
            f[SF_U][lane] = none; f[SF_V][lane] = none; f[SF_P][lane] = none;
            f[SF_ET][lane] = none; f[SF_RHO][lane] = none; f[SF_DQ][lane] = none;
            if (base == 0) {
                f[SF_D2][lane] = D + D;
                f[SF_O][lane] = o;
                f[SF_R][lane] = own ? unset() : r + r;
                if (lane == 0) R.item[pos.stage] = S;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&R.full[pos.stage]);
            pos.next();
            base += 8;
        } while (base < ntake);
        last = (it << 1) | pass;
        if (last == a.skip_code) last = -1;  // test hook: that item hands nothing on
        S = Sn;
    }
}

__device__ __forceinline__ void sweep_poll(const SweepArgs& a, RingD& R, const BoxD* boxes, int kbeg, int kend, int lane) {
    const int k = lane & 3;
    RingPos pos;
    int entries = 0;
    for (int kk = kbeg; kk < kend; ++kk) {
        int ntake = 0, base = 0;
        do {
            if (!mbar_wait(&R.full[pos.stage], pos.phase, RingWait(&R.abort, a))) return;
            double(*f)[32] = R.f[pos.stage];
            const int4 S = R.item[pos.stage];  // (base > 0: the stage's older item, unused)
            if (base == 0) ntake = S.w;
            const long long cs = __double_as_longlong(ld_field(&f[SF_CODE][lane]));
            const int code = (int)cs;
            int src = src_of(cs);
            bool nb = is_unset(ld_field(&f[SF_DQ][lane]));
            bool own = base == 0 && lane < 4 && is_unset(ld_field(&f[SF_R][lane]));
            const double2* p = a.out + 5 * ((size_t)(code & 1) * a.n + (nb ? code >> 1 : 0));
            const double* po = reinterpret_cast<const double*>(a.out + 5 * (size_t)(own ? S.x : 0)) + 5 + lane;
            long long t0 = 0;
            for (int spins = 0; nb || own; ++spins) {
                if (nb) {
                    double2 x0, x1;
                    double rho, dq;
                    if (src >= 0) {
                        const BoxD& b = boxes[src >> kSrcBits];
                        const int idx = src & ((1 << kSrcBits) - 1), seq = ld_acquire(&b.seq[idx % kBox]);
                        const volatile double* q = reinterpret_cast<const volatile double*>(b.rec[idx % kBox]);
                        x0.x = q[0]; x0.y = q[1]; x1.x = q[2]; x1.y = q[3];
                        rho = q[4]; dq = q[5 + k];
                        __threadfence_block();
                        const bool same = seq == idx && *(const volatile int*)&b.seq[idx % kBox] == idx;
                        if (!same) x0.x = unset();
                        if ((seq < 0 ? ~seq : seq) > idx) src = -1;  // the slot has moved on
                    } else {
                        x0 = ld_relaxed2(p); x1 = ld_relaxed2(p + 1);
                        rho = ld_relaxed(reinterpret_cast<const double*>(p) + 4);
                        dq = ld_relaxed(reinterpret_cast<const double*>(p) + 5 + k);
                    }
                    if (!(is_unset(x0.x) || is_unset(x0.y) || is_unset(x1.x) || is_unset(x1.y) || is_unset(rho) || is_unset(dq))) {
                        st_field(&f[SF_U][lane], x0.x); st_field(&f[SF_V][lane], x0.y); st_field(&f[SF_P][lane], x1.x);
                        st_field(&f[SF_ET][lane], x1.y); st_field(&f[SF_RHO][lane], rho); st_field(&f[SF_DQ][lane], dq);
                        nb = false;
                    }
                }
                if (own) {
                    const double r = ld_relaxed(po);
                    if (!is_unset(r)) { st_field(&f[SF_R][lane], r); own = false; }
                }
                if ((nb || own) && !poller_go_on(spins, t0, a, &R.abort)) {
                    *(volatile int*)&R.abort = 1;
                    break;
                }
            }
            if (__any_sync(0xffffffffu, nb || own)) return;  // a wait gave up; the error is recorded
            __syncwarp();
            if (lane == 0) st_release(&R.ready, ++entries);
            pos.next();
            base += 8;
        } while (base < ntake);
    }
}

// The sweep warp.  Per item, for each face or edge whose neighbour precedes
// the entity in this pass (reference order): the neighbour's values come from
// registers when the warp itself computed that neighbour last, else from the
// ring; the term (CCFVM: area*(F(qold+dq) - F(qold)) - omega*lam*dq, NCFVM:
// sign*(F*ds - F(qold)*ds) - omega*la*dq) is formed per component, lanes 0..3
// add the terms in order (the reference's summation order) and divide by the
// diagonal; the new state is spread to all lanes, which keep its primitives
// for the next item while lanes 0..4 publish the record.  Every rounded
// operation and its operand order is the reference's, but for its factor 0.5
// on the terms, which doubles res and the diagonal instead (a scaling by two
// commutes with every rounding short of the subnormal range).
//
// Sums and products are register FMAs (64 cycles each); the two divisions (590
// cycles each on the FP64 unit) run on the integer pipe (240).  An item then
// takes about 2 500 cycles and a level of the graph 3 400 (its hand-offs
// between blocks are the rest): NCFVM 1024x512 sweeps 9.69 -> 6.15 ms, 128x64
// 1.15 -> 0.74, FP32 form at 512x256 3.47 -> 2.17, CCFVM 320x160 2.41 -> 1.47.
// Per-lane selection by a mask (all ones: a) that the compiler does not know
// to be a comparison of k: as a plain conditional it became branches around
// the FMA that takes the value, one copy of it per value (64 cycles each).
__device__ __forceinline__ unsigned lane_mask(bool on) {
    unsigned m = on ? 0xffffffffu : 0u;
    asm volatile("" : "+r"(m));
    return m;
}
__device__ __forceinline__ double pick(unsigned m, double a, double b) {
    return dmake((dhi(a) & m) | (dhi(b) & ~m), (dlo(a) & m) | (dlo(b) & ~m));
}
__device__ __forceinline__ float pick(unsigned m, float a, float b) {
    return __uint_as_float((__float_as_uint(a) & m) | (__float_as_uint(b) & ~m));
}

// An entry of the ring in registers.
struct SweepEntry {
    double f1, nx, ny, ds, ol, u, v, p, et, rho, dq, D2, o, r;
    long long code;
    int4 item;
    __device__ __forceinline__ void load(const RingD& R, int stage, int lane, bool first) {
        const double(*f)[32] = R.f[stage];
        if (first) {
            item = R.item[stage];
            D2 = f[SF_D2][lane]; o = f[SF_O][lane]; r = f[SF_R][lane];
        }
        code = __double_as_longlong(f[SF_CODE][lane]);
        u = f[SF_U][lane]; v = f[SF_V][lane]; p = f[SF_P][lane];
        et = f[SF_ET][lane]; rho = f[SF_RHO][lane]; dq = f[SF_DQ][lane];
        f1 = f[SF_F1][lane]; nx = f[SF_NX][lane]; ny = f[SF_NY][lane]; ds = f[SF_DS][lane]; ol = f[SF_OL][lane];
    }
};

template <bool kCC>
__device__ __forceinline__ void sweep_items(const SweepArgs& a, RingD& R, BoxD& box, double* wx, int kbeg, int kend, int lane) {
    const int k = lane & 3;
    const double gm1 = in_register(a.gm1), one = opaque_one(), mzero = opaque_mzero();
    const unsigned m0 = lane_mask(k == 0), m2 = lane_mask(k == 2), m01 = lane_mask(k < 2);
    const unsigned ml1 = lane_mask(lane == 1), ml01 = lane_mask(lane < 2);
    RingPos pos;
    int last = -1;  // code of the warp's previous item; its values below, in every lane
    double Lu = 0.0, Lv = 0.0, Lp = 0.0, Let = 0.0, Lrho = 0.0, Ldq = 0.0;
    SweepEntry X;
    X.r = 0.0;
    int entries = 0;
    for (int kk = kbeg; kk < kend; ++kk) {
        double cres = 0.0;  // lanes 0..3: sum over the terms of component k
        unsigned Y = 0;     // the diagonal's reciprocal digits, off the chain
        const int idx = kk - kbeg, bslot = idx % kBox;
        if (lane == 0) box_open(box, idx);
        int it = 0, pass = 0, ntake = 0, base = 0;
        do {
            if (!entry_wait(&R.ready, ++entries, RingWait(&R.abort, a))) return;
            X.load(R, pos.stage, lane, base == 0);
            __syncwarp();
            if (lane == 0) mbar_arrive(&R.empty[pos.stage]);
            pos.next();
            if (base == 0) {
                it = X.item.x; pass = X.item.y; ntake = X.item.w;
                Y = div_recip(X.D2);
                if (ntake == 0) break;
            }
            const int code = (int)X.code;
            if (code == last && code >= 0) { X.u = Lu; X.v = Lv; X.p = Lp; X.et = Let; X.rho = Lrho; X.dq = Ldq; }
            // normal flux (CCFVM/lusgs.F90:348-357, NCFVM/lusgs.f90:144-150)
            // component k, then the term; idle slots compute on zeros.  Lane k
            // = 0 forms (et + p)*un, k = 1 rho*un, k = 2 and 3 rho*un*(u or v)
            // + p*(nx or ny): one FMA with per-lane operands does an addition
            // in some lanes and a product in others (x*1 + y, x*y + -0; B + -0
            // is B).
            const double un = add64(mul64(X.u, X.nx), mul64(X.v, X.ny));
            const double hp = __fma_rn(pick(m0, X.et, X.p), pick(m0, one, pick(m2, X.nx, X.ny)), pick(m0, X.p, mzero));
            const double A = mul64(pick(m0, hp, X.rho), un);
            const double B = __fma_rn(A, pick(m01, one, pick(m2, X.u, X.v)), mzero);
            const double o = __fma_rn(B, one, pick(m01, mzero, hp));
            const double df = kCC ? mul64(X.ds, sub64(o, X.f1)) : flip64(sub64(mul64(o, X.ds), X.f1), X.code < 0);
            const double t = sub64(df, mul64(X.ol, X.dq));
            // the terms in order, from 0.0 (the first addition is exact)
            const int nr = min(8, ntake - base);
            wx[lane] = t;
            __syncwarp();
            int e = 0;
            if (base == 0) { cres = zero_plus(wx[k]); e = 1; }
            for (; e < nr; ++e) cres = add64(cres, wx[4 * e + k]);
            __syncwarp();
            base += 8;
        } while (base < ntake);
        // dq and qold + dq (CCFVM/lusgs.F90:276-279, 314-317; NCFVM/lusgs.f90:
        // 78-81, 117-120), component k in lane k
        double d;
        if (pass == 0) {
            d = div_digits(sub64(neg64(X.r), cres), X.D2, Y);
        } else {  // from the entity's own forward dq
            d = sub64((it << 1) == last ? Ldq : X.r, div_digits(cres, X.D2, Y));
        }
        const double q = add64(X.o, d);
        // con2prim (CCFVM/types/pri.F90:13-37, NCFVM/All_modules.f90:146-169):
        // rho = q1, then E/rho, rhou/rho, rhov/rho in lanes 0, 2, 3
        if (lane < 4) { wx[lane] = q; wx[5 + lane] = d; }
        __syncwarp();
        const double2 qa = reinterpret_cast<const double2*>(wx)[0], qb = reinterpret_cast<const double2*>(wx)[1];
        const double E = qa.x, rn = qa.y;
        const double quo = div_digits(q, rn);
        // the four products of the pressure and the record as one
        // multiplication: lane 0 e*rho, lane 1 0.5*rho, lane 2 u*u, lane 3 v*v
        const double pr = mul64(pick(ml1, 0.5, quo), pick(ml01, rn, quo));
        if (lane < 4) { wx[10 + lane] = quo; wx[14 + lane] = pr; }
        if (lane == 1) wx[4] = rn;
        __syncwarp();
        const double2 pa = reinterpret_cast<const double2*>(wx)[7], pb = reinterpret_cast<const double2*>(wx)[8];
        Lu = wx[12]; Lv = wx[13]; Ldq = wx[5 + k];
        const double2 piece = reinterpret_cast<const double2*>(wx)[lane < 2 || lane > 4 ? 6 : lane];  // u v | rho d0 | d1 d2 | d3 -
        __syncwarp();
        const double qq = add64(pb.x, pb.y);                    // u*u + v*v
        Lp = mul64(gm1, sub64(E, mul64(pa.y, qq)));             // gm1*(E - 0.5*rho*qq)
        Let = pa.x; Lrho = rn;
        last = (it << 1) | pass;
        if (last == a.skip_code) {  // test hook: this item publishes nothing and hands nothing on
            last = -1;
        } else {
            // lanes 0..4 store the record's five 16-byte pieces in one
            // predicated instruction
            double2* dst = a.out + 5 * ((size_t)pass * a.n + it) + (lane < 5 ? lane : 0);
            const double x = lane == 1 ? Lp : piece.x, y = lane == 1 ? Let : piece.y;
            if (lane < 5) box.rec[bslot][lane] = make_double2(x, y);
            __syncwarp();
            if (lane == 0) st_release(&box.seq[bslot], idx);
            asm volatile(
                "{\n\t.reg .pred pa;\n\t"
                "setp.ne.s32 pa, %0, 0;\n\t"
                "@pa st.relaxed.gpu.global.v2.f64 [%1], {%2, %3};\n\t}"
                : : "r"((int)(lane < 5)), "l"(dst), "d"(x), "d"(y) : "memory");
            if (pass == 1 && lane == 2) a.qc[it] = make_double4(E, rn, qb.x, qb.y);
        }
    }
}

// ------------------------------------------------------------ mixed (delta form)
// The FP32 sweep cannot form F(qold + dq) - F(qold) as a difference of two
// O(1) fluxes: near convergence that difference drowns in FP32 rounding and
// the solve stalls.  It forms the change directly from dq (dflux_k), so its
// FP32 error is relative to the change itself; items publish dq only (FP32 for
// the terms, FP64 for the entity's own backward step) and form no primitives.
struct SweepRecM {
    float rho, ru, rv, E, u, v, p, un, nx, ny;  // the slot's record, as dflux_k reads it
};

// LU-SGS normal flux change F(q + dq) - F(q) along (nx, ny), component k (the
// lane's masks), in FP32 and in delta form: from dq and q's state and
// primitives, never as the difference of two O(1) fluxes, so its rounding
// error is relative to the change itself.
// F = ((E + p) u.n, rho u.n, rho u.n u + p nx, rho u.n v + p ny).
__device__ __forceinline__ float dflux_k(const SweepRecM& e, float gm1, const float dq[4], unsigned m0, unsigned m1,
                                         unsigned m2) {
    const float dE = dq[0], dr = dq[1], dru = dq[2], drv = dq[3];
    const float rn = e.rho + dr;
    const float du = (dru - e.u * dr) / rn, dv = (drv - e.v * dr) / rn;
    const float u2 = e.u + du, v2 = e.v + dv;
    const float dp = gm1 * (dE - 0.5f * (dru * u2 + e.ru * du + drv * v2 + e.rv * dv));
    const float dun = du * e.nx + dv * e.ny;
    const float un2 = e.un + dun;
    const float df1 = dr * un2 + e.rho * dun;  // change of rho u.n
    const float run = e.rho * e.un;
    // k = 0 (dE + dp) un2 + (E + p) dun, k = 1 df1, k = 2 and 3 df1 (u2 or v2)
    // + run (du or dv) + dp (nx or ny)
    const float s = pick(m0, dE + dp, df1) * pick(m0, un2, pick(m2, u2, v2)) + pick(m0, e.E + e.p, run) * pick(m0, dun, pick(m2, du, dv));
    return pick(m1, df1, pick(m0, s, s + dp * pick(m2, e.nx, e.ny)));
}

// Fields of an entry: two floats to a field.
enum { MF_R01, MF_R23, MF_UV, MF_PUN, MF_N, MF_DSOL, MF_DQ01, MF_DQ23, MF_D, MF_O, MF_R, MF_CODE, MF_COUNT };
typedef SweepRing<MF_COUNT> RingM;
typedef SweepBox<1> BoxM;  // dq in FP32

// kCC: the reference halves the sum of the terms; here res is doubled and the
// diagonal's reciprocal halved instead.  (NCFVM halves each term in FP32.)
template <bool kCC>
__device__ __forceinline__ void sweep_feed_mixed(const SweepArgs& a, RingM& R, int kbeg, int kend, int lane) {
    const int slot = lane >> 2;
    RingPos pos;
    int last = -1;
    int4 S = a.sched[kbeg];
    for (int kk = kbeg; kk < kend; ++kk) {
        const int4 Sn = kk + 1 < kend ? a.sched[kk + 1] : make_int4(0, 0, 0, 0);
        const int it = S.x, pass = S.y, ntake = S.w;
        int base = 0;
        do {
            const bool take = base + slot < ntake;
            float4 x = make_float4(1.f, 0.f, 0.f, 0.f), b = make_float4(0.f, 0.f, 0.f, 0.f), c = b, d = b;
            double D = 1.0, o = 1.0, r = 0.0;
            int src = -1;
            if (take) {
                src = a.rec_src[S.z + base + slot];
                const float4* p = reinterpret_cast<const float4*>(a.rec) + 4 * (size_t)(S.z + base + slot);
                x = p[0]; b = p[1]; c = p[2]; d = p[3];
            }
            if (base == 0 && lane < 4) {
                D = a.diag[it];
                o = reinterpret_cast<const double*>(&a.qold[it])[lane];
                if (pass == 0) r = reinterpret_cast<const double*>(&a.res[it])[lane];
            }
            const int code = take ? (__float_as_int(d.y) << 1) | pass : -1;
            const bool nb = take && code != last, own = base == 0 && lane < 4 && pass == 1 && (it << 1) != last;
            if (!mbar_wait(&R.empty[pos.stage], pos.phase ^ 1, RingWait(&R.abort, a))) return;
            double(*f)[32] = R.f[pos.stage];
            f[MF_R01][lane] = pack2(x.x, x.y); f[MF_R23][lane] = pack2(x.z, x.w);
            f[MF_UV][lane] = pack2(b.x, b.y); f[MF_PUN][lane] = pack2(b.z, b.w);
            f[MF_N][lane] = pack2(c.x, c.y); f[MF_DSOL][lane] = pack2(c.z, c.w);
            f[MF_CODE][lane] = dmake((d.x < 0.f ? 0x80000000u : 0u) | (unsigned)(src + 1), (unsigned)code);
            // (an idle slot computes on ones: a zero numerator takes the FP32
            // division's slow path, some 300 cycles of every item)
            const double none = nb ? unset() : pack2(1.f, 1.f);
            f[MF_DQ01][lane] = none; f[MF_DQ23][lane] = none;
            if (base == 0) {
                f[MF_D][lane] = kCC ? dhalf(D) : D;
                f[MF_O][lane] = o;
                f[MF_R][lane] = own ? unset() : (kCC ? r + r : r);
                if (lane == 0) R.item[pos.stage] = S;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&R.full[pos.stage]);
            pos.next();
            base += 8;
        } while (base < ntake);
        last = (it << 1) | pass;
        if (last == a.skip_code) last = -1;
        S = Sn;
    }
}

__device__ __forceinline__ void sweep_poll_mixed(const SweepArgs& a, RingM& R, const BoxM* boxes, int kbeg, int kend, int lane) {
    RingPos pos;
    int entries = 0;
    for (int kk = kbeg; kk < kend; ++kk) {
        int ntake = 0, base = 0;
        do {
            if (!mbar_wait(&R.full[pos.stage], pos.phase, RingWait(&R.abort, a))) return;
            double(*f)[32] = R.f[pos.stage];
            const int4 S = R.item[pos.stage];
            if (base == 0) ntake = S.w;
            const long long cs = __double_as_longlong(ld_field(&f[MF_CODE][lane]));
            const int code = (int)cs;
            int src = src_of(cs);
            bool nb = is_unset(ld_field(&f[MF_DQ23][lane]));
            bool own = base == 0 && lane < 4 && is_unset(ld_field(&f[MF_R][lane]));
            const float4* p = a.outf + (size_t)(code & 1) * a.n + (nb ? code >> 1 : 0);
            const double* po = reinterpret_cast<const double*>(a.outd + (own ? S.x : 0)) + lane;
            long long t0 = 0;
            for (int spins = 0; nb || own; ++spins) {
                if (nb) {
                    float w[4];
                    if (src >= 0) {
                        const BoxM& b = boxes[src >> kSrcBits];
                        const int idx = src & ((1 << kSrcBits) - 1), seq = ld_acquire(&b.seq[idx % kBox]);
                        const volatile float* q = reinterpret_cast<const volatile float*>(b.rec[idx % kBox]);
                        w[0] = q[0]; w[1] = q[1]; w[2] = q[2]; w[3] = q[3];
                        __threadfence_block();
                        const bool same = seq == idx && *(const volatile int*)&b.seq[idx % kBox] == idx;
                        if (!same) w[0] = __uint_as_float(kUnsetF);
                        if ((seq < 0 ? ~seq : seq) > idx) src = -1;  // the slot has moved on
                    } else {
                        peek_f4(p, w);
                    }
                    if (set_f4(w)) {
                        st_field(&f[MF_DQ01][lane], pack2(w[0], w[1]));
                        st_field(&f[MF_DQ23][lane], pack2(w[2], w[3]));
                        nb = false;
                    }
                }
                if (own) {
                    const double r = ld_relaxed(po);
                    if (!is_unset(r)) { st_field(&f[MF_R][lane], r); own = false; }
                }
                if ((nb || own) && !poller_go_on(spins, t0, a, &R.abort)) {
                    *(volatile int*)&R.abort = 1;
                    break;
                }
            }
            if (__any_sync(0xffffffffu, nb || own)) return;
            __syncwarp();
            if (lane == 0) st_release(&R.ready, ++entries);
            pos.next();
            base += 8;
        } while (base < ntake);
    }
}

struct SweepEntryM {
    double r01, r23, uv, pun, nn, dsol, q01, q23, D, o, r;
    long long code;
    int4 item;
    __device__ __forceinline__ void load(const RingM& R, int stage, int lane, bool first) {
        const double(*f)[32] = R.f[stage];
        if (first) {
            item = R.item[stage];
            D = f[MF_D][lane]; o = f[MF_O][lane]; r = f[MF_R][lane];
        }
        code = __double_as_longlong(f[MF_CODE][lane]);
        q01 = f[MF_DQ01][lane]; q23 = f[MF_DQ23][lane];
        r01 = f[MF_R01][lane]; r23 = f[MF_R23][lane]; uv = f[MF_UV][lane]; pun = f[MF_PUN][lane];
        nn = f[MF_N][lane]; dsol = f[MF_DSOL][lane];
    }
};

template <bool kCC>
__device__ __forceinline__ void sweep_items_mixed(const SweepArgs& a, RingM& R, BoxM& box, int kbeg, int kend, int lane) {
    const unsigned all = 0xffffffffu;
    const int k = lane & 3;
    const float gm1 = (float)a.gm1;
    const unsigned m0 = lane_mask(k == 0), m1 = lane_mask(k == 1), m2 = lane_mask(k == 2);
    RingPos pos;
    int last = -1;
    float LF[4] = {0.f, 0.f, 0.f, 0.f};  // previous item's dq (FP32)
    double Lk = 0.0;                     // and in FP64, component k
    SweepEntryM X;
    X.r = 0.0;
    int entries = 0;
    for (int kk = kbeg; kk < kend; ++kk) {
        double cres = 0.0;
        const int idx = kk - kbeg, bslot = idx % kBox;
        if (lane == 0) box_open(box, idx);
        int it = 0, pass = 0, ntake = 0, base = 0;
        do {
            if (!entry_wait(&R.ready, ++entries, RingWait(&R.abort, a))) return;
            X.load(R, pos.stage, lane, base == 0);
            __syncwarp();
            if (lane == 0) mbar_arrive(&R.empty[pos.stage]);
            pos.next();
            if (base == 0) {
                it = X.item.x; pass = X.item.y; ntake = X.item.w;
                if (ntake == 0) break;
            }
            const bool mine = (int)X.code == last && (int)X.code >= 0;
            const float dq[4] = {mine ? LF[0] : low_f(X.q01), mine ? LF[1] : high_f(X.q01), mine ? LF[2] : low_f(X.q23),
                                 mine ? LF[3] : high_f(X.q23)};
            const SweepRecM E = {low_f(X.r01), high_f(X.r01), low_f(X.r23), high_f(X.r23), low_f(X.uv), high_f(X.uv),
                                 low_f(X.pun), high_f(X.pun), low_f(X.nn), high_f(X.nn)};
            const float df = dflux_k(E, gm1, dq, m0, m1, m2);
            const float dqk = k == 0 ? dq[0] : (k == 1 ? dq[1] : (k == 2 ? dq[2] : dq[3]));
            const double t = widen(kCC ? low_f(X.dsol) * df - high_f(X.dsol) * dqk
                                       : 0.5f * ((X.code < 0 ? -df : df) * low_f(X.dsol) - high_f(X.dsol) * dqk));
            const int nr = min(8, ntake - base);
            int e = 0;
            if (base == 0) { cres = zero_plus(__shfl_sync(all, t, k)); e = 1; }  // 0.0 + t0, exact
            for (; e < nr; ++e) cres = add64(cres, __shfl_sync(all, t, 4 * e + k));
            base += 8;
        } while (base < ntake);
        double d;
        if (pass == 0) {
            d = mul64(sub64(neg64(X.r), cres), X.D);
        } else {  // from the entity's own forward dq
            d = sub64((it << 1) == last ? Lk : X.r, mul64(cres, X.D));
        }
        const float df = narrow(d);
        LF[0] = __shfl_sync(all, df, 0);
        LF[1] = __shfl_sync(all, df, 1);
        LF[2] = __shfl_sync(all, df, 2);
        LF[3] = __shfl_sync(all, df, 3);
        const double L0 = __shfl_sync(all, d, 0), L1 = __shfl_sync(all, d, 1), L2 = __shfl_sync(all, d, 2),
                     L3 = __shfl_sync(all, d, 3);
        Lk = k == 0 ? L0 : (k == 1 ? L1 : (k == 2 ? L2 : L3));
        last = (it << 1) | pass;
        const size_t slotr = (size_t)pass * a.n + it;
        if (last == a.skip_code) {  // test hook: this item publishes nothing and hands nothing on
            last = -1;
        } else {
            if (lane == 0) {
                box.rec[bslot][0] = make_double2(pack2(LF[0], LF[1]), pack2(LF[2], LF[3]));
                st_release(&box.seq[bslot], idx);
            }
            publish_mixed(lane, a.outf + slotr, reinterpret_cast<double2*>(a.outd + slotr), LF, L0, L1, L2, L3);
            if (pass == 1 && lane < 4) reinterpret_cast<double*>(&a.qc[it])[lane] = add64(X.o, d);
        }
    }
}

// The body of both solvers' sweep kernels, one block per SM.
template <bool kCC, bool kMixed>
__device__ __forceinline__ void sweep_block(const SweepArgs& a, const int* __restrict__ woff) {
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ __align__(16) double wxs[kSweepPairs][32];  // per sweep warp: exchange of lane values
    typedef typename std::conditional<kMixed, RingM, RingD>::type Ring;
    typedef typename std::conditional<kMixed, BoxM, BoxD>::type Box;
    Ring* rings = reinterpret_cast<Ring*>(sweep_smem);
    Box* boxes = reinterpret_cast<Box*>(sweep_smem + kSweepPairs * sizeof(Ring));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wib = warp % kSweepPairs, role = warp / kSweepPairs;
    if (threadIdx.x < kSweepPairs) { ring_init(rings[threadIdx.x]); box_init(boxes[threadIdx.x]); }
    __syncthreads();
    const int gw = blockIdx.x * kSweepPairs + wib;
    const int kbeg = woff[gw], kend = woff[gw + 1];
    if (kbeg >= kend) return;
    Ring& R = rings[wib];
    if constexpr (kMixed) {
        if (role == 0) sweep_items_mixed<kCC>(a, R, boxes[wib], kbeg, kend, lane);
        else if (role == 1) sweep_feed_mixed<kCC>(a, R, kbeg, kend, lane);
        else sweep_poll_mixed(a, R, boxes, kbeg, kend, lane);
    } else {
        if (role == 0) sweep_items<kCC>(a, R, boxes[wib], wxs[wib], kbeg, kend, lane);
        else if (role == 1) sweep_feed(a, R, kbeg, kend, lane);
        else sweep_poll(a, R, boxes, kbeg, kend, lane);
    }
}

template <bool kMixed>
constexpr int sweep_smem_bytes() {
    return kSweepPairs * (int)(kMixed ? sizeof(RingM) + sizeof(BoxM) : sizeof(RingD) + sizeof(BoxD));
}

// Lets a sweep kernel take its dynamic shared memory (over 48 KB).
template <bool kMixed, class K>
cudaError_t sweep_allow_smem(K kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sweep_smem_bytes<kMixed>());
}

}  // namespace uns
