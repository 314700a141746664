// xtma.cu -- TMA-fed x-march stage kernel (the fast path of the fused stage).
//
// A CTA owns TZ z rows x one velocity block (32 velocities in FP64, 64 in FP32)
// x one flavour half and marches along x:
//   * a producer warpgroup (one issuing lane) loads, for every x plane the CTA
//     touches, the plane's [TZ+2R rows][4 fields][velocities] box with one TMA
//     tensor load (cp.async.bulk.tensor.4d; two where the periodic z wrap
//     cuts it), the TZ cells' moments with a bulk copy, and the stage's
//     pointwise input (U in S2 and S3, B in S4; none in S1) of the plane that
//     the box completes, into shared-memory rings whose completion is tracked
//     by "full" mbarriers (expect_tx bytes).  A box is used twice: as the front
//     (x+R) of the march, where all its rows enter the stencil sums, and R
//     planes later for its centre values, so each state value crosses HBM once;
//   * consumer warps never exchange data and there is no CTA-wide barrier in
//     the march: a warp waits only on full barriers and arrives on a slot's
//     "empty" barrier after its last use;
//   * each consumer thread owns two z rows of one 8-byte value (a double, or two
//     floats in packed arithmetic) per field: the 2R+2 rows it reads from a box
//     serve both rows' z stencils (8 shared loads per field for two points
//     instead of 14), and the per-velocity constants are held in registers;
//   * the x stencil is kept in transposed form: 2R partial sums per value,
//     each front value added to all of them, so nothing is shifted and the
//     products of a value do not depend on each other;
//   * moment partials (FP64 products and sums; FP32 state may sum in float
//     within the block, stored as double): a warp's half-warps exchange values
//     so that the lower one keeps the grid's even row and the upper one the odd
//     one (no sum depends on the tile that a row falls into), each lane forms the 12 products (3
//     combinations x 4 weights, the weights in a lane-permuted order set once
//     per tile) of its own and its partner's velocities, and the half-warp
//     reduce-scatters them with 12 shuffle-adds;
//   * a stopped instance of a batch (its halt flag set by the device-side
//     stop test) has its tiles skipped.
// All mbarrier waits are bounded: on expiry the kernel records the timeout in
// the status word, stops marching and, before returning, waits (again
// bounded) for the copies it issued.  nz need not be a multiple of TZ (ZTiles).
//
// What bounds it, measured on a 512 x 256 x 642 FP64 grid (KO6): S1 2.6 ms (2
// state passes, 4.1 TB/s) is held by instruction latency at 8 consumer warps
// per SM (two per scheduler: the partial sums alone take 96 registers); S2 4.6,
// S3 3.1, S4 3.1 ms run at 4.7-5.3 TB/s of the 6.5 a plain copy reaches.  The
// form before -- 16 warps of one point per thread, a 7-deep register queue in x
// shifted every plane, weights read from shared memory, plain loads of the
// pointwise inputs, warp 0 issuing the copies -- took 3.9 / 5.0 / 4.5 / 4.6 ms:
// 404-467 instructions and 112 shared-memory wavefronts per 32 points against
// about 240 and 70 now, with the shared-memory pipe at 65 %.
// FP32 (same grid): 2.2 / 2.8 / 2.4 / 2.5 -> 1.7 / 2.2 / 1.7 / 1.8 ms.
//
// The file is compiled in parts (NUOSC_PART, build.py), each with its share of the
// kernels: the whole in one piece takes 7 minutes.  (nvcc's --split-compile halves
// that, but one source then gave one of two codes by chance, 5 to 8 % apart, small
// grids up to 18 %.)  What the compiler decided in the one or the other way is
// written out: a loop for the fronts that complete no centre, loads in program
// order, no branch on what is the same in every plane.  Against the better of the
// two codes (geometric mean over 16 to 512 cells a side, 12 to 642 velocities):
// steps FP64 1.05, FP32 1.08, calRHS 1.07 and 1.09, batches 1.06 to 1.10.
//
// The march of one tile is a device function shared by two kernels: k_xtma
// (one tile per CTA, one instance per launch) and k_xtma_batch (a persistent
// grid whose CTAs take tiles of many instances from a work-list).
#include "internal.cuh"
#include "physics.cuh"
#include "tail.cuh"

#include <cuda.h>

#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>

#ifndef NUOSC_PART
#error "compiled once per part: -DNUOSC_PART=0 ... 10"
#endif
#pragma nv_diag_suppress 177  // each part leaves some functions unused

namespace nuosc {

namespace {

// bounded mbarrier waits: a poll of a phase that has not completed suspends
// the thread for about 4 us on B200 (nuosc_selftest_wait_timeout), so 2^18
// polls give up after about 1 s
constexpr unsigned kWaitSpins = 1u << 18;

// One 8-byte value of the march: a double, or two floats of adjacent velocities
// in one register pair (packed f32x2 arithmetic).  A thread owns one such value
// per row and field, so a warp covers 32 velocities in FP64 and 64 in FP32, and
// RW z rows.  Every product that is added to something is an explicit fma and
// the other operations are not contracted, so all kernels that share the march
// round alike (a batch member equals its solo run bit for bit).
template <typename T>
constexpr int vpt() {
    return 8 / (int)sizeof(T);
}
template <typename T>
constexpr int vblock() {
    return 32 * vpt<T>();
}
constexpr int RW = 2;
constexpr int threads_of(int tz) { return 32 * (tz / RW) + 128; }  // consumer warps and the producer's warpgroup

struct f2 {
    unsigned long long v;
};
__device__ __forceinline__ f2 pack(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double vmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double vsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 vadd(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 vmul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 vsub(f2 a, f2 b) { return vfma(b, pack(-1.f, -1.f), a); }
__device__ __forceinline__ f2 vneg(f2 a) { return f2{a.v ^ 0x8000000080000000ull}; }

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Loads and predicated stores of a value, in program order (volatile) and without a
// branch: conditions that are the same in every plane (a lane past the last
// velocity, a row that is not the tile's) must not become control flow, which the
// compiler hoists out of the march by copying the loop, and worse code.
//   ldg: *p from global memory where `on`, else 0;  lds: from shared memory
//   st_if: to global memory where `on`
template <typename T>
struct VecOf;
template <>
struct VecOf<double> {
    using V = double;
    static __device__ __forceinline__ V splat(double x) { return x; }
    static __device__ __forceinline__ V make(const double (&x)[1]) { return x[0]; }
    static __device__ __forceinline__ void get(V a, double (&x)[1]) { x[0] = a; }
    static __device__ __forceinline__ V ldg(const double *p, int on) {
        V r;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @p ld.global.f64 %0, "
            "[%1];\n}\n"
            : "=d"(r)
            : "l"(p), "r"(on)
            : "memory");
        return r;
    }
    static __device__ __forceinline__ V lds(const double *p) {
        V r;
        asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(r) : "r"(smem_u32(p)));
        return r;
    }
    static __device__ __forceinline__ void st_if(double *p, V a, int on) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.global.f64 [%0], %1;\n}\n" ::"l"(p), "d"(a),
                     "r"(on)
                     : "memory");
    }
    static __device__ __forceinline__ V zero() { return 0.0; }
    static __device__ __forceinline__ unsigned long long bits(V a) { return __double_as_longlong(a); }
};
template <>
struct VecOf<float> {
    using V = f2;
    static __device__ __forceinline__ V splat(double x) { return pack((float)x, (float)x); }
    static __device__ __forceinline__ V make(const double (&x)[2]) { return pack((float)x[0], (float)x[1]); }
    static __device__ __forceinline__ void get(V a, float (&x)[2]) {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x[0]), "=f"(x[1]) : "l"(a.v));
    }
    static __device__ __forceinline__ V ldg(const float *p, int on) {
        V r;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n mov.b64 %0, 0;\n @p ld.global.b64 %0, [%1];\n}\n"
            : "=l"(r.v)
            : "l"(p), "r"(on)
            : "memory");
        return r;
    }
    static __device__ __forceinline__ V lds(const float *p) {
        V r;
        asm volatile("ld.shared.b64 %0, [%1];\n" : "=l"(r.v) : "r"(smem_u32(p)));
        return r;
    }
    static __device__ __forceinline__ void st_if(float *p, V a, int on) {
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.global.b64 [%0], %1;\n}\n" ::"l"(p), "l"(a.v),
                     "r"(on)
                     : "memory");
    }
    static __device__ __forceinline__ V zero() { return f2{0ull}; }
    static __device__ __forceinline__ unsigned long long bits(V a) { return a.v; }
};

struct __align__(64) TmaMaps {
    CUtensorMap zr;   // box of TZ+2R rows (plane box with both halos)
    CUtensorMap tzr;  // TZ+R rows (a box cut by the wrap)
    CUtensorMap r;    // R rows (wrapped halo)
    CUtensorMap pu;   // TZ rows of the stage's U register (pointwise input)
    CUtensorMap pa;   // TZ rows of the final stage's B input (acc_src; pointwise)
    // the same three box shapes over a slab's halo buffer (planes right of the slab),
    // kHalo maps further on
    CUtensorMap hzr, htzr, hr;
    static constexpr int kHalo = 5;
};

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// register split between the warpgroups of a CTA (RegSplit)
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N));
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned spins = kWaitSpins) {
#pragma unroll 1
    for (unsigned it = 0; it < spins; ++it) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// make generic-proxy writes of a tensor map in global memory visible to the TMA
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap *m) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(m) : "memory");
}
__device__ __forceinline__ void mbar_inval(unsigned bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                            unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];\n" ::"r"(dst),
        "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void sink_if(unsigned dst, unsigned long long x, int on) {
    asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p st.shared.b64 [%0], %1;\n}\n" ::"r"(dst), "l"(x), "r"(on)
                 : "memory");
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

constexpr int up128(int x) { return (x + 127) / 128 * 128; }

// one ring slot: box [ZR][4][VB] T | moments [TZ][12] double
template <typename T, int TZ, int R>
struct Slot {
    static constexpr int VB = vblock<T>();
    static constexpr int ZR = TZ + 2 * R;
    static constexpr int box = 0;
    static constexpr int mb = up128(box + (int)sizeof(T) * ZR * 4 * VB);
    static constexpr int bytes = up128(mb + 8 * TZ * NMOM);
    static constexpr unsigned tx = sizeof(T) * ZR * 4 * VB + 8 * TZ * NMOM;  // bytes landing per plane
};

// The stencil of one field at one point, eps_z KO_z + eps_x KO_x + fz ADV_z
// + fx ADV_x with
//   KO  (unit strength) 6th: s[0]+s[6] - 6 (s[1]+s[5]) + 15 (s[2]+s[4]) - 20 s[3]
//                       4th: s[0]+s[4] - 4 (s[1]+s[3]) + 6 s[2]
//   ADV = s[C-2] - s[C+2] - 8 (s[C-1] - s[C+1]) (the 4th-order central
//         difference before its factor f = -v/(12 dx)),
// is evaluated as one weighted sum per axis: the four neighbours at offsets
// -2, -1, +1, +2 carry per-velocity weights (KO and ADV coefficients folded
// together, stencil_weights), the pair at +-3 (6th difference only) the uniform
// eps, and the centre, shared by both axes, -20 (eps_z + eps_x) or
// 6 (eps_z + eps_x).  That is 14 (6th) or 10 (4th) FP64 operations per field
// instead of 22 (18) for the separate KO and ADV sums.
//   6th: w = {-6 eps + f, 15 eps - 8 f, 15 eps + 8 f, -6 eps - f}
//   4th: w = {eps + f, -4 eps - 8 f, -4 eps + 8 f, eps - f}
template <int R>
__device__ __forceinline__ void stencil_weights(double eps, double f, double (&w)[4]) {
    if (R == 3) {
        w[0] = fma(-6.0, eps, f);
        w[1] = fma(15.0, eps, -8 * f);
        w[2] = fma(15.0, eps, 8 * f);
        w[3] = fma(-6.0, eps, -f);
    } else {
        w[0] = __dadd_rn(eps, f);
        w[1] = fma(-4.0, eps, -8 * f);
        w[2] = fma(-4.0, eps, 8 * f);
        w[3] = __dsub_rn(eps, f);
    }
}

// inp (physics.cuh) with its fmas explicit
__device__ __forceinline__ double contract4(const double *m, double vx, double vy, double vz) {
    return fma(-m[3], vz, fma(-m[2], vy, fma(-m[1], vx, m[0])));
}

// s/3 + t as third_plus (physics.cuh)
template <typename T>
__device__ __forceinline__ typename VecOf<T>::V vthird_plus(typename VecOf<T>::V s, typename VecOf<T>::V t) {
    using O = VecOf<T>;
    const auto third = O::splat(1.0 / 3.0);
    const auto q = vmul(s, third);
    const auto r = vfma(q, O::splat(-3.0), s);
    return vadd(q, vfma(r, third, t));
}

// one axis's differences of calRHS, taken before any product (adv_axis, ko_axis
// of physics.cuh): s[-2] - s[2] - 8 (s[-1] - s[1]) and the unit-strength KO sum
template <typename T, int R, typename V>
__device__ __forceinline__ V adv_diff(const V (&s)[2 * R + 1]) {
    using O = VecOf<T>;
    return vfma(O::splat(-8.0), vsub(s[R - 1], s[R + 1]), vsub(s[R - 2], s[R + 2]));
}
template <typename T, int R, typename V>
__device__ __forceinline__ V ko_sum(const V (&s)[2 * R + 1]) {
    using O = VecOf<T>;
    const V t2 = vadd(s[R - 2], s[R + 2]), t1 = vadd(s[R - 1], s[R + 1]);
    if constexpr (R == 3) {
        const V t3 = vadd(s[0], s[6]);
        return vfma(O::splat(-20.0), s[3], vfma(O::splat(15.0), t1, vfma(O::splat(-6.0), t2, t3)));
    } else {
        return vfma(O::splat(6.0), s[2], vfma(O::splat(-4.0), t1, t2));
    }
}

// statically allocated per-CTA scratch of the march
struct MarchShared {
    unsigned long long sink;  // a lane's values of a row that is not the tile's to store
    int abort;                // a bounded wait expired
};

template <typename T, int TZ>
constexpr int tma_ctas_per_sm() {
    return TZ == 16 ? 1 : 2;
}

// Ring geometry of one march.  A box lives from its issue, D planes ahead of
// its front use, to its centre use, R planes after it; a stage with a pointwise
// input (U in S2 and S3, B in S4) has a second ring of D plane pieces of it.  D
// is what the shared memory of one (TZ = 16) or two (TZ = 8) CTAs per SM holds.
template <typename T, int R, int MODE, int TZ>
struct MarchCfg {
    static constexpr bool PU = MODE == MODE_SY || MODE == MODE_S2B;  // reads U pointwise
    static constexpr bool PA = MODE == MODE_S4B;                     // reads B pointwise
    static constexpr bool PW = PU || PA;
    static constexpr int D = PW ? (R == 3 ? 3 : 4) : (TZ == 8 && R == 3 ? 4 : 5);
    static constexpr int NS = R + D;
    static constexpr int PS = PW ? D : 0, PSM = PW ? D : 1;
    static constexpr unsigned pbytes = sizeof(T) * TZ * 4 * vblock<T>();
    static constexpr size_t ring = (size_t)NS * Slot<T, TZ, R>::bytes;
    static constexpr size_t bars = ring + PS * pbytes;
    static constexpr size_t smem = bars + 2 * NS * 8;  // box ring | pointwise ring | mbarriers
};

// Registers per thread after the split: a CTA starts with the even share of the
// SM's 65,536 (168 for 256 + 128 threads, 128 for two CTAs of 128 + 128), its
// producer warpgroup gives up all but `producer`, which is what the consumers
// take: 256 x 232 + 128 x 40 = 384 x 168, 128 x 216 + 128 x 40 = 256 x 128.
template <int TZ>
struct RegSplit {
    static constexpr int producer = 40, consumer = TZ == 16 ? 232 : 216;
};

}  // namespace

// value of x, re-read from (shared) memory at each use when V: keeps values
// that are loop-invariant but cheap to re-read out of the register file
template <bool V, typename P>
__device__ __forceinline__ P rd(const P &x) {
    if constexpr (V) return *(const volatile P *)&x;
    else return x;
}

// One tile of work: z rows z0..z0+TZ-1, velocity block vb (of nvb), x planes
// xs..xe-1, flavour half `half`.  The first `skip` rows are the tile before's
// (ZTiles): nothing of them is stored here.
struct Tile {
    int z0, vb, nvb, xs, xe, half, skip;
};

// The march of one tile of the instance (maps, a): every thread of the CTA calls
// xtma_produce (the last warpgroup) or xtma_consume (the others); both return
// true when a bounded wait expired (the status word is set and the tile is
// incomplete).  Called by the single-instance kernel (one tile per CTA; a and
// maps in kernel parameter space) and by the persistent batched kernel (many
// tiles per CTA, of many instances; SA: a in shared memory); the arithmetic per
// (cell, velocity) does not depend on which.
//
// Producer: one lane loads box j (plane xs + j, periodic) and, for the stages
// with a pointwise input, that input's TZ rows of plane j - R, into slots
// j % NS and (j - R) % PS; one full barrier per box slot (phase j / NS) counts
// the bytes of both.  It may refill a slot when every consumer warp has
// arrived on the slot's empty barrier, D planes later.
// fault_tx (the self-test of the bounded waits) over-declares the bytes of box
// R of the instance's first tile: all its copies land, its phase never completes.
template <typename T, int R, int MODE, int TZ, bool SA>
__device__ __forceinline__ bool xtma_produce(const TmaMaps &maps, const StageArgs<T> &a, const Tile &t,
                                             unsigned char *smem, MarchShared &sh, bool early = false) {
    using S = Slot<T, TZ, R>;
    using CF = MarchCfg<T, R, MODE, TZ>;
    constexpr int NS = CF::NS, ZR = S::ZR;
    unsigned long long *bars = (unsigned long long *)(smem + CF::bars);  // full[NS], empty[NS]
    const bool lead = threadIdx.x == 32 * (TZ / RW);
    if (lead) {
        sh.abort = 0;
        for (int s = 0; s < 2 * NS; ++s) mbar_init(smem_u32(&bars[s]), s < NS ? 1u : (unsigned)(TZ / RW));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    int issued = 0;  // last box issued + 1
    if (lead) {
        const int nx = a.g.nx, nz = a.g.nz, c0 = t.vb * S::VB, c1 = 4 * t.half, nplanes = t.xe - t.xs;
        const bool halo = a.halo != nullptr;
        // the box in z, the same for every plane: one piece, or two where the periodic
        // wrap cuts it (the first tile's after R rows, the last one's before the last R)
        const int cut = t.z0 == 0 ? R : t.z0 + TZ == nz ? TZ + R : ZR;
        const int za = t.z0 == 0 ? nz - R : t.z0 - R;
        const CUtensorMap *piece1 = cut == ZR ? &maps.zr : cut == R ? &maps.r : &maps.tzr;
        const CUtensorMap *piece2 = cut == R ? &maps.tzr : &maps.r;
        const double *mom = a.mom_in + (long long)t.z0 * NMOM;
        const unsigned fault_tx = t.z0 == 0 && t.vb == 0 && t.xs == 0 && t.half == 0 ? a.fault_tx : 0u;
        if (!SA && early) grid_wait();
        int s = 0, ps = 0;       // slots of box j and of the pointwise rows of plane j - R
        unsigned refills = 0;    // times slot s has been filled
#pragma unroll 1
        for (int j = 0; j < nplanes + R; ++j) {  // centres xs..xe-1 and fronts up to xe-1+R
            if (refills > 0 && (*(volatile int *)&sh.abort || !mbar_wait(smem_u32(&bars[NS + s]), (refills - 1) & 1))) {
                sh.abort = 1;
                break;
            }
            const unsigned full = smem_u32(&bars[s]);
            unsigned char *sp = smem + s * S::bytes;
            const bool pw = CF::PS > 0 && j >= R;
            mbar_expect_tx(full, S::tx + (pw ? CF::pbytes : 0u) + (j == R ? fault_tx : 0u));
            // past the last plane it wraps (periodic) or, in a slab, comes from
            // the halo buffer's right planes (box plane x - nx + R).  Boxes
            // start at plane xs >= 0, so the left halo is never a box.
            const int xl = t.xs + j;  // < nx + R < 2 nx
            const bool hal = xl >= nx && halo;
            const int x = hal ? xl - nx + R : xl >= nx ? xl - nx : xl, h = hal ? TmaMaps::kHalo : 0;
            tma_load_4d(smem_u32(sp + S::box), piece1 + h, c0, c1, za, x, full);
            if (cut < ZR)
                tma_load_4d(smem_u32(sp + S::box + cut * 4 * S::VB * (int)sizeof(T)), piece2 + h, c0, c1, 0, x, full);
            // the cell moments are read at a box's centre use, which is always an
            // interior plane; a halo box (front use only) loads plane nx-1's, unread
            bulk_load(smem_u32(sp + S::mb), mom + (long long)(hal ? nx - 1 : x) * nz * NMOM, 8u * TZ * NMOM, full);
            if (pw) {
                tma_load_4d(smem_u32(smem + CF::ring + ps * CF::pbytes), CF::PU ? &maps.pu : &maps.pa, c0, c1, t.z0,
                            t.xs + j - R, full);
                ps = ps + 1 < CF::PSM ? ps + 1 : 0;
            }
            if (++s == NS) s = 0, ++refills;
            issued = j + 1;
        }
    }
    __syncthreads();
    const bool aborted = sh.abort != 0;
    if (lead) {
        if (aborted) {
            // a wait expired: report it, then wait (bounded) for the copies of
            // the last NS boxes issued -- the only ones that may still be in
            // flight: box j - NS of a slot was consumed (so had landed) before
            // box j was issued into it -- before the CTA's shared memory is
            // reused or released
            if (a.status) atomicExch(a.status, NUOSC_TIMEOUT_CODE);
            for (int j = issued > NS ? issued - NS : 0; j < issued; ++j)
                mbar_wait(smem_u32(&bars[j % NS]), (unsigned)((j / NS) & 1));
        }
        for (int s = 0; s < 2 * NS; ++s) mbar_inval(smem_u32(&bars[s]));
    }
    return aborted;
}

// VAC compiles the vacuum term in (it then runs where a.c.pmo != 0), RAG the rows
// that are the tile before's (grids that TZ does not divide).
template <typename T, int R, int MODE, int TZ, bool VAC, bool SA, bool M64, bool RAG>
__device__ __forceinline__ bool xtma_consume(const StageArgs<T> &a, const Tile &t, unsigned char *smem,
                                             MarchShared &sh, bool early = false) {
    using S = Slot<T, TZ, R>;
    using CF = MarchCfg<T, R, MODE, TZ>;
    using O = VecOf<T>;
    using V = typename O::V;
    constexpr int NP = vpt<T>();  // velocities per thread
    constexpr int VB = S::VB;     // velocities per CTA
    constexpr int NS = CF::NS;
    unsigned long long *bars = (unsigned long long *)(smem + CF::bars);  // full[NS], empty[NS]

    const Geom g = a.g;
    const int z0 = t.z0, vb = t.vb, nvb = t.nvb, xs = t.xs, half = t.half;
    const int lane = threadIdx.x & 31, r = (threadIdx.x >> 5) * RW;  // this warp's rows r, r + 1
    const int v = vb * VB + NP * lane;  // first of this thread's NP velocities
    const bool vact = v < g.nvs;        // nvs is a multiple of NP, so all NP are active together
    const int nplanes = t.xe - xs, nboxes = nplanes + R;
    const int zr = z0 + r;  // < nz
    const long long fs = g.fs;
    const long long P = (long long)g.nz * g.nvs;
    const long long hoff = (long long)half * 4 * fs;
    const T *in = a.in + hoff;
    const int vc = vact ? v : 0;
    const long long own = (long long)zr * g.nvs + vc;
    // per-plane addressing in 32 bits: within one flavour half, a field's
    // offset f fs (f <= 3), a plane's x P and a cell's moment-partial index
    // all fit (xtma_supported requires 3 fs < 2^32); only the half's own
    // offset, hoff, needs 64 bits
    const unsigned fs32 = (unsigned)fs, P32 = (unsigned)P, own32 = (unsigned)own;
    // RAG: where both rows are the tile before's the warp only takes its part in the
    // ring; where the first is (keep0 false) the second alone is stored
    const bool keep0 = !RAG || t.skip <= r;
    const int put[RW] = {vact && keep0, vact}, sink = !keep0 && lane == 0;
    __syncthreads();  // the barriers are initialised
    if (RAG && t.skip >= r + RW) {
        for (int j = 0; j < nboxes; ++j) {
            if (!mbar_wait(smem_u32(&bars[j % NS]), (unsigned)((j / NS) & 1)) || *(volatile int *)&sh.abort) {
                sh.abort = 1;
                break;
            }
            if (j >= R && lane == 0) mbar_arrive(smem_u32(&bars[NS + (j - R) % NS]));
        }
        __syncthreads();
        return sh.abort != 0;
    }

    // the R planes left of the segment (periodic, or from a slab's halo buffer),
    // loaded ahead of the constants so that their latencies overlap
    V pre[R][4][RW];
    if (!SA && early) grid_wait();
    {
        const T *halo = rd<SA>(a.halo);
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const int pl = xs - R + b;
            const bool hal = halo != nullptr && pl < 0;
            const int px = pl >= 0 ? pl : hal ? pl + R : pl + g.nx;  // (xs >= 0, nx > R)
            const T *src = (hal ? halo + (long long)half * 8 * R * P : in) + ((long long)px * P + own);
            long long step = hal ? 2 * R * P : fs;
            asm volatile("" : "+l"(src), "+l"(step));  // one code for both sources
#pragma unroll
            for (int f = 0; f < 4; ++f)
#pragma unroll
                for (int w = 0; w < RW; ++w) pre[b][f][w] = O::ldg(src + f * step + w * g.nvs, vact);
        }
    }

    // per-velocity constants, in registers.  Lane-permuted moment weights: slot s
    // of a lane holds weight s ^ wq (weights w, w vx, w vy, w vz), wq = lane bits
    // 3..2, the order the moment reduce-scatter needs; of this lane's
    // velocities and of its partner's (lane ^ 16).
    using M = std::conditional_t<M64, double, float>;
    const int wq = (lane >> 2) & 3;
    const int vp = vb * VB + NP * (lane ^ 16);
    double vx[NP], vy[NP], vz[NP];
    M wo[NP][4], wp[NP][4];
    V wz[4], wx[4], fz, fx;
    {
        double tz[4][NP], tx[4][NP], tfz[NP], tfx[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            vx[p] = a.q.vx[vc + p];
            vy[p] = a.q.vy[vc + p];
            vz[p] = a.q.vz[vc + p];
            tfz[p] = vz[p] * a.c.fzs;
            tfx[p] = vx[p] * a.c.fxs;
            double w4z[4], w4x[4];
            stencil_weights<R>(a.c.kz, __dmul_rn(vz[p], a.c.fzs), w4z);
            stencil_weights<R>(a.c.kx, __dmul_rn(vx[p], a.c.fxs), w4x);
#pragma unroll
            for (int j = 0; j < 4; ++j) tz[j][p] = w4z[j], tx[j][p] = w4x[j];
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int vi = (o ? vp : v) + p;
                const bool in_row = vi < g.nvs;
                const int vj = in_row ? vi : 0;
                const double wd = in_row ? a.q.vw[vj] : 0.0;
                const double v4w[4] = {wd, a.q.vx[vj] * wd, a.q.vy[vj] * wd, a.q.vz[vj] * wd};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = j ^ wq;
                    const M w = M(k == 0 ? v4w[0] : k == 1 ? v4w[1] : k == 2 ? v4w[2] : v4w[3]);
                    if (o) wp[p][j] = w;
                    else wo[p][j] = w;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) wz[j] = O::make(tz[j]), wx[j] = O::make(tx[j]);
        fz = O::make(tfz);
        fx = O::make(tfx);
    }
    const V kz = O::splat(a.c.kz), kx = O::splat(a.c.kx), mu = O::splat(a.c.mu);
    const V kc = O::splat((R == 3 ? -20.0 : 6.0) * (a.c.kz + a.c.kx));  // centre weight of both axes
    const V cA = O::splat(a.cA), cY = O::splat(a.cY);
    const V p2s = O::splat(2 * a.c.pmo * a.c.st), p2c = O::splat(2 * a.c.pmo * a.c.ct), ps = O::splat(a.c.pmo * a.c.st);
    const bool vac = VAC && (!SA || a.c.pmo != 0.0);  // a batch's instances without a vacuum term skip it

    // x stencil in transposed form: sx[f][row][k] is the partial sum of the
    // centre plane (front - R + k) over the planes before the front.  A front
    // value F completes centre front - R and is added, with its tap's weight,
    // to the R..2R-1 others; the move to the next slot is the fma's own
    // destination, so nothing is shifted, and the 2R+1 products of a value are
    // independent of each other.
    // calRHS keeps the last 2R planes' values themselves (sx[f][row][k] = plane
    // front - 2R + k) and takes differences first, as the reference does: the
    // folded weights multiply whole values, whose rounding is that of the state
    // -- harmless in dt k, which is added to the state, but up to 10 times the
    // direct kernel's error (2e-6 against 2e-7 in float) when k is the result.
    constexpr bool RHS = MODE == MODE_RHS;
    V sx[4][RW][2 * R];
    auto tap = [&](int k) -> V {  // weight of a front value in centre (front - R + k)
        return R == 3 ? (k == 0 || k == 6 ? kx : k == 1 ? wx[3] : k == 2 ? wx[2] : k == 3 ? kc : k == 4 ? wx[1] : wx[0])
                      : (k == 0 ? wx[3] : k == 1 ? wx[2] : k == 2 ? kc : k == 3 ? wx[1] : wx[0]);
    };
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int w = 0; w < RW; ++w) {
            auto &q = sx[f][w];
#pragma unroll
            for (int k = 0; k < 2 * R; ++k) q[k] = O::zero();
#pragma unroll
            for (int b = 0; b < R; ++b) {
                const V F = pre[b][f][w];
                if constexpr (RHS) {
                    q[R + b] = F;
                } else {
#pragma unroll
                    for (int k = 0; k + 1 < 2 * R; ++k) q[k] = vfma(tap(k + 1), F, q[k + 1]);
                    q[2 * R - 1] = vmul(tap(2 * R), F);
                }
            }
        }
    // front j of the march: box j's values enter the x sums; y = the completed
    // stencil sums of centre j - R.  In FP64 a value's own centre term and z sum enter
    // with it, in one chain with the x sum.  In FP32 that chain's terms, up to 10 times
    // the state, cost up to 1.4 times the error of a whole solve (a batch member 8.9e-8
    // of the state after 60 steps, 6.3e-8 with the sums apart): there the z sum is
    // formed by itself, when its plane is the centre, and the centre term comes last.
    constexpr bool APART = sizeof(T) == 4;
    auto front = [&](const T *box, V (&y)[4][RW]) {
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            V zs[2 * R + RW];
#pragma unroll
            for (int k = APART ? R : 0; k < (APART ? R + RW : 2 * R + RW); ++k)
                zs[k] = O::lds(&box[((r + k) * 4 + f) * VB + NP * lane]);
#pragma unroll
            for (int w = 0; w < RW; ++w) {
                const V F = zs[R + w];
                auto &q = sx[f][w];
                y[f][w] = vfma(tap(0), F, q[0]);
#pragma unroll
                for (int k = 0; k + 1 < 2 * R; ++k)
                    q[k] = APART && k == R - 1 ? q[k + 1] : vfma(tap(k + 1), F, q[k + 1]);
                q[2 * R - 1] = vmul(tap(2 * R), F);
                if constexpr (!APART) {
                    V z = q[R - 1];
                    z = vfma(wz[0], zs[w + R - 2], z);
                    z = vfma(wz[1], zs[w + R - 1], z);
                    z = vfma(wz[2], zs[w + R + 1], z);
                    z = vfma(wz[3], zs[w + R + 2], z);
                    if (R == 3) z = vfma(kz, vadd(zs[w], zs[w + 2 * R]), z);
                    q[R - 1] = z;
                }
            }
        }
    };

    // box j has landed (false: a wait ran out, or another warp's did; looked at every 4th plane)
    auto ready = [&](int j) {
        if (mbar_wait(smem_u32(&bars[j % NS]), (unsigned)((j / NS) & 1)) && !((j & 3) == 0 && *(volatile int *)&sh.abort))
            return true;
        sh.abort = 1;
        return false;
    };
    // the first R fronts complete no centre: a loop of their own, as a condition on j
    // in one loop left it to the compiler whether to make two of it
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < R; ++j) {
        ok = ok && ready(j);
        if (!ok) break;
        const T *fb = (const T *)(smem + j % NS * S::bytes + S::box);
        if constexpr (RHS) {
#pragma unroll
            for (int f = 0; f < 4; ++f)
#pragma unroll
                for (int w = 0; w < RW; ++w) {
                    auto &q = sx[f][w];
#pragma unroll
                    for (int k = 0; k + 1 < 2 * R; ++k) q[k] = q[k + 1];
                    q[2 * R - 1] = O::lds(&fb[((r + R + w) * 4 + f) * VB + NP * lane]);
                }
        } else {
            V y[4][RW];
            front(fb, y);
        }
    }
#pragma unroll 1
    for (int j = R; ok && j < nboxes; ++j) {
        const int i = j - R, x = xs + i;  // centre plane completed by front j
        const unsigned ox = (unsigned)x * P32 + own32;  // element offset of (x, zr, v) within a field
        const int sf = j % NS, sc = i % NS;
        ok = ready(j);
        if (!ok) break;
        V y[4][RW], cen[4][RW];
        const T *fb = (const T *)(smem + sf * S::bytes + S::box);
        const unsigned char *sp = smem + sc * S::bytes;
        const T *zb = (const T *)(sp + S::box);
        if constexpr (RHS) {
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                V zs[2 * R + RW];
#pragma unroll
                for (int k = 0; k < 2 * R + RW; ++k) zs[k] = O::lds(&zb[((r + k) * 4 + f) * VB + NP * lane]);
#pragma unroll
                for (int w = 0; w < RW; ++w) {
                    const V F = O::lds(&fb[((r + R + w) * 4 + f) * VB + NP * lane]);
                    auto &q = sx[f][w];
                    V z7[2 * R + 1], x7[2 * R + 1];
#pragma unroll
                    for (int k = 0; k <= 2 * R; ++k) z7[k] = zs[w + k], x7[k] = k < 2 * R ? q[k < 2 * R ? k : 0] : F;
                    cen[f][w] = zs[R + w];
                    y[f][w] = vadd(vfma(fz, adv_diff<T, R>(z7), vmul(fx, adv_diff<T, R>(x7))),
                                   vfma(kz, ko_sum<T, R>(z7), vmul(kx, ko_sum<T, R>(x7))));
#pragma unroll
                    for (int k = 0; k + 1 < 2 * R; ++k) q[k] = q[k + 1];
                    q[2 * R - 1] = F;
                }
            }
        } else {
            front(fb, y);
        }
        if constexpr (!RHS) {
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                V zs[2 * R + RW];
#pragma unroll
                for (int k = APART ? 0 : R; k < (APART ? 2 * R + RW : R + RW); ++k)
                    zs[k] = O::lds(&zb[((r + k) * 4 + f) * VB + NP * lane]);
#pragma unroll
                for (int w = 0; w < RW; ++w) {
                    cen[f][w] = zs[R + w];
                    if constexpr (APART) {
                        V z = vmul(wz[0], zs[w + R - 2]);
                        if (R == 3) z = vfma(wz[0], zs[w + R - 2], vmul(kz, vadd(zs[w], zs[w + 2 * R])));
                        z = vfma(wz[1], zs[w + R - 1], z);
                        z = vfma(wz[2], zs[w + R + 1], z);
                        z = vfma(wz[3], zs[w + R + 2], z);
                        y[f][w] = vfma(kc, cen[f][w], vadd(z, y[f][w]));
                    }
                }
            }
        }
        V pin[4][RW];  // the pointwise input: U (S2, S3) or B (S4)
        if (CF::PU || CF::PA) {
            const T *pb = (const T *)(smem + CF::ring + i % CF::PSM * CF::pbytes);
#pragma unroll
            for (int f = 0; f < 4; ++f)
#pragma unroll
                for (int w = 0; w < RW; ++w) pin[f][w] = O::lds(&pb[((r + w) * 4 + f) * VB + NP * lane]);
        }
        V outm[4][RW], outb[4][RW];
#pragma unroll
        for (int w = 0; w < RW; ++w) {
            double m[NMOM];
            const double2 *m2 = (const double2 *)((const double *)(sp + S::mb) + (r + w) * NMOM);
#pragma unroll
            for (int k = 0; k < NMOM / 2; ++k) {
                const double2 t = m2[k];
                m[2 * k] = t.x;
                m[2 * k + 1] = t.y;
            }
            double ia[NP], ib[NP], ie[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                ia[p] = contract4(m, vx[p], vy[p], vz[p]);
                ib[p] = contract4(m + 4, vx[p], vy[p], vz[p]);
                ie[p] = contract4(m + 8, vx[p], vy[p], vz[p]);
            }
            // commutator and vacuum terms (nuosc_class.cpp:187-200, 280-287)
            const V am = vmul(mu, O::make(ia)), bm = vmul(mu, O::make(ib)), em = vmul(mu, O::make(ie));
            const V ee = cen[0][w], mm = cen[1][w], emr = cen[2][w], emi = cen[3][w];
            const V nd = vsub(mm, ee);
            const V h = vfma(emi, am, vmul(emr, bm));
            V kk[4];
            kk[0] = vfma(O::splat(2.0), h, y[0][w]);
            kk[1] = vfma(O::splat(-2.0), h, y[1][w]);
            kk[2] = vfma(nd, bm, vfma(vneg(em), emi, y[2][w]));
            kk[3] = vfma(nd, am, vfma(em, emr, y[3][w]));
            if (VAC && vac) {
                kk[0] = vfma(vneg(p2s), emi, kk[0]);
                kk[1] = vfma(p2s, emi, kk[1]);
                kk[2] = vfma(vneg(p2c), emi, kk[2]);
                kk[3] = vfma(p2c, emr, vfma(vneg(ps), nd, kk[3]));
            }
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const V c = cen[f][w];
                if (MODE == MODE_RHS) {
                    outm[f][w] = kk[f];
                } else if (MODE == MODE_S1Y) {
                    outm[f][w] = vfma(cY, kk[f], c);  // Y2
                } else if (MODE == MODE_SY) {
                    outm[f][w] = vfma(cY, kk[f], pin[f][w]);  // Y4
                } else if (MODE == MODE_S2B) {
                    const V u = pin[f][w];
                    outb[f][w] = vfma(cA, kk[f], vadd(u, c));  // B = U + Y2 + dt k2
                    outm[f][w] = vfma(cY, kk[f], u);          // Y3
                } else {
                    outm[f][w] = vthird_plus<T>(vadd(pin[f][w], c), vmul(cA, kk[f]));  // (B + Y4)/3 + dt/6 k4
                }
            }
        }
        T *dp = (MODE == MODE_S4B || MODE == MODE_RHS ? rd<SA>(a.acc_dst) : rd<SA>(a.y_dst)) + hoff + ox;
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int w = 0; w < RW; ++w) O::st_if(dp + f * fs32 + w * g.nvs, outm[f][w], put[w]);
        if (MODE == MODE_S2B) {
            T *bp = rd<SA>(a.acc_dst) + hoff + ox;
#pragma unroll
            for (int f = 0; f < 4; ++f)
#pragma unroll
                for (int w = 0; w < RW; ++w) O::st_if(bp + f * fs32 + w * g.nvs, outb[f][w], put[w]);
        }
        if (RAG)
#pragma unroll
            for (int f = 0; f < 4; ++f) sink_if(smem_u32(&sh.sink), O::bits(outm[f][0]), sink);
        // The centre use is the box's last (a right-halo box has none: its slot is
        // not filled again).  The arrive comes after the stores: they need every
        // value this plane read from shared memory, so no such read can still be
        // under way when the producer refills the slots (an arrive that only
        // follows the loads in program order may overtake them in the pipeline); the
        // values of a row that is not stored are written to sh.sink instead.
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars[NS + sc]));
        if constexpr (MODE != MODE_RHS) {
            // the half-warp that keeps a row decides whose product is rounded first
            // (its own velocity's), so the lower one keeps the row that is even in
            // the grid: RAG tiles may start at an odd one
            const bool b4 = RAG ? ((lane >> 4) ^ z0) & 1 : lane & 16;
            T ko[4][NP], kp[4][NP];  // the kept row's values: this lane's velocities, the partner's
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                T t0[NP], t1[NP];
                O::get(outm[f][0], t0);
                O::get(outm[f][1], t1);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    ko[f][p] = b4 ? t1[p] : t0[p];
                    if (!M64 || sizeof(T) == 4 || f >= 2) kp[f][p] = __shfl_xor_sync(0xffffffffu, b4 ? t0[p] : t1[p], 16);
                    else kp[f][p] = b4 ? t0[p] : t1[p];
                }
            }
            M acc[3][4];
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const T *q4[4] = {o ? &kp[0][p] : &ko[0][p], o ? &kp[1][p] : &ko[1][p], o ? &kp[2][p] : &ko[2][p],
                                      o ? &kp[3][p] : &ko[3][p]};
                    M dd = M(*q4[0]) - M(*q4[1]);
                    if (M64 && sizeof(T) == 8 && o) dd = __shfl_xor_sync(0xffffffffu, dd, 16);
                    const M d[3] = {M(*q4[2]), M(*q4[3]), dd};
#pragma unroll
                    for (int jw = 0; jw < 4; ++jw) {
                        const M w = o ? wp[p][jw] : wo[p][jw];
#pragma unroll
                        for (int c = 0; c < 3; ++c) acc[c][jw] = o == 0 && p == 0 ? w * d[c] : fma(w, d[c], acc[c][jw]);
                    }
                }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                acc[c][0] += __shfl_xor_sync(0xffffffffu, acc[c][2], 8);
                acc[c][1] += __shfl_xor_sync(0xffffffffu, acc[c][3], 8);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c][0] += __shfl_xor_sync(0xffffffffu, acc[c][1], 4);
            const bool b1 = (lane >> 1) & 1, b0 = lane & 1;
            M k0 = b1 ? acc[2][0] : acc[0][0];
            k0 += __shfl_xor_sync(0xffffffffu, b1 ? acc[0][0] : acc[2][0], 2);
            const M k1 = acc[1][0] + __shfl_xor_sync(0xffffffffu, acc[1][0], 2);
            M kk = (!b1 && b0) ? k1 : k0;
            kk += __shfl_xor_sync(0xffffffffu, (b1 || b0) ? k0 : k1, 1);
            if (!(b1 && b0) && (b4 || keep0)) {  // lane holds moment 4c + wq of its kept row
                const int c = b1 ? 2 : (int)b0;
                const double v = (double)kk;
                const unsigned cell = (unsigned)x * (unsigned)rd<SA>(a.g.nz) + (unsigned)(zr + (b4 ? 1 : 0));
                rd<SA>(a.mom_part)[((cell * (unsigned)nvb + (unsigned)vb) * 2u + (unsigned)half) * NMOM + 4 * c + wq] =
                    (half || c == 1) ? v : -v;
            }
        }
    }
    __syncthreads();
    const bool aborted = sh.abort != 0;
    if constexpr (MODE == MODE_RHS) {  // a caller without a status word sees an incomplete tile as NaN
        if (aborted)
            for (int x = xs; x < t.xe; ++x)
#pragma unroll
                for (int f = 0; f < 4; ++f)
#pragma unroll
                    for (int w = 0; w < RW; ++w)
                        O::st_if(a.acc_dst + hoff + f * fs + (long long)x * P + own + w * g.nvs, O::splat(nan("")), put[w]);
    }
    return aborted;
}

// The tail velocities of a lone solve's launch: block column nvbm, if launched,
// runs them (first velocity v0, twp lanes per (cell, half)), in launches of up to
// kTailWaves waves: its CTAs fill the last wave and spare a kernel (us per step:
// 64x64x162 FP64 208 -> 167, 128x128x162 566 -> 497, 75x150x642 FP32 773 -> 733,
// 256x256x642 FP32, 5 waves, 4290 -> 3950).  Beyond that a tail CTA, one of few
// threads per SM and every load a miss, costs more than the kernel that fills the
// SMs with threads (512x256x642 FP64, 18 waves: 14.7 ms against 13.8).
constexpr int kTailWaves = 6;
struct StageTail {
    int nvbm, v0, twp;
    bool early;  // one wave: let the next kernel be launched from the start
};

// grid (velocity blocks run by this kernel + a tail column where there is a tail,
// z tiles, 2 x x-segments); nvb: velocity blocks of the moment partials
template <typename T, int R, int MODE, int TZ, bool VAC, bool M64, bool RAG>
__global__ void __launch_bounds__(threads_of(TZ), tma_ctas_per_sm<T, TZ>())
    k_xtma(const __grid_constant__ TmaMaps maps, const StageArgs<T> a, const ZTiles zt, int LX, int nvb,
           const StageTail f) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ MarchShared sh;
    constexpr int NC = 32 * (TZ / RW);  // consumer threads
    if (f.early) grid_launch_dependents();
    const int xs = (blockIdx.z >> 1) * LX;
    const Tile t{zt.row(blockIdx.y), (int)blockIdx.x, nvb, xs, min(xs + LX, a.g.nx),
                 (int)blockIdx.z & 1, RAG ? zt.shared_rows(blockIdx.y, TZ) : 0};
    if (blockIdx.x == f.nvbm) {
        // the tail velocities of the tile's cells: lane l of (plane, row)
        if (f.early) grid_wait();
        const int n = (t.xe - t.xs) * TZ * f.twp, step = threads_of(TZ);
        for (int o = threadIdx.x; o - (int)(threadIdx.x & 31) < n; o += step) {
            const int l = o & (f.twp - 1), c = o / f.twp;
            const long long cell = (long long)(xs + c / TZ) * a.g.nz + t.z0 + c % TZ;
            const int v = f.v0 + l;
            const bool own = o < n && (!RAG || c % TZ >= t.skip);
            tail_point<T, R == 3, MODE>(a, cell, t.half, v, own && v < a.g.nvs, own, f.twp, nvb, l);
        }
    } else if (threadIdx.x >= NC) {
        setmaxnreg_dec<RegSplit<TZ>::producer>();
        xtma_produce<T, R, MODE, TZ, false>(maps, a, t, smem, sh, f.early);
    } else {
        setmaxnreg_inc<RegSplit<TZ>::consumer>();
        xtma_consume<T, R, MODE, TZ, VAC, false, M64, RAG>(a, t, smem, sh, f.early);
    }
}

// One instance's stage in a batched launch: its tensor maps (over the stage's
// input register), stage arguments and tile counts.  Lives in device memory;
// the TMA reads the maps from there.
template <typename T>
struct __align__(64) BatchItem {
    TmaMaps maps;
    StageArgs<T> a;
    int ntz, nvb, lx, nseg;
    int nvbm;  // velocity blocks run by the march (nvb - 1 when a tail kernel runs the last)
};

// Persistent batched stage kernel.  The tiles of all instances form one list
// (instances in the order of the table -- largest first --, each instance's
// tiles in the single-instance kernel's CTA order: velocity block fastest,
// then z rows, then flavour half and x segment) that the CTAs take from an
// atomic cursor, so the tiles in flight stay a narrow window of the list, as
// in a hardware-scheduled grid (neighbouring tiles share halo rows in L2 and
// DRAM pages).  Tile k of instance i is the tile the single-instance kernel
// runs as its CTA k, so each instance's result is the same bits as its own
// launch.  The tile's StageArgs are copied to shared memory and re-read there at each use
// (the single-instance kernel reads them from the constant bank), which keeps
// them out of the register file that the march's x-queue fills.  VAC compiles
// the vacuum term in (for batches with any pmo != 0); it is then switched per
// instance at run time.
template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
__global__ void __launch_bounds__(threads_of(TZ), tma_ctas_per_sm<T, TZ>())
    k_xtma_batch(const BatchItem<T> *items, const long long *__restrict__ starts, int ninst, long long nitems,
                 unsigned long long *counter, const int *__restrict__ halt) {
    constexpr int NW = (int)(sizeof(StageArgs<T>) / 8);
    constexpr int NC = 32 * (TZ / RW);  // consumer threads
    static_assert(sizeof(StageArgs<T>) % 8 == 0 && NW <= 128, "StageArgs copy: one 8-byte word per producer thread");
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ MarchShared sh;
    __shared__ __align__(16) StageArgs<T> s_a;
    __shared__ const TmaMaps *s_mp;
    __shared__ Tile s_t;
    __shared__ int s_inst;  // instance (-1: no tiles left, -2: a stopped instance's tile)
    if (threadIdx.x >= NC) {
        setmaxnreg_dec<RegSplit<TZ>::producer>();
        for (;;) {
            __syncthreads();  // every thread is done with the previous tile's arguments
            if (threadIdx.x == NC) {
                const long long it = (long long)atomicAdd(counter, 1ull);
                s_inst = -1;
                if (it < nitems) {
                    int lo = 0, hi = ninst - 1;  // last instance whose first tile is <= it
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (starts[mid] <= it) lo = mid;
                        else hi = mid - 1;
                    }
                    const BatchItem<T> &e = items[lo];
                    int loc = (int)(it - starts[lo]);  // ((seg * 2 + half) * ntz + zt) * nvbm + vb
                    s_inst = (halt && halt[lo]) ? -2 : lo;
                    s_t.vb = loc % e.nvbm;
                    loc /= e.nvbm;
                    s_t.z0 = loc % e.ntz * TZ;
                    loc /= e.ntz;
                    s_t.half = loc & 1;
                    s_t.xs = (loc >> 1) * e.lx;
                    s_t.xe = min(s_t.xs + e.lx, e.a.g.nx);
                    s_t.nvb = e.nvb;
                    s_t.skip = 0;
                    s_mp = &e.maps;
                    // this thread issues every TMA load of the tile; the maps were written
                    // through the generic proxy (a host copy when the work-list was built)
                    tensormap_acquire(&e.maps.zr);
                    tensormap_acquire(&e.maps.tzr);
                    tensormap_acquire(&e.maps.r);
                    if (MarchCfg<T, R, MODE, TZ>::PU) tensormap_acquire(&e.maps.pu);
                    if (MarchCfg<T, R, MODE, TZ>::PA) tensormap_acquire(&e.maps.pa);
                }
            }
            __syncthreads();
            const int lo = s_inst;
            if (lo == -1) break;
            if (lo == -2) continue;  // every thread: the loop's first barrier comes next
            const int w = threadIdx.x - NC;
            if (w < NW) reinterpret_cast<long long *>(&s_a)[w] = reinterpret_cast<const long long *>(&items[lo].a)[w];
            __syncthreads();  // s_a is complete
            if (xtma_produce<T, R, MODE, TZ, true>(*s_mp, s_a, s_t, smem, sh)) break;
        }
    } else {
        setmaxnreg_inc<RegSplit<TZ>::consumer>();
        for (;;) {
            __syncthreads();
            __syncthreads();
            const int lo = s_inst;
            if (lo == -1) break;
            if (lo == -2) continue;
            __syncthreads();
            if (xtma_consume<T, R, MODE, TZ, VAC, true, M64, false>(s_a, s_t, smem, sh)) break;
        }
    }
}

// Self-test of the bounded wait that the march kernels use: one warp waits on
// an mbarrier that nothing completes (initialised for two arrivals, given
// one).  The wait gives up after `spins` polls; the kernel then records the
// timeout in the status word, as a march does, invalidates the barrier and
// returns.  Nothing else is touched, so the context stays usable.
#if NUOSC_PART == 0
__global__ void k_wait_selftest(int *status, unsigned spins) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 2u);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        mbar_arrive(smem_u32(&bar));  // one arrival of two: phase 0 never completes
        if (!mbar_wait(smem_u32(&bar), 0u, spins)) atomicExch(status, NUOSC_TIMEOUT_CODE);
        mbar_inval(smem_u32(&bar));
    }
}

cudaError_t launch_wait_selftest(int *status, unsigned spins, cudaStream_t s) {
    k_wait_selftest<<<1, 32, 0, s>>>(status, spins);
    return cudaGetLastError();
}
#endif

// ------------------------------------------------------------------ host side
namespace {

bool tma_mode(int mode) { return mode == MODE_S1Y || mode == MODE_S2B || mode == MODE_SY || mode == MODE_S4B; }

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// (looked up by the first caller; others wait for it)
EncodeFn encode_fn() {
    static const EncodeFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        return ok ? (EncodeFn)p : nullptr;
    }();
    return fn;
}

// 4D view of one register: (v, field, z, x) with box {VB, 4, rows, 1}
template <typename T>
bool make_map(CUtensorMap *m, const T *base, const Geom &g, int rows) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)g.nvs, 8, (cuuint64_t)g.nz, (cuuint64_t)g.nx};
    const cuuint64_t strides[3] = {(cuuint64_t)g.fs * sizeof(T), (cuuint64_t)g.nvs * sizeof(T),
                                   (cuuint64_t)g.nz * g.nvs * sizeof(T)};
    const cuuint32_t box[4] = {(cuuint32_t)vblock<T>(), 4, (cuuint32_t)rows, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUtensorMapDataType dt = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    return fn(m, dt, 4, (void *)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// velocity blocks the march runs: all of them, or all but the tail block
template <typename T>
int march_vblocks(const Geom &g) {
    const int v0 = xtma_tail_v0<T>(g);
    return v0 == g.nvs ? xtma_num_vblocks<T>(g) : v0 / vblock<T>();
}

}  // namespace

template <typename T>
int xtma_waves(const Geom &g, XTile t, int sms) {
    const int cols = march_vblocks<T>(g) + (xtma_tail_v0<T>(g) < g.nvs ? 1 : 0);
    const int lx = t.lx < g.nx ? t.lx : g.nx;
    const long long ctas = 2ll * cols * ((g.nz + t.tz - 1) / t.tz) * ((g.nx + lx - 1) / lx);
    const long long slots = (long long)sms * (t.tz == 16 ? 1 : 2);
    return (int)((ctas + slots - 1) / slots);
}

namespace {

// the stencil input's boxes, and the TZ-row boxes of the stage's pointwise
// inputs (U, A) where the stage has them (zeroed maps otherwise)
template <typename T>
bool make_maps(TmaMaps *m, const StageArgs<T> &a, int tz, int r) {
    memset((void *)&m->pu, 0, sizeof m->pu);
    memset((void *)&m->pa, 0, sizeof m->pa);
    memset((void *)&m->hzr, 0, 3 * sizeof m->hzr);
    // a slab's halo buffer as a register of 2R planes
    Geom h = a.g;
    h.nx = 2 * r;
    h.fs = (long long)h.nx * h.nz * h.nvs;
    return make_map<T>(&m->zr, a.in, a.g, tz + 2 * r) && make_map<T>(&m->tzr, a.in, a.g, tz + r) &&
           make_map<T>(&m->r, a.in, a.g, r) &&
           (!a.u || make_map<T>(&m->pu, a.u, a.g, tz)) && (!a.acc_src || make_map<T>(&m->pa, a.acc_src, a.g, tz)) &&
           (!a.halo || (make_map<T>(&m->hzr, a.halo, h, tz + 2 * r) && make_map<T>(&m->htzr, a.halo, h, tz + r) &&
                        make_map<T>(&m->hr, a.halo, h, r)));
}

template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
cudaError_t launch_t(const StageArgs<T> &a, XTile t, cudaStream_t s) {
    using CF = MarchCfg<T, R, MODE, TZ>;
    static_assert(tma_ctas_per_sm<T, TZ>() * (CF::smem + sizeof(MarchShared) + sizeof(StageArgs<T>) + 64 + 1024) <= 228 * 1024,
                  "ring exceeds shared memory");
    TmaMaps maps;
    if (!make_maps<T>(&maps, a, TZ, R)) return cudaErrorInvalidValue;
    const size_t smem = CF::smem;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const ZTiles zt(a.g.nz, TZ);
    const auto kern = a.g.nz % TZ ? k_xtma<T, R, MODE, TZ, VAC, M64, true> : k_xtma<T, R, MODE, TZ, VAC, M64, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (t.lx > a.g.nx) t.lx = a.g.nx;  // (one segment)
    const int nseg = (a.g.nx + t.lx - 1) / t.lx;
    const int nvb = xtma_num_vblocks<T>(a.g), nvbm = march_vblocks<T>(a.g), v0 = xtma_tail_v0<T>(a.g);
    const bool tail = v0 < a.g.nvs, column = tail && xtma_waves<T>(a.g, t, sms) <= kTailWaves;
    // velocity blocks fastest: the CTAs resident at once read whole velocity
    // rows of a few z rows (DRAM page locality) rather than one block of many rows
    dim3 grid(nvbm + column, zt.n, nseg * 2);
    const StageTail f{nvbm, v0, tail_lanes(a.g.nvs - v0), t.early};
    e = launch_dependent(t.early, kern, grid, threads_of(TZ), smem, s, maps, a, zt, t.lx, nvb, f);
    if (e == cudaSuccess && tail && !column) e = launch_stage_tail<T>(a, MODE, R == 3, v0, nvb, s);
    if (t.launched) *t.launched += tail && !column ? 2 : 1;
    return e;
}

}  // namespace

// The launchers below are instantiated in parts 1 to 10.
template <typename T, int TZ>
cudaError_t launch_rhs_t(const StageArgs<T> &a, bool ko6, XTile t, cudaStream_t s) {
    if (a.c.pmo != 0.0)
        return ko6 ? launch_t<T, 3, MODE_RHS, TZ, true, true>(a, t, s) : launch_t<T, 2, MODE_RHS, TZ, true, true>(a, t, s);
    return ko6 ? launch_t<T, 3, MODE_RHS, TZ, false, true>(a, t, s) : launch_t<T, 2, MODE_RHS, TZ, false, true>(a, t, s);
}

namespace {

template <typename T, int R, int TZ, bool VAC, bool M64>
cudaError_t launch_tm(const StageArgs<T> &a, int mode, XTile t, cudaStream_t s) {
    switch (mode) {
    case MODE_S1Y: return launch_t<T, R, MODE_S1Y, TZ, VAC, M64>(a, t, s);
    case MODE_S2B: return launch_t<T, R, MODE_S2B, TZ, VAC, M64>(a, t, s);
    case MODE_SY: return launch_t<T, R, MODE_SY, TZ, VAC, M64>(a, t, s);
    case MODE_S4B: return launch_t<T, R, MODE_S4B, TZ, VAC, M64>(a, t, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

template <typename T, int R, int TZ, bool M64>
cudaError_t launch_tv(const StageArgs<T> &a, int mode, XTile t, cudaStream_t s) {
    return a.c.pmo != 0.0 ? launch_tm<T, R, TZ, true, M64>(a, mode, t, s)
                          : launch_tm<T, R, TZ, false, M64>(a, mode, t, s);
}

namespace {

// ---- batched launch: one persistent grid per stage over many instances
template <typename T, int R, int MODE, int TZ>
constexpr size_t batch_smem() {
    return MarchCfg<T, R, MODE, TZ>::smem;
}

template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
int batch_grid_t(int device) {
    const size_t smem = batch_smem<T, R, MODE, TZ>();
    auto kern = k_xtma_batch<T, R, MODE, TZ, VAC, M64>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads_of(TZ), smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || per_sm < 1)
        return -1;
    return per_sm * sms;
}

template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
cudaError_t batch_launch_t(const void *items, const long long *starts, int n, long long ntiles,
                           unsigned long long *counter, const int *halt, int grid, cudaStream_t s) {
    k_xtma_batch<T, R, MODE, TZ, VAC, M64><<<grid, threads_of(TZ), batch_smem<T, R, MODE, TZ>(), s>>>(
        (const BatchItem<T> *)items, starts, n, ntiles, counter, halt);
    return cudaGetLastError();
}

// dispatch of (mode, ko6, tz, vac) onto the template instances of F
template <typename T, bool M64, template <typename, int, int, int, bool, bool> class F, typename... Args>
auto batch_dispatch(int mode, bool ko6, int tz, bool vac, Args... args) {
#define NUOSC_BATCH_V(R, M, Z) \
    (vac ? F<T, R, M, Z, true, M64>::run(args...) : F<T, R, M, Z, false, M64>::run(args...))
#define NUOSC_BATCH_TZ(R, M) (tz == 16 ? NUOSC_BATCH_V(R, M, 16) : NUOSC_BATCH_V(R, M, 8))
#define NUOSC_BATCH_MODE(R)                                                                                   \
    (mode == MODE_S1Y   ? NUOSC_BATCH_TZ(R, MODE_S1Y)                                                         \
     : mode == MODE_S2B ? NUOSC_BATCH_TZ(R, MODE_S2B)                                                         \
     : mode == MODE_SY  ? NUOSC_BATCH_TZ(R, MODE_SY)                                                          \
                        : NUOSC_BATCH_TZ(R, MODE_S4B))
    return ko6 ? NUOSC_BATCH_MODE(3) : NUOSC_BATCH_MODE(2);
#undef NUOSC_BATCH_MODE
#undef NUOSC_BATCH_TZ
#undef NUOSC_BATCH_V
}

template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
struct BatchGrid {
    static int run(int device) { return batch_grid_t<T, R, MODE, TZ, VAC, M64>(device); }
};
template <typename T, int R, int MODE, int TZ, bool VAC, bool M64>
struct BatchLaunch {
    static cudaError_t run(const void *items, const long long *starts, int n, long long ntiles,
                           unsigned long long *counter, const int *halt, int grid, cudaStream_t s) {
        return batch_launch_t<T, R, MODE, TZ, VAC, M64>(items, starts, n, ntiles, counter, halt, grid, s);
    }
};

}  // namespace

template <typename T, bool M64>
int batch_grid_m(int mode, bool ko6, int tz, bool vac, int device) {
    return batch_dispatch<T, M64, BatchGrid>(mode, ko6, tz, vac, device);
}

template <typename T, bool M64>
cudaError_t batch_launch_m(const void *items, const long long *starts, int n, long long ntiles,
                           unsigned long long *counter, const int *halt, int mode, bool ko6, int tz, bool vac, int grid,
                           cudaStream_t s) {
    return batch_dispatch<T, M64, BatchLaunch>(mode, ko6, tz, vac, items, starts, n, ntiles, counter, halt, grid, s);
}

#define NUOSC_STAGES(X, T, R, M64)                                                          \
    X template cudaError_t launch_tv<T, R, 16, M64>(const StageArgs<T> &, int, XTile, cudaStream_t); \
    X template cudaError_t launch_tv<T, R, 8, M64>(const StageArgs<T> &, int, XTile, cudaStream_t);
#define NUOSC_RHS(X, T)                                                                   \
    X template cudaError_t launch_rhs_t<T, 16>(const StageArgs<T> &, bool, XTile, cudaStream_t);    \
    X template cudaError_t launch_rhs_t<T, 8>(const StageArgs<T> &, bool, XTile, cudaStream_t);
#define NUOSC_BATCH(X, T, M64)                                                              \
    X template int batch_grid_m<T, M64>(int, bool, int, bool, int);                                   \
    X template cudaError_t batch_launch_m<T, M64>(const void *, const long long *, int, long long,    \
                                                  unsigned long long *, const int *, int, bool, int, \
                                                  bool, int, cudaStream_t);
#if NUOSC_PART == 1
NUOSC_STAGES(, double, 3, true)
#elif NUOSC_PART == 2
NUOSC_STAGES(, double, 2, true)
#elif NUOSC_PART == 3
NUOSC_STAGES(, float, 3, true)
#elif NUOSC_PART == 4
NUOSC_STAGES(, float, 2, true)
#elif NUOSC_PART == 5
NUOSC_STAGES(, float, 3, false)
#elif NUOSC_PART == 6
NUOSC_STAGES(, float, 2, false)
#elif NUOSC_PART == 7
NUOSC_RHS(, double)
NUOSC_RHS(, float)
#elif NUOSC_PART == 8
NUOSC_BATCH(, double, true)
#elif NUOSC_PART == 9
NUOSC_BATCH(, float, true)
#elif NUOSC_PART == 10
NUOSC_BATCH(, float, false)
#else  // part 0: the host side, to the end of the file
NUOSC_STAGES(extern, double, 3, true)
NUOSC_STAGES(extern, double, 2, true)
NUOSC_STAGES(extern, float, 3, true)
NUOSC_STAGES(extern, float, 2, true)
NUOSC_STAGES(extern, float, 3, false)
NUOSC_STAGES(extern, float, 2, false)
NUOSC_RHS(extern, double)
NUOSC_RHS(extern, float)
NUOSC_BATCH(extern, double, true)
NUOSC_BATCH(extern, float, true)
NUOSC_BATCH(extern, float, false)

namespace {

// moment partials summed in FP64 (always for FP64 state; for FP32 state per
// the tile's msum) or in float within a velocity block
template <typename T, int R, int TZ>
cudaError_t launch_tms(const StageArgs<T> &a, int mode, XTile t, cudaStream_t s) {
    if constexpr (sizeof(T) == 8) return launch_tv<T, R, TZ, true>(a, mode, t, s);
    else return t.msum ? launch_tv<T, R, TZ, true>(a, mode, t, s) : launch_tv<T, R, TZ, false>(a, mode, t, s);
}

}  // namespace

template <typename T>
bool xtma_fits(const Geom &g, XTile t) {
    // nz >= tz + 6: the widest box (tz + 2R rows, R <= 3) fits in the z extent;
    // 3 fs < 2^32: the march's per-plane offsets within a flavour half are
    // 32-bit (registers of up to 91 GB in FP64, 45 GB in FP32: every state
    // whose four registers fit a B200)
    return (t.tz == 8 || t.tz == 16) && g.nz >= t.tz + 6 && g.nx >= 4 &&
           g.nvs % vpt<T>() == 0 && 3 * g.fs < (1ll << 32) && encode_fn() != nullptr;
}

template <typename T>
bool xtma_supported(const Geom &g, XTile t) {
    return g.nz % t.tz == 0 && xtma_fits<T>(g, t);
}

bool xtma_grid_ok(const Geom &g, XTile t) {
    return (g.nz + t.tz - 1) / t.tz <= 65535 && (g.nx + t.lx - 1) / t.lx <= 32767;
}

// x planes per CTA.  A segment costs its planes plus about 10 more (the launch of
// the CTA, the constants, R planes left of it and R right of it), and a launch
// costs whole waves of CTAs, so the number of segments minimises waves x (lx +
// 10); among segment counts within 2 % the fewest.  Measured (us per FP64 step, the choice in
// brackets): 32x32x42 [2] 32, 4: 39, 16: 87, 32: 145; 64x64x162 [22] 138, 16: 196,
// 32: 170, 64: 289; 128x128x162 [43] 483, 32: 522, 64: 608; 100x90x162 [50] 271,
// 34: 351, 100: 468; 128x128x642 [64] 1825, 32: 1712, 128: 2037.
//
// Where many whole waves make all counts cost the same, two limits stand.  CTAs
// drift apart along a long march, and neighbouring velocity blocks then no longer
// read a DRAM page together: at most 192 planes (ms per step: 256x256x642 FP64 lx
// 256: 7.5, 128: 7.3, 86: 7.1; 1024x256x642 FP64 lx 1024: 32.6, 512: 29.1, 64 to
// 256: 28.7 to 29.0).  And a segment spans at most 2 GiB of a register, as the
// pages in use at a time grow with it: 1024x1024x642 FP64 (172 GB) lx 1024: 128,
// 256: 122, 128: 122, 64: 117.5, 48: 116.3 (the choice), 32: 118, 24: 120.6; FP32
// lx 1024: 64.8, 94 to 96 (the choice): 63.2, 48: 64.1; 512x512x642 FP32 lx 512:
// 16.6, 171: 15.1.  (128x1024x642 FP64 pays 1 %: lx 128 14.15, 43 14.35.)
template <typename T>
int xtma_lx(const Geom &g, int tz, int sms) {
    const long long slots = (long long)sms * (tz == 16 ? 1 : 2);
    const int cols = march_vblocks<T>(g) + (xtma_tail_v0<T>(g) < g.nvs ? 1 : 0);  // (the tail column too)
    const long long per = (long long)((g.nz + tz - 1) / tz) * cols * 2;  // CTAs per segment
    const double span = (double)g.nx * g.nz * g.nvs * 8 * sizeof(T) / (1ll << 31);  // 2 GiB pieces of a register
    int first = (g.nx + 191) / 192, best = 1;
    if (span > first) first = span < g.nx ? (int)ceil(span) : g.nx;
    double cost = -1.0;
    for (int n = first; n <= g.nx; ++n) {
        // n or more segments (at least n / 2 once rounded) cannot cost less than this
        if (cost >= 0.0 && (double)per * (n / 2) / (double)slots * 11.0 > cost) break;
        const int lx = (g.nx + n - 1) / n, nseg = (g.nx + lx - 1) / lx;
        const double c = (double)((per * nseg + slots - 1) / slots) * (lx + 10);
        if (cost < 0.0 || c < 0.98 * cost) {
            cost = c;
            best = lx;
        }
    }
    return best;
}

template <typename T>
size_t xtma_batch_item_bytes() {
    return sizeof(BatchItem<T>);
}

template <typename T>
long long xtma_batch_fill(void *item, const StageArgs<T> &a, bool ko6, int tz, int lx) {
    if (!xtma_supported<T>(a.g, XTile{tz, lx, vblock<T>()}) || lx < 1 || !a.mom_part) return -1;
    BatchItem<T> e;
    memset((void *)&e, 0, sizeof e);
    if (!make_maps<T>(&e.maps, a, tz, ko6 ? 3 : 2)) return -1;
    e.a = a;
    e.ntz = a.g.nz / tz;
    e.nvb = xtma_num_vblocks<T>(a.g);
    e.nvbm = march_vblocks<T>(a.g);
    e.lx = lx;
    e.nseg = (a.g.nx + lx - 1) / lx;
    memcpy(item, (const void *)&e, sizeof e);
    return (long long)e.ntz * e.nvbm * 2 * e.nseg;
}

template <typename T>
int xtma_batch_grid(int mode, bool ko6, int tz, bool vac, bool m64, int device) {
    if ((tz != 8 && tz != 16) || !tma_mode(mode)) return -1;
    if constexpr (sizeof(T) == 8) return batch_grid_m<T, true>(mode, ko6, tz, vac, device);
    else
        return m64 ? batch_grid_m<T, true>(mode, ko6, tz, vac, device)
                   : batch_grid_m<T, false>(mode, ko6, tz, vac, device);
}

template <typename T>
cudaError_t launch_stage_xtma_batch(const void *items, const long long *starts, int n, long long ntiles,
                                    unsigned long long *counter, const int *halt, int mode, bool ko6, int tz,
                                    bool vac, bool m64, int grid, cudaStream_t s) {
    if ((tz != 8 && tz != 16) || !tma_mode(mode) || n < 1 || grid < 1)
        return cudaErrorInvalidValue;
    if constexpr (sizeof(T) == 8)
        return batch_launch_m<T, true>(items, starts, n, ntiles, counter, halt, mode, ko6, tz, vac, grid, s);
    else
        return m64 ? batch_launch_m<T, true>(items, starts, n, ntiles, counter, halt, mode, ko6, tz, vac, grid, s)
                   : batch_launch_m<T, false>(items, starts, n, ntiles, counter, halt, mode, ko6, tz, vac, grid, s);
}

template <typename T>
int xtma_num_vblocks(const Geom &g) {
    return (g.nvs + vblock<T>() - 1) / vblock<T>();
}

template <typename T>
bool xtma_all_tail(const Geom &g) {
    return march_vblocks<T>(g) < 1;
}

template <typename T>
int xtma_tail_v0(const Geom &g) {
    const int nvb = xtma_num_vblocks<T>(g), last = (nvb - 1) * vblock<T>();
    return 4 * (g.nvs - last) <= vblock<T>() ? last : g.nvs;
}

template <typename T>
cudaError_t launch_stage_xtma(const StageArgs<T> &a, int mode, bool ko6, XTile t, bool early, long long *launched,
                              cudaStream_t s) {
    t.early = early;
    t.launched = launched;
    if (!a.mom_part || !xtma_fits<T>(a.g, t)) return cudaErrorInvalidValue;
    if (t.tz == 16) return ko6 ? launch_tms<T, 3, 16>(a, mode, t, s) : launch_tms<T, 2, 16>(a, mode, t, s);
    return ko6 ? launch_tms<T, 3, 8>(a, mode, t, s) : launch_tms<T, 2, 8>(a, mode, t, s);
}

// calRHS on the march: 2 state passes (plus the moment pass before it) instead
// of the direct kernel's 13 or 9 loads per value from L2.  Whole call, moment
// pass included: 128x128x642 FP64, KO6 1152 -> 474 us (140 of them the moment
// pass); 250x130x162 FP32, KO4 301 -> 157 us.  The direct kernel stays for nz <
// 14, for buffers without 16-byte rows and where rhs_xtma_pays says so.
template <typename T>
XTile rhs_tile(const Geom &g) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int tz = g.nz >= 22 ? 16 : 8;
    return XTile{tz, xtma_lx<T>(g, tz, sms), vblock<T>()};
}

template <typename T>
bool rhs_xtma_fits(const Geom &g, const void *in, const void *out) {
    // the tensor maps and the vector accesses need 16-byte aligned rows; a
    // caller's own buffers may have neither
    return g.nvs * sizeof(T) % 16 == 0 && (uintptr_t)in % 16 == 0 && (uintptr_t)out % 16 == 0 &&
           xtma_fits<T>(g, XTile{g.nz >= 22 ? 16 : 8, 0, vblock<T>()}) &&
           ((g.nx <= 32767 && g.nz <= 65535) || xtma_grid_ok(g, rhs_tile<T>(g)));
}

// The smallest calls are one latency chain (launch, constants, first box): the
// direct kernel's is shorter with the 4th difference, its 9 loads per value in
// flight at once.  Below 40,000 values a field, whole call, direct and march:
// 16x16x42 FP32 9.1 and 10.5 us, 24x16x92 9.3 and 10.5, FP64 24x16x42 10.1 and 10.4;
// 16x16x162 (41,472) FP32 12.3 and 11.1; 6th difference 16x16x42 10.3 and 10.5,
// 24x16x92 FP64 12.3 and 10.5.
bool rhs_xtma_pays(const Geom &g, bool ko6) { return ko6 || g.fs >= 40000; }

template <typename T>
cudaError_t launch_rhs_xtma(const StageArgs<T> &a, bool ko6, long long *launched, cudaStream_t s) {
    XTile t = rhs_tile<T>(a.g);
    t.launched = launched;
    if (xtma_all_tail<T>(a.g)) {
        if (launched) ++*launched;
        return launch_stage_tail<T>(a, MODE_RHS, ko6, 0, 1, s);
    }
    return t.tz == 16 ? launch_rhs_t<T, 16>(a, ko6, t, s) : launch_rhs_t<T, 8>(a, ko6, t, s);
}

template bool rhs_xtma_fits<double>(const Geom &, const void *, const void *);
template bool rhs_xtma_fits<float>(const Geom &, const void *, const void *);
template cudaError_t launch_rhs_xtma<double>(const StageArgs<double> &, bool, long long *, cudaStream_t);
template cudaError_t launch_rhs_xtma<float>(const StageArgs<float> &, bool, long long *, cudaStream_t);
template bool xtma_supported<double>(const Geom &, XTile);
template bool xtma_fits<double>(const Geom &, XTile);
template int xtma_lx<double>(const Geom &, int, int);
template int xtma_waves<double>(const Geom &, XTile, int);
template int xtma_waves<float>(const Geom &, XTile, int);
template int xtma_lx<float>(const Geom &, int, int);
template bool xtma_fits<float>(const Geom &, XTile);
template bool xtma_supported<float>(const Geom &, XTile);
template int xtma_num_vblocks<double>(const Geom &);
template int xtma_num_vblocks<float>(const Geom &);
template int xtma_tail_v0<double>(const Geom &);
template bool xtma_all_tail<double>(const Geom &);
template bool xtma_all_tail<float>(const Geom &);
template int xtma_tail_v0<float>(const Geom &);
template cudaError_t launch_stage_xtma<double>(const StageArgs<double> &, int, bool, XTile, bool, long long *,
                                               cudaStream_t);
template cudaError_t launch_stage_xtma<float>(const StageArgs<float> &, int, bool, XTile, bool, long long *,
                                              cudaStream_t);
template size_t xtma_batch_item_bytes<double>();
template size_t xtma_batch_item_bytes<float>();
template long long xtma_batch_fill<double>(void *, const StageArgs<double> &, bool, int, int);
template long long xtma_batch_fill<float>(void *, const StageArgs<float> &, bool, int, int);
template int xtma_batch_grid<double>(int, bool, int, bool, bool, int);
template int xtma_batch_grid<float>(int, bool, int, bool, bool, int);
template cudaError_t launch_stage_xtma_batch<double>(const void *, const long long *, int, long long,
                                                     unsigned long long *, const int *, int, bool, int, bool, bool,
                                                     int, cudaStream_t);
template cudaError_t launch_stage_xtma_batch<float>(const void *, const long long *, int, long long,
                                                    unsigned long long *, const int *, int, bool, int, bool, bool,
                                                    int, cudaStream_t);

#endif  // NUOSC_PART

}  // namespace nuosc
