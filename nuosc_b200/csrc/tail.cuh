// tail.cuh -- one point of the last, nearly empty velocity block of a stage (or of
// calRHS): shared by the march kernel's tail CTAs (xtma.cu) and the tail kernels
// (tail.cu).
#pragma once
#include "internal.cuh"
#include "physics.cuh"

namespace nuosc {

// *p; issued in program order, so that all of a field's loads are in flight at once
__device__ __forceinline__ double ld_now(const double *p) {
    double r;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ float ld_now(const float *p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p));
    return r;
}

// One (cell, velocity, flavour half) of the tail; every lane of the warp
// calls it (the moment reduction shuffles across the twp lanes of a cell and
// half), act says whether the lane holds a real point.  twp: lanes per
// (cell, half) (power of 2); put: the lane's (cell, half) is one whose partial
// this call writes.  The commutator couples the four fields of a
// half only to each other once the moments are known, so a half is a
// complete unit of work.
template <typename T, bool KO6, int MODE>
__device__ __forceinline__ void tail_point(const StageArgs<T> &a, const long long cell, const int half, const int v,
                                           const bool act, const bool put, const int twp, const int nvb,
                                           const int lane_in_cell) {
    const Geom g = a.g;
    double mom[NMOM];
#pragma unroll
    for (int k = 0; k < NMOM; ++k) mom[k] = 0.0;
    if (act) {
        const int i = (int)((unsigned)cell / (unsigned)g.nz), j = (int)((unsigned)cell - (unsigned)i * (unsigned)g.nz);
        constexpr int R = KO6 ? 3 : 2;
        const long long hoff = (long long)half * 4 * g.fs;
        const long long P = (long long)g.nz * g.nvs, col = (long long)j * g.nvs + v, ctr = (long long)i * P + col;
        const T *in = a.in + hoff;
        const T *halo = a.halo ? a.halo + (long long)half * 8 * R * P : nullptr;
        // neighbours: field-0 pointers of this half and the x ones' field stride --
        // inside the register (periodic), or a slab's halo buffer
        const T *zp[7], *xp[7];
        long long xfs[7];
#pragma unroll
        for (int k = -3; k <= 3; ++k) {
            const int kk = (k < -R || k > R) ? 0 : k;
            const int jz = j + kk, pl = i + kk;  // (nz, nx > 3: one wrap at most)
            zp[k + 3] = in + (ctr + (long long)(jz < 0 ? kk + g.nz : jz >= g.nz ? kk - g.nz : kk) * g.nvs);
            const bool out = pl < 0 || pl >= g.nx, hal = out && halo != nullptr;
            const int px = pl < 0 ? (hal ? pl + R : pl + g.nx) : pl >= g.nx ? (hal ? pl - g.nx + R : pl - g.nx) : pl;
            xp[k + 3] = (hal ? halo : in) + ((long long)px * P + col);
            xfs[k + 3] = hal ? 2 * R * P : g.fs;
        }
        const double vxd = a.q.vx[v], vyd = a.q.vy[v], vzd = a.q.vz[v], wd = a.q.vw[v];
        const T fx = T(vxd * a.c.fxs), fz = T(vzd * a.c.fzs);
        const T kx = T(a.c.kx), kz = T(a.c.kz);
        const double *m = a.mom_in + cell * NMOM;
        const T ia = T(inp(m, vxd, vyd, vzd)), ib = T(inp(m + 4, vxd, vyd, vzd)), ie = T(inp(m + 8, vxd, vyd, vzd));
        T c4[4], a4[4], k4[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            T zs[7], xs[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const bool used = k >= 3 - R && k <= 3 + R;
                zs[k] = used ? ld_now(zp[k] + f * g.fs) : T(0);
                xs[k] = used && k != 3 ? ld_now(xp[k] + f * xfs[k]) : T(0);
            }
            xs[3] = c4[f] = zs[3];
            a4[f] = adv_axis(zs, fz) + adv_axis(xs, fx);
            k4[f] = ko_axis<T, KO6>(zs, kz) + ko_axis<T, KO6>(xs, kx);
        }
        T kv[4];
        commutator_half(c4, ia, ib, ie, a.c, kv, a4, k4);
        const long long o = ctr + hoff;
        const T cA = T(a.cA), cY = T(a.cY);
        T outm[4];  // the written state whose moments the next stage needs
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const long long idx = o + f * g.fs;
            if (MODE == MODE_RHS) {
                a.acc_dst[idx] = kv[f];
            } else if (MODE == MODE_S1Y) {
                outm[f] = c4[f] + cY * kv[f];  // Y2
                a.y_dst[idx] = outm[f];
            } else if (MODE == MODE_SY) {
                outm[f] = a.u[idx] + cY * kv[f];  // Y4
                a.y_dst[idx] = outm[f];
            } else if (MODE == MODE_S2B) {
                const T u = a.u[idx];
                a.acc_dst[idx] = (u + c4[f]) + cA * kv[f];  // B = U + Y2 + dt k2
                outm[f] = u + cY * kv[f];                   // Y3
                a.y_dst[idx] = outm[f];
            } else {
                outm[f] = third_plus(a.acc_src[idx] + c4[f], cA * kv[f]);  // (B + Y4)/3 + dt/6 k4
                a.acc_dst[idx] = outm[f];
            }
        }
        // velocity-moment contributions (nuosc_class.cpp:69-71): moment 4c + j
        // = weight j (w, w vx, w vy, w vz) x combination c of the half
        if constexpr (MODE != MODE_RHS) {  // (calRHS writes no state)
            const double w4[4] = {wd, vxd * wd, vyd * wd, vzd * wd};
            double d[3];
            if (half == 0) moment_terms<false>(outm[0], outm[1], outm[2], outm[3], d[0], d[1], d[2]);
            else moment_terms<true>(outm[0], outm[1], outm[2], outm[3], d[0], d[1], d[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int jw = 0; jw < 4; ++jw) mom[4 * c + jw] = w4[jw] * d[c];
        }
    }
    if constexpr (MODE != MODE_RHS) {
        // sum over the lanes of the (cell, half) (xor offsets below twp stay inside its group)
        for (int off = twp >> 1; off > 0; off >>= 1)
#pragma unroll
            for (int k = 0; k < NMOM; ++k) mom[k] += __shfl_xor_sync(0xffffffffu, mom[k], off);
        if (lane_in_cell == 0 && put) {
            double *p = a.mom_part + ((cell * nvb + (nvb - 1)) * 2 + half) * NMOM;
#pragma unroll
            for (int k = 0; k < NMOM; ++k) p[k] = mom[k];
        }
    }
}

}  // namespace nuosc
