// tail.cu -- the last, nearly empty velocity block of an x-march stage.
//
// The TMA x-march kernel runs 32 (FP64) or 64 (FP32) velocities per CTA, one
// 8-byte value per lane.  When nv leaves only a few velocities in the last block
// (642 = 20 x 32 + 2 in FP64, 644 = 10 x 64 + 4 in FP32), a CTA for that
// block would issue a full block's instructions for a handful of active
// lanes -- up to a tenth of the stage's issue slots.  Those tail velocities
// are computed here instead, one thread per (cell, tail velocity, flavour
// half) with 4 fields (tail.cuh), the stencil read with plain loads (the
// tail columns of a few planes stay in L2), the same fused RK epilogue, and
// the velocity-moment partials of the written state summed over the tail
// lanes of the (cell, half) into the last block's slots of the partial
// array, so the fixed-order moment_finalize is unchanged.
//
// A solve stepped alone in launches of up to 6 waves runs its tail in CTAs of
// the march launch itself (xtma.cu); the kernels here run the tails of larger
// launches and of a batch, and a solve whose velocities all fit the tail (12
// velocities in FP32).
#include "internal.cuh"
#include "tail.cuh"

namespace nuosc {

namespace {

constexpr int TAIL_BLOCK = 256;

// thread t: lane l = t % twp of (cell, half) = (t / twp) / 2, (t / twp) % 2
template <typename T, bool KO6, int MODE>
__global__ void __launch_bounds__(TAIL_BLOCK, 3) k_stage_tail(const StageArgs<T> a, int v0, int twp, int nvb) {
    const long long t = (long long)blockIdx.x * TAIL_BLOCK + threadIdx.x;
    const int l = (int)(t & (twp - 1));
    const long long ch = t / twp, cell = ch >> 1;
    const int v = v0 + l;
    tail_point<T, KO6, MODE>(a, cell, (int)(ch & 1), v, cell < a.g.ncell && v < a.g.nvs, cell < a.g.ncell,
                             twp, nvb, l);
}

// many instances' tails in one launch: item i covers threads [starts[i],
// starts[i] + 2 ncell_i twp_i), each range a multiple of 32 threads so that
// no warp spans two instances
template <typename T, bool KO6, int MODE>
__global__ void __launch_bounds__(TAIL_BLOCK, 2) k_stage_tail_batch(const TailItem<T> *__restrict__ items,
                                                                 const long long *__restrict__ starts, int n,
                                                                 long long total, const int *__restrict__ halt) {
    const long long t = (long long)blockIdx.x * TAIL_BLOCK + threadIdx.x;
    if (t - (threadIdx.x & 31) >= total) return;  // whole warps past the end
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (starts[mid] <= t) lo = mid;
        else hi = mid - 1;
    }
    const TailItem<T> &e = items[lo];
    if (halt && halt[e.member]) return;  // a stopped instance: no work (whole warps: one item per warp)
    const long long u = t - starts[lo];
    const int l = (int)(u & (e.twp - 1));
    const long long ch = u / e.twp, cell = ch >> 1;
    const int v = e.v0 + l;
    tail_point<T, KO6, MODE>(e.a, cell, (int)(ch & 1), v, cell < e.a.g.ncell && v < e.a.g.nvs, cell < e.a.g.ncell,
                             e.twp, e.nvb, l);
}

template <typename T, bool KO6>
cudaError_t launch_tail_ko(const StageArgs<T> &a, int mode, int v0, int twp, int nvb, cudaStream_t s) {
    const long long threads = a.g.ncell * 2 * twp;
    const unsigned blocks = (unsigned)((threads + TAIL_BLOCK - 1) / TAIL_BLOCK);
    switch (mode) {
    case MODE_RHS: k_stage_tail<T, KO6, MODE_RHS><<<blocks, TAIL_BLOCK, 0, s>>>(a, v0, twp, nvb); break;
    case MODE_S1Y: k_stage_tail<T, KO6, MODE_S1Y><<<blocks, TAIL_BLOCK, 0, s>>>(a, v0, twp, nvb); break;
    case MODE_S2B: k_stage_tail<T, KO6, MODE_S2B><<<blocks, TAIL_BLOCK, 0, s>>>(a, v0, twp, nvb); break;
    case MODE_SY: k_stage_tail<T, KO6, MODE_SY><<<blocks, TAIL_BLOCK, 0, s>>>(a, v0, twp, nvb); break;
    case MODE_S4B: k_stage_tail<T, KO6, MODE_S4B><<<blocks, TAIL_BLOCK, 0, s>>>(a, v0, twp, nvb); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename T, bool KO6>
cudaError_t launch_tail_batch_ko(const TailItem<T> *items, const long long *starts, int n, long long total,
                                 const int *halt, int mode, cudaStream_t s) {
    const unsigned blocks = (unsigned)((total + TAIL_BLOCK - 1) / TAIL_BLOCK);
    switch (mode) {
    case MODE_S1Y: k_stage_tail_batch<T, KO6, MODE_S1Y><<<blocks, TAIL_BLOCK, 0, s>>>(items, starts, n, total, halt); break;
    case MODE_S2B: k_stage_tail_batch<T, KO6, MODE_S2B><<<blocks, TAIL_BLOCK, 0, s>>>(items, starts, n, total, halt); break;
    case MODE_SY: k_stage_tail_batch<T, KO6, MODE_SY><<<blocks, TAIL_BLOCK, 0, s>>>(items, starts, n, total, halt); break;
    case MODE_S4B: k_stage_tail_batch<T, KO6, MODE_S4B><<<blocks, TAIL_BLOCK, 0, s>>>(items, starts, n, total, halt); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace

int tail_lanes(int width) {
    int twp = 1;
    while (twp < width) twp *= 2;
    return twp;
}

template <typename T>
cudaError_t launch_stage_tail(const StageArgs<T> &a, int mode, bool ko6, int v0, int nvb, cudaStream_t s) {
    const int width = a.g.nvs - v0;
    if (width < 1 || width > 32 || (!a.mom_part && mode != MODE_RHS) || nvb < 1) return cudaErrorInvalidValue;
    const int twp = tail_lanes(width);
    return ko6 ? launch_tail_ko<T, true>(a, mode, v0, twp, nvb, s) : launch_tail_ko<T, false>(a, mode, v0, twp, nvb, s);
}

template <typename T>
cudaError_t launch_stage_tail_batch(const TailItem<T> *items, const long long *starts, int n, long long total,
                                    const int *halt, int mode, bool ko6, cudaStream_t s) {
    if (n < 1 || total < 1) return cudaErrorInvalidValue;
    return ko6 ? launch_tail_batch_ko<T, true>(items, starts, n, total, halt, mode, s)
               : launch_tail_batch_ko<T, false>(items, starts, n, total, halt, mode, s);
}

template cudaError_t launch_stage_tail<double>(const StageArgs<double> &, int, bool, int, int, cudaStream_t);
template cudaError_t launch_stage_tail<float>(const StageArgs<float> &, int, bool, int, int, cudaStream_t);
template cudaError_t launch_stage_tail_batch<double>(const TailItem<double> *, const long long *, int, long long,
                                                     const int *, int, bool, cudaStream_t);
template cudaError_t launch_stage_tail_batch<float>(const TailItem<float> *, const long long *, int, long long,
                                                    const int *, int, bool, cudaStream_t);

}  // namespace nuosc
