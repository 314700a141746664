// internal.cuh -- device-side data layout, kernel argument blocks and launch
// entry points shared by the CUDA kernels and the C-ABI host layer.
//
// HBM layout of one register (a FieldVar of the reference): 8 fields, each
// [x][z][v] with the velocity innermost and `nvs` velocities per (x,z) row
// (nv rounded up so every row starts on a 16-byte boundary).  No ghost cells
// are stored: the stencils wrap x and z periodically in-kernel, which is what
// updatePeriodicBoundary's ghost fill amounts to for the plus-shaped stencil
// (nuosc_boundary.cpp:4-52).  Padding velocities carry zero weight, zero
// velocity and zero state, so every kernel may process them and they stay 0.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nuosc {

constexpr int NF = 8;  // ee, mm, emr, emi, bee, bmm, bemr, bemi

// Seeded draws of the initial data: a counter-based hash (splitmix64
// finaliser) of (seed, i, j), uniform in [0, 1) with 53 bits; host and device
// give the same value.  Replaces the reference's rand() (nuosc_init.cpp:5, 33).
__host__ __device__ inline uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__host__ __device__ inline double seeded_uniform(uint64_t seed, int i, int j) {
    const uint64_t key = ((uint64_t)(uint32_t)i << 32) | (uint64_t)(uint32_t)j;
    return (double)(mix64(mix64(seed) ^ key) >> 11) * 0x1.0p-53;
}
constexpr int NMOM = 12;  // emRm[4], emIp[4], eemm[4] (nuosc_class.cpp:28-31)

struct Geom {
    int nx, nz, nv, nvs;
    long long fs;     // elements per field = nx*nz*nvs
    long long ncell;  // nx*nz
};

// Physics coefficients of calRHS (nuosc_class.cpp:112-183, nuosc_class.h:120-122).
struct Coeffs {
    double fxs, fzs;  // advection: factor_x = vx * fxs, fxs = -1/(12 dx) (same for z)
    double kx, kz;    // KO strength: -ko/dx/64 (6th difference) or -ko/dx/16 (4th)
    double mu, pmo, ct, st;
    // KO weights of the symmetric sums s_k = x[-k] + x[+k] and of the centre,
    // per axis, for the fused stencil of the x-march kernel:
    //   6th difference: k3 = eps, k2 = -6 eps, k1 = 15 eps, centre -20 (eps_x + eps_z)
    //   4th difference: k3 = 0,   k2 = eps,    k1 = -4 eps, centre   6 (eps_x + eps_z)
    double kz3, kz2, kz1, kx3, kx2, kx1, kc;
};

struct Quad {
    const double *vx, *vy, *vz, *vw;  // [nvs], zero in the padding
};

// One RK stage: k = L(in); then, by mode,
//   MODE_RHS : acc_dst = k
//   MODE_S1  : acc_dst = in + cA*k ;          y_dst = in + cY*k
//   MODE_S23 : acc_dst = acc_src + cA*k ;     y_dst = u  + cY*k
//   MODE_S4  : acc_dst = acc_src + cA*k
// (the classic 16-pass sequence of the direct and cp.async paths), and the
// 12-pass sequence of the TMA path:
//   MODE_S1Y : y_dst = in + cY*k                       (Y2 = U + dt/2 k1)
//   MODE_S2B : y_dst = u + cY*k ; acc_dst = (u + in) + cA*k
//                                   (Y3 = U + dt/2 k2, B = U + Y2 + dt k2)
//   MODE_SY  : y_dst = u + cY*k                        (Y4 = U + dt k3)
//   MODE_S4B : acc_dst = (acc_src + in)/3 + cA*k
// In S4B, in = Y4, acc_src = B and cA = dt/6: (B + Y4)/3 = U + dt/6 k1 +
// dt/3 k2 + dt/3 k3, so the update is U + dt/6 (k1 + 2 k2 + 2 k3 + k4)
// without reading U.
enum StageMode {
    MODE_RHS = 0, MODE_S1 = 1, MODE_S23 = 2, MODE_S4 = 3, MODE_S1Y = 5, MODE_SY = 6, MODE_S4B = 7, MODE_S2B = 8
};

template <typename T>
struct StageArgs {
    const T *in;
    const T *u;
    const T *acc_src;
    T *acc_dst;
    T *y_dst;
    const double *mom_in;  // [ncell][12] moments of `in`
    double *mom_part;      // x-march: per-(cell, v-block, half) partial moments of the new state
    Quad q;
    Geom g;
    Coeffs c;
    double cA, cY;
    int *status;           // device status word (bounded waits)
    // test of the TMA kernels' bounded waits (0 in normal use): the first
    // front box of the instance's first tile declares this many bytes more
    // than its copies deliver, so every wait on it runs out
    unsigned fault_tx;
    // x-slab of a domain-decomposed solve (nullptr: the stencil wraps x
    // periodically inside the register): the R planes on each side of the
    // slab, [8 fields][2R planes][nz][nvs], planes 0..R-1 left of plane 0 and
    // R..2R-1 right of plane nx-1, filled by the halo exchange before the stage
    const T *halo;
};

// element offset of plane p in [-R, 0) or [nx, nx + R) of field F (0..7) in a
// slab's halo buffer
__host__ __device__ inline long long halo_offset(int F, int p, int nx, int R, long long P) {
    const int hp = p < 0 ? p + R : p - nx + R;
    return ((long long)F * 2 * R + hp) * P;
}

// The z tiles of a march: ceil(nz / tz) tiles of tz rows (at least two: nz >= tz +
// 6).  Where tz does not divide nz they are spread evenly and overlap.
// Neighbouring tiles are at least 3 >= R rows apart, so only the first and the
// last tile's box crosses the periodic end and the box pieces are those of an
// exact division.  Tile t starts at row t (nz - tz) / (tiles - 1), formed as t q +
// t rem / (tiles - 1) with the host's q and rem: the product in one piece leaves 32
// bits from nz = 131,080 (8 rows) or 185,377 (16 rows), while t and rem are below
// 65,535, the largest grid's y extent, and their product below 2^32.
struct ZTiles {
    unsigned n, q, rem;
    ZTiles(int nz, int tz)
        : n((unsigned)((nz + tz - 1) / tz)), q((unsigned)(nz - tz) / (n - 1)), rem((unsigned)(nz - tz) % (n - 1)) {}
    __host__ __device__ int row(unsigned t) const { return (int)(t * q + t * rem / (n - 1)); }
    // rows at the start of tile t that tile t - 1 has too: they are tile t - 1's to
    // store, so that every row is stored by one tile (q is tz where tz divides nz)
    __host__ __device__ int shared_rows(unsigned t, int tz) const {
        return t > 0 && q != (unsigned)tz ? tz - (row(t) - row(t - 1)) : 0;
    }
};

// Programmatic dependent launch, between the march and the moment finalize of a
// lone solve whose march is a single wave (`early`): each kernel lets the next one
// be launched from its start, and waits for the one before it (complete, its
// writes visible) before it touches anything that depends on it.  Other launches
// are ordinary and do not wait: under load the wait alone costs a CTA about 10 us
// (512x256x642, 18 waves: finalize 0.10 -> 0.16 ms, S1 2.65 -> 2.87).
#ifdef __CUDACC__
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
template <typename... P, typename... A>
inline cudaError_t launch_dependent(bool early, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
#endif

// ---------------------------------------------------------------- launches
// halt (null by default): a batch member's stop flag; when set, nothing is done
template <typename T>
cudaError_t launch_moments(const T *reg, double *mom, Quad q, Geom g, cudaStream_t s, const int *halt = nullptr);
template <typename T>
cudaError_t launch_stage_direct(const StageArgs<T> &a, int mode, bool ko6, cudaStream_t s);

// x-march kernel: tile shape chosen by the autotuner (tile.cu)
struct XTile {
    int tz;        // z rows per CTA
    int lx;        // x planes marched per CTA (0 in the tile table: xtma_lx picks it for the grid)
    int vb;        // velocities per CTA (32)
    int kind = 0;  // preferred x-march kernel from the tile table: 2 cp.async, 3 TMA, 0 either
    int msum = 1;  // FP32 TMA march: moment partials summed in FP64 (1) or in float within a block (0)
    bool early = false;  // of one launch: it is a single wave (xtma_waves)
    long long *launched = nullptr;  // of one launch: where its kernels are counted
};
template <typename T>
bool xmarch_supported(const Geom &g, bool ko6, XTile t);
// its tile where the handle's is not the user's or the tile table's
XTile xmarch_tile(const Geom &g, XTile t, int sms);
template <typename T>
cudaError_t launch_stage_xmarch(const StageArgs<T> &a, int mode, bool ko6, XTile t, cudaStream_t s);
// TMA-fed variant of the x-march kernel (xtma.cu).  fits: it runs this grid
// (nz >= tz + 6); supported: and nz % tz == 0, which batches, x-slabs and an
// explicitly requested TMA kernel need
template <typename T>
bool xtma_fits(const Geom &g, XTile t);
template <typename T>
bool xtma_supported(const Geom &g, XTile t);
// its launch has a grid the device takes (65,535 z tiles, 32,767 segments)
bool xtma_grid_ok(const Geom &g, XTile t);
// x planes per CTA for grid g on a device of `sms` SMs
template <typename T>
int xtma_lx(const Geom &g, int tz, int sms);
// The stage, the tail velocities included; not for grids with xtma_all_tail.  The
// launchers of the march add the kernels they start (one, or two with a tail
// kernel) to *launched.
template <typename T>
cudaError_t launch_stage_xtma(const StageArgs<T> &a, int mode, bool ko6, XTile t, bool early, long long *launched,
                              cudaStream_t s);
// waves of CTAs (a tail column included) of the stage's launch on `sms` SMs.  One:
// all CTAs are resident at once, and the kernel after it may be launched, and wait,
// while it runs (with more, waiting CTAs would take SMs from the ones still to come)
template <typename T>
int xtma_waves(const Geom &g, XTile t, int sms);
// every velocity fits the tail block: launch_stage_tail runs the stage
template <typename T>
bool xtma_all_tail(const Geom &g);
// calRHS (MODE_RHS: acc_dst = L(in), mom_in = the moments of in) on the TMA
// march, for grids and buffers it fits
template <typename T>
bool rhs_xtma_fits(const Geom &g, const void *in, const void *out);
// whether it is the faster kernel there
bool rhs_xtma_pays(const Geom &g, bool ko6);
template <typename T>
cudaError_t launch_rhs_xtma(const StageArgs<T> &a, bool ko6, long long *launched, cudaStream_t s);
// velocity blocks of the TMA kernel's moment partials (32 velocities per block in FP64, 64 in FP32)
template <typename T>
int xtma_num_vblocks(const Geom &g);
// Batched TMA stage (xtma.cu): one persistent launch runs one RK stage of many
// instances.  Each instance has an entry (its tensor maps and StageArgs) in a
// device table; the CTAs of a persistent grid take the tiles of all
// instances from an atomic work-list cursor.
// Tile k of an instance is the tile its own launch runs as CTA k, so each
// instance gets the same bits as when stepped alone.
template <typename T>
size_t xtma_batch_item_bytes();
// Encodes the table entry of one instance into `item` (host memory,
// xtma_batch_item_bytes bytes); returns the instance's tile count, or -1 when
// the instance cannot run with this tz.
template <typename T>
long long xtma_batch_fill(void *item, const StageArgs<T> &a, bool ko6, int tz, int lx);
// CTAs of a persistent launch on `device` (also sets the kernel's dynamic
// shared-memory limit); -1 on failure.  vac: some instance has pmo != 0;
// m64: FP32 moment partials summed in FP64 (XTile::msum; FP64 always is).
template <typename T>
int xtma_batch_grid(int mode, bool ko6, int tz, bool vac, bool m64, int device);
// starts[i] = tiles of instances 0..i-1 (instances ordered as the caller
// wants them served); grid = xtma_batch_grid(...); *counter must be 0 at the
// launch (the work-list cursor); halt[i] != 0 (halt may be null): instance i
// has stopped, its tiles are skipped
template <typename T>
cudaError_t launch_stage_xtma_batch(const void *items, const long long *starts, int n, long long ntiles,
                                    unsigned long long *counter, const int *halt, int mode, bool ko6, int tz,
                                    bool vac, bool m64, int grid, cudaStream_t s);
// Tail of the TMA x-march stage (tail.cu): when the last velocity block of
// the TMA kernel would hold at most a quarter block of real velocities, the
// velocities from xtma_tail_v0 on are computed by a one-thread-per-(cell,
// velocity) kernel that writes the last block's moment partials; the TMA
// kernel then runs the full blocks only.  Returns nvs when there is no tail.
template <typename T>
int xtma_tail_v0(const Geom &g);
int tail_lanes(int width);  // lanes per cell: width rounded up to a power of 2
template <typename T>
cudaError_t launch_stage_tail(const StageArgs<T> &a, int mode, bool ko6, int v0, int nvb, cudaStream_t s);
template <typename T>
struct TailItem {
    StageArgs<T> a;
    int v0, twp, nvb;
    int member;  // the instance's index in the batch (its halt flag)
};
// starts[i]: first thread of item i (ranges of 2 * ncell * twp threads, one
// per (cell, flavour half, tail lane), each rounded up to a multiple of 32);
// total: threads of all items; halt as for launch_stage_xtma_batch
template <typename T>
cudaError_t launch_stage_tail_batch(const TailItem<T> *items, const long long *starts, int n, long long total,
                                    const int *halt, int mode, bool ko6, cudaStream_t s);
// moment_finalize of many instances in one launch (xmarch.cu); starts[i] =
// sum over instances 0..i-1 of ncell * 12
struct FinalizeItem {
    const double *part;
    double *mom;
    long long ncell;
    int nvb;
};
cudaError_t launch_moment_finalize_batch(const FinalizeItem *items, const long long *starts, int n, long long total,
                                         const int *halt, cudaStream_t s);
// *halt = step when *halt is 0 and the analysis sums `sums` (launch_analysis's
// out) meet the reference's stop criterion: a non-finite value or
// max||P|-1| >= 10 (nuosc_ana.cpp:131) (kernels.cu)
cudaError_t launch_halt_check(const double *sums, int *halt, int step, cudaStream_t s);
// value a kernel writes into StageArgs::status when a bounded wait expires
constexpr int NUOSC_TIMEOUT_CODE = 1;
// one warp waits `spins` polls on an mbarrier that never completes, then sets
// *status = NUOSC_TIMEOUT_CODE (xtma.cu; the self-test of the bounded waits)
cudaError_t launch_wait_selftest(int *status, unsigned spins, cudaStream_t s);

// records msg as the calling thread's nuosc_last_error() and returns code (capi.cu)
int set_last_error(int code, const char *msg);
int xmarch_num_vblocks(const Geom &g, XTile t);
// early: the march launches around it are single waves (xtma_waves)
cudaError_t launch_moment_finalize(const double *part, double *mom, Geom g, int nvb, bool early, cudaStream_t s);

template <typename T>
cudaError_t launch_init(T *reg, const double *G0, const double *G0b, Geom g, int ipt, double eps0,
                        double sigma, double z0, double dz, uint64_t seed, const double *zprof, int xoff,
                        cudaStream_t s);
// Analysis partial sums; `part` holds ANA_BLOCKS * ANA_NQ doubles, `out` ANA_NQ sums
// and *status (0 without a status word).
constexpr int ANA_NQ = 12;
constexpr int ANA_BLOCKS = 296;
template <typename T>
cudaError_t launch_analysis(const T *reg, const double *G0, const double *G0b, const double *vw, Geom g,
                            double *part, double *out, const int *status, cudaStream_t s);
template <typename T>
cudaError_t launch_gather(const T *reg, int field, const int *xidx, int sx, const int *vidx, int sv,
                          const double *G0, const double *G0b, Geom g, double *out, cudaStream_t s);
template <typename T>
cudaError_t launch_import(T *reg_field, const double *src, Geom g, int layout, int gx, int gz, cudaStream_t s);
template <typename T>
cudaError_t launch_export(const T *reg_field, double *dst, Geom g, int layout, int gx, int gz, cudaStream_t s);
template <typename T>
cudaError_t launch_vectorize(T *dst, const T *a, double c, const T *b, const T *d, Geom g, cudaStream_t s);
template <typename T>
cudaError_t launch_renormalize(T *reg, const double *G0, const double *G0b, Geom g, cudaStream_t s,
                               const int *halt = nullptr);

}  // namespace nuosc
