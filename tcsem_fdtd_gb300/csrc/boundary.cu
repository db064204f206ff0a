// Air-interface boundary pipeline: Bz on the top plane (non-uniform) ->
// uniform L1 x M1 plane -> 2-D FFT -> upward-continuation filters -> inverse
// FFT -> bilinear remap back to the staggered BxAir / ByAir planes.
//
// The reference (UpContinuation_gpu.cu:166-274, SplineGridConvIR2R.cu:539-752)
// materialises the whole uniform plane three times per step (cuSPARSE spline
// solves, one R2C and two C2R cuFFT calls).  Every stage of that chain is
// linear and the spline remap is separable, BzAir = Py . Bz . Px^T, so this
// pipeline instead
//   1. remaps each of the M old rows to L1 uniform points with dense spline
//      weights (precomputed from the same natural-spline rule) and FFTs it
//      along x -- M rows, not M1, two real rows packed in one complex
//      transform;
//   2. per x-frequency column: applies Py in the x-frequency domain, FFTs
//      along y, multiplies by the two continuation filters, inverse-FFTs
//      along y and keeps only the rows the final bilinear remap samples;
//   3. inverse-FFTs those rows along x with Bx and By packed as the real and
//      imaginary parts of one complex transform;
//   4. bilinearly remaps into plane k = -1 of the Bx/By buffers.
// All transforms are in-shared-memory mixed-radix Stockham FFTs of arbitrary
// length written here (no cuFFT).
#include "boundary_body.cuh"

namespace tcsem {


// ---- single-survey kernels
template <typename T>
__global__ void __launch_bounds__(kBndThreads) k_rows_fwd(BoundaryDev<T> bd, const T *__restrict__ bz,
                                                          const T *__restrict__ tot, int nch, Geom g,
                                                          StepGate gate) {
    if (gate.base && gate.step() >= gate.nsteps) return;
    rows_fwd_cta<T>(bd, bz, tot, nch, g, blockIdx.x);
}
template <typename T> __global__ void __launch_bounds__(kBndThreads) k_cols(BoundaryDev<T> bd, StepGate gate) {
    if (gate.base && gate.step() >= gate.nsteps) return;
    cols_cta<T>(bd, blockIdx.x);
}
template <typename T> __global__ void __launch_bounds__(kBndThreads) k_rows_inv(BoundaryDev<T> bd, StepGate gate) {
    if (gate.base && gate.step() >= gate.nsteps) return;
    rows_inv_cta<T>(bd, blockIdx.x);
}
template <typename T> __global__ void k_bilinear(BoundaryDev<T> bd, T *bx, T *by, Geom g, StepGate gate) {
    if (gate.base && gate.step() >= gate.nsteps) return;
    bilinear_cta<T>(bd, bx, by, g, blockIdx.x, gridDim.x);
}

// ---- batched kernels: block b works for slot idx.slot_of(b)
// (FP32: six blocks on an SM, 40 registers.  With 46 it was five, and 8 surveys of up to 64 x 64 x 48 took 56.3 us per step
// instead of 49.7; the others measured, 4 to 8 of up to 200 x 180 x 120, take the same.)
template <typename T>
__device__ __forceinline__ const BoundarySlot<T> *bnd_slot(const BoundarySlot<T> *slots, const BatchIndex &idx,
                                                           int s, int &lb) {
    const int q = idx.slot_of(blockIdx.x);
    const BoundarySlot<T> *d = slots + q;
    if ((long)*d->step_base + s >= d->nsteps) return nullptr;
    lb = blockIdx.x - idx.off[q];
    return d;
}
template <typename T>
__global__ void __launch_bounds__(kBndThreads, sizeof(T) == 4 ? 6 : 4)
    k_rows_fwd_b(const BoundarySlot<T> *__restrict__ slots, const __grid_constant__ BatchIndex idx, int s) {
    int lb;
    const BoundarySlot<T> *d = bnd_slot(slots, idx, s, lb);
    if (d) rows_fwd_cta<T>(d->bd, d->bz, d->tot, d->nch, d->g, lb);
}
template <typename T>
__global__ void __launch_bounds__(kBndThreads, sizeof(T) == 4 ? 6 : 4)
    k_cols_b(const BoundarySlot<T> *__restrict__ slots, const __grid_constant__ BatchIndex idx, int s) {
    int lb;
    const BoundarySlot<T> *d = bnd_slot(slots, idx, s, lb);
    if (d) cols_cta<T>(d->bd, lb);
}
template <typename T>
__global__ void __launch_bounds__(kBndThreads)
    k_rows_inv_b(const BoundarySlot<T> *__restrict__ slots, const __grid_constant__ BatchIndex idx, int s) {
    int lb;
    const BoundarySlot<T> *d = bnd_slot(slots, idx, s, lb);
    if (d) rows_inv_cta<T>(d->bd, lb);
}
template <typename T>
__global__ void k_bilinear_b(const BoundarySlot<T> *__restrict__ slots, const __grid_constant__ BatchIndex idx, int s) {
    int lb;
    const BoundarySlot<T> *d = bnd_slot(slots, idx, s, lb);
    if (d) {
        const int q = idx.slot_of(blockIdx.x);
        bilinear_cta<T>(d->bd, d->bx, d->by, d->g, lb, idx.off[q + 1] - idx.off[q]);
    }
}

template <typename T> static size_t smem_rows(const BoundaryDev<T> &bd, int L) { return rows_fwd_layout(bd, L).total; }
template <typename T> static size_t smem_cols(const BoundaryDev<T> &bd) { return cols_layout(bd).total; }
template <typename T> size_t cols_apart(const BoundaryDev<T> &bd) { return cols_layout(bd).apart; }
// The columns' blocks start while the row stage's still hold some SMs, and crowd on the others.  Alone, 369 blocks of a
// 736 x 736 plane (35 KB each) in FP32: 47 or 37 us for the whole boundary from one process to the next, 35.4 with at most
// three on an SM; in FP64 160.  No region on top of another (55 and 110 KB): 36 to 39, and 170.
template <typename T> size_t cols_even(const BoundaryDev<T> &bd) {
    int dev = 0, sms = 0, sm = 0, most = 0, own = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&own, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
        return 0;
    const int share = (bd.H + sms - 1) / sms, bytes = sm / share - own;
    return share == 1 || bytes <= 0 ? 0 : (size_t)(bytes < most ? bytes : most) / 128 * 128;
}
template <typename T> static size_t smem_inv(const BoundaryDev<T> &bd) { return rows_inv_layout(bd).total; }

template <typename T> size_t boundary_smem_need(const BoundaryDev<T> &bd, int L) {
    size_t a = smem_rows(bd, L), b = cols_layout(bd).apart, c = smem_inv(bd);  // the limit on planes is that of regions apart
    return a > b ? (a > c ? a : c) : (b > c ? b : c);
}

template <typename T> cudaError_t boundary_configure(const BoundaryDev<T> &bd, int L) {
    cudaError_t e = allow_shared(k_rows_fwd<T>, smem_rows(bd, L));
    if (e == cudaSuccess) e = allow_shared(k_cols<T>, cols_layout(bd).apart);
    if (e == cudaSuccess) e = allow_shared(k_rows_inv<T>, smem_inv(bd));
    return e;
}

template <typename T> BoundaryBlocks boundary_blocks(const BoundaryDev<T> &bd, const Geom &g) {
    BoundaryBlocks b;
    b.rows_fwd = (g.M + 1) / 2;
    b.cols = bd.H;
    b.rows_inv = bd.S;
    b.bilinear = ((g.L + 1) * g.M + g.L * (g.M + 1) + 255) / 256;
    b.smem_rows = smem_rows(bd, g.L);
    b.smem_cols = smem_cols(bd);
    b.smem_inv = smem_inv(bd);
    return b;
}

template <typename T> cudaError_t boundary_configure_batched(const size_t *smem) {
    cudaError_t e = allow_shared(k_rows_fwd_b<T>, smem[0]);
    if (e == cudaSuccess) e = allow_shared(k_cols_b<T>, smem[1]);
    if (e == cudaSuccess) e = allow_shared(k_rows_inv_b<T>, smem[2]);
    return e;
}

// a launch that may begin while the previous kernel on the stream is still running
// (programmatic dependent launch; the kernel waits with pdl_wait_prev before its reads)
template <typename... P, typename... A>
static void launch_after(bool pdl, void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

template <typename T>
cudaError_t launch_boundary_batched(const BoundarySlot<T> *slots, const BatchIndex *idx, const size_t *smem, int s,
                                    cudaStream_t st) {
    if (idx[0].total()) k_rows_fwd_b<T><<<idx[0].total(), kBndThreads, smem[0], st>>>(slots, idx[0], s);
    if (idx[1].total()) launch_after(true, k_cols_b<T>, idx[1].total(), kBndThreads, smem[1], st, slots, idx[1], s);
    if (idx[2].total()) launch_after(true, k_rows_inv_b<T>, idx[2].total(), kBndThreads, smem[2], st, slots, idx[2], s);
    if (idx[3].total()) launch_after(true, k_bilinear_b<T>, idx[3].total(), 256, (size_t)0, st, slots, idx[3], s);
    return cudaGetLastError();
}

template <typename T>
void launch_boundary(const BoundaryDev<T> &bd, const Geom &g, const T *bz, const T *tot, int nch, T *bx, T *by,
                     StepGate gate, cudaStream_t st, size_t cols_smem, bool pdl) {
    k_rows_fwd<T><<<(g.M + 1) / 2, kBndThreads, smem_rows(bd, g.L), st>>>(bd, bz, tot, nch, g, gate);
    // The column stage starts early only where the caller asks (beside a long sweep its early CTAs
    // would take slots the sweep's single wave needs at the start of a step); the last two stages
    // always do: by then the sweep's CTAs are all resident.
    const size_t cols = smem_cols(bd) > cols_smem ? smem_cols(bd) : cols_smem;
    launch_after(pdl, k_cols<T>, bd.H, kBndThreads, cols, st, bd, gate);
    launch_after(true, k_rows_inv<T>, bd.S, kBndThreads, smem_inv(bd), st, bd, gate);
    int n = (g.L + 1) * g.M + g.L * (g.M + 1);
    launch_after(true, k_bilinear<T>, (n + 255) / 256, 256, (size_t)0, st, bd, bx, by, g, gate);
}

#define INST(T)                                                                                            \
    template size_t cols_apart<T>(const BoundaryDev<T> &);                                                        \
    template size_t cols_even<T>(const BoundaryDev<T> &);                                                         \
    template size_t boundary_smem_need<T>(const BoundaryDev<T> &, int);                                   \
    template cudaError_t boundary_configure<T>(const BoundaryDev<T> &, int);                              \
    template void launch_boundary<T>(const BoundaryDev<T> &, const Geom &, const T *, const T *, int, T *, T *,  \
                                     StepGate, cudaStream_t, size_t, bool);                                     \
    template BoundaryBlocks boundary_blocks<T>(const BoundaryDev<T> &, const Geom &);                     \
    template cudaError_t launch_boundary_batched<T>(const BoundarySlot<T> *, const BatchIndex *, const size_t *, int, \
                                                    cudaStream_t);                                        \
    template cudaError_t boundary_configure_batched<T>(const size_t *);
INST(float)
INST(double)
#undef INST

}  // namespace tcsem
