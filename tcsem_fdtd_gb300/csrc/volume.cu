// Volume kernels: DuFort-Frankel E update, source injection and B update on
// the staggered non-uniform grid.
//
// Two forms:
//  * reference-structured kernels (k_update_e, k_source, k_update_bxy,
//    k_update_bz) that update one field set in place, stage by stage, as
//    ElectricalField/Bderivate do (ElectricalFiled.cu:89-475, Bderivate.cu:79-265);
//  * the production fused sweep (k_sweep): one pass over the volume per
//    time step that reads the old E/B/sigma planes and writes the new E and B
//    into the other buffer of a ping-pong pair.  It marches z bottom-up so the
//    div B = 0 prefix for Bz (Bderivate.cu:202-265) runs in a register, and each
//    CTA recomputes the one-cell halo of E/B it needs instead of waiting for
//    its neighbours.  Algorithmic traffic: 7 words read + 6 written per cell.
#include "kernels.cuh"
#include "async.cuh"
#include "check.cuh"
#include "sweep.cuh"

namespace tcsem {

// ------------------------------------------------------------------ helpers

template <typename T> __device__ __forceinline__ T recip(T x) { return T(1) / x; }

// DuFort-Frankel update of one E component (ElectricalFiled.cu:138-139):
//   E <- (2g - s dt)/(2g + s dt) E + 4 dt/(2g + s dt) curl / mu0
template <typename T>
__device__ __forceinline__ T df_update(const StepScalars<T> &s, T sigma, T e_old, T curl) {
    T sdt = sigma * s.dt;
    T r = recip(s.lam2 + sdt);
    return (s.lam2 - sdt) * r * e_old + s.c4 * r * curl;
}

// ----------------------------------------------------- reference-structured
//
// One block per 32 x 8 cells of a plane: a host that steps a small grid stage by stage waits for latency, and a
// thread that walks a column waits for every plane of it.  64 x 64 x 48 in FP32 (device time, cold): E 82.6 us as
// columns, 5.2 as planes; Bx and By 55.0 and 4.4.  256 x 256 x 160, the whole call of E: 519 and 126 us.

template <typename T>
__global__ void k_update_e(Geom g, FieldSet<T> f, const T *__restrict__ con, Axis<T> ax, StepScalars<T> s, int *err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    if (i >= g.L || j >= g.M) return;
    const long long PS = g.PS, XP = g.XP;
    const bool vx = j >= 1, vy = i >= 1, vz = vx && vy;
    const T rdy2 = vx ? ax.rdy2[j] : T(0), rdx2 = vy ? ax.rdx2[i] : T(0), rzs = ax.rdzs[k];
    const long long c = g.at(i, j, k);
    if (!TCSEM_IN(c + PS, g.total(), err) || !TCSEM_IN(c - PS - XP - 1, g.total(), err)) return;
    if (vx) {  // UpdateEx, ElectricalFiled.cu:89-175
        T sg = T(0.5) * (T(0.5) * (con[c - XP] + con[c]) + T(0.5) * (con[c - PS - XP] + con[c - PS]));
        T curl = (f.bz[c] - f.bz[c - XP]) * rdy2 - (f.by[c] - f.by[c - PS]) * rzs;
        f.ex[c] = df_update(s, sg, f.ex[c], curl);
    }
    if (vy) {  // UpdateEy, :178-274
        T sg = T(0.25) * (con[c - 1] + con[c] + con[c - PS - 1] + con[c - PS]);
        T curl = (f.bx[c] - f.bx[c - PS]) * rzs - (f.bz[c] - f.bz[c - 1]) * rdx2;
        f.ey[c] = df_update(s, sg, f.ey[c], curl);
    }
    if (vz) {  // UpdateEz, :277-345
        T sg = T(0.25) * (con[c - XP - 1] + con[c - XP] + con[c - 1] + con[c]);
        T curl = (f.by[c] - f.by[c - 1]) * rdx2 - (f.bx[c] - f.bx[c - XP]) * rdy2;
        f.ez[c] = df_update(s, sg, f.ez[c], curl);
    }
}

// AddTx_x/_y/_z (ElectricalFiled.cu:347-475): one thread per injected cell
template <typename T>
__global__ void k_source(Geom g, FieldSet<T> f, SourceTable<T> src, T wave, int *err) {
    for (int sgi = 0; sgi < src.nseg; sgi++) {
        for (int q = threadIdx.x; q < src.count[sgi]; q += blockDim.x) {
            int i = src.i[sgi], j = src.j[sgi], k = src.k[sgi];
            T *e = src.comp[sgi] == 0 ? f.ex : src.comp[sgi] == 1 ? f.ey : f.ez;
            if (src.comp[sgi] == 0) i += q; else if (src.comp[sgi] == 1) j += q; else k += q;
            if (TCSEM_IN(g.at(i, j, k), g.total(), err)) e[g.at(i, j, k)] -= wave * src.coef[src.off[sgi] + q];
        }
        __syncthreads();
    }
}

// UpdateBx/UpdateBy, Bderivate.cu:79-200
template <typename T>
__global__ void k_update_bxy(Geom g, FieldSet<T> f, Axis<T> ax, T dtb, int *err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    if (i >= g.L || j >= g.M) return;
    const long long PS = g.PS, XP = g.XP;
    const T rdy = ax.rdy[j], rdx = ax.rdx[i], rdz = ax.rdz[k];
    const long long c = g.at(i, j, k);
    if (!TCSEM_IN(c + PS, g.total(), err) || !TCSEM_IN(c, g.total(), err)) return;
    if (i >= 1) f.bx[c] += ((f.ey[c + PS] - f.ey[c]) * rdz - (f.ez[c + XP] - f.ez[c]) * rdy) * dtb;
    if (j >= 1) f.by[c] += ((f.ez[c + 1] - f.ez[c]) * rdx - (f.ex[c + PS] - f.ex[c]) * rdz) * dtb;
}

// UpdateBz, Bderivate.cu:202-265: div B = 0, integrated from the bottom up.  A block owns 32 columns of a row: its
// eight warps form the terms of 64 planes, one warp adds them up (only the sums are serial), all store.
// 64 x 64 x 48 (cold): 28.6 us as one thread per column, plane after plane, 8.1 us.
constexpr int kBzPlanes = 64, kBzWarps = 8;
template <typename T>
__global__ void __launch_bounds__(32 * kBzWarps) k_update_bz(Geom g, const T *__restrict__ bx, const T *__restrict__ by,
                                                            T *__restrict__ bz, Axis<T> ax, int *err) {
    __shared__ T d[kBzPlanes][32];
    const int lane = threadIdx.x, i = blockIdx.x * 32 + lane, j = blockIdx.y, w = threadIdx.y;
    const long long PS = g.PS, XP = g.XP;
    const bool in = i < g.L;
    const T rdx = in ? ax.rdx[i] : T(0), rdy = ax.rdy[j];
    T acc = T(0);
    for (int k0 = g.N - 1; k0 >= 0; k0 -= kBzPlanes) {
        const int n = min(kBzPlanes, k0 + 1);
#pragma unroll
        for (int q = w; q < kBzPlanes; q += kBzWarps) {
            const long long c = g.at(i, j, k0 - q);
            if (q < n && in && TCSEM_IN(c + XP, g.total(), err) && TCSEM_IN(c, g.total(), err))
                d[q][lane] = (bx[c + 1] - bx[c]) * rdx + (by[c + XP] - by[c]) * rdy;
        }
        __syncthreads();
        if (w == 0)
            for (int q = 0; q < n; q++) {
                acc += ax.dzk[k0 - q] * d[q][lane];
                d[q][lane] = acc;
            }
        __syncthreads();
#pragma unroll
        for (int q = w; q < kBzPlanes; q += kBzWarps) {
            const long long c = g.at(i, j, k0 - q);
            if (q < n && in && TCSEM_IN(c, g.total(), err)) bz[c] = d[q][lane];
        }
        __syncthreads();
    }
}

template <typename T>
void launch_update_e(const Geom &g, FieldSet<T> f, const T *con, const Axis<T> &ax, StepScalars<T> s,
                     const SourceTable<T> &src, int *err, cudaStream_t st) {
    dim3 blk(32, 8), grd((g.L + 31) / 32, (g.M + 7) / 8, g.N);
    k_update_e<T><<<grd, blk, 0, st>>>(g, f, con, ax, s, err);
    if (src.nseg > 0 && s.wave != T(0)) k_source<T><<<1, 128, 0, st>>>(g, f, src, s.wave, err);
}

template <typename T>
void launch_bderivate(const Geom &g, FieldSet<T> f, const Axis<T> &ax, T dtb, int *err, cudaStream_t st) {
    dim3 blk(32, 8), grd((g.L + 31) / 32, (g.M + 7) / 8, g.N), col(32, kBzWarps), cols(grd.x, g.M);
    k_update_bxy<T><<<grd, blk, 0, st>>>(g, f, ax, dtb, err);
    k_update_bz<T><<<cols, col, 0, st>>>(g, f.bx, f.by, f.bz, ax, err);
}


template <typename T>
__global__ void __launch_bounds__(fs3::NT, sizeof(T) == 4 ? 2 : 1)
    k_sweep(const __grid_constant__ SweepMaps maps, Geom g, const T *__restrict__ tin, T *__restrict__ tout,
            Axis<T> ax, StepScalars<T> sdir, const StepScalars<T> *__restrict__ table,
            StepGate gate, SourceTable<T> src, ZChunks zc, int cbase, int rev, int *err) {
    StepScalars<T> s = sdir;
    if (gate.base) {
        const long st = gate.step();
        if (st >= gate.nsteps) return;
        s = table[st];
    }
    const int c = cbase + (int)(rev ? gridDim.z - 1 - blockIdx.z : blockIdx.z);
    sweep_cta<T, false, 2>(maps, g, tin, tout, ax, s, src, zc, blockIdx.x, blockIdx.y, c, err);
}

// every slot of a batch in one launch: block b belongs to the slot whose range of idx holds it
template <typename T>
__global__ void __launch_bounds__(fs3::NT, sizeof(T) == 4 ? 2 : 1)
    k_sweep_batched(const SweepSlot<T> *__restrict__ slots, const __grid_constant__ BatchIndex idx, int s, int c0, Piece piece) {
    const int q = idx.slot_of(blockIdx.x);
    const SweepSlot<T> &d = slots[q];
    const long st = (long)*d.step_base + s;
    if (st >= d.nsteps) return;
    const int lb = blockIdx.x - idx.off[q];
    const int bx = lb % d.tiles_x, rest = lb / d.tiles_x, by = rest % d.tiles_y, c = c0 + rest / d.tiles_y;
    sweep_cta<T>(d.maps, d.g, d.tin, d.tout, d.ax, d.table[st], d.src, d.zc, bx, by, c, d.err, AirAfterKernel(), piece, d.bz_new);
}

template <typename T>
void launch_fused_sweep(const SweepMaps &maps, const Geom &g, const T *tin, T *tout, const Axis<T> &ax,
                        StepScalars<T> s, const StepScalars<T> *table, StepGate gate,
                        const SourceTable<T> &src, const ZChunks &zc, int c0, int c1, bool rev, int *err,
                        cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sweep_tiles_x(g.L), sweep_tiles_y(g.M, zc.rows), c1 - c0);
    cfg.blockDim = dim3(fs3::NT);
    cfg.dynamicSmemBytes = fs3::smem_bytes_n<T>(g.N);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_sweep<T>, maps, g, tin, tout, ax, s, table, gate, src, zc, c0, rev ? 1 : 0, err);
}

// more than half of an SM's shared memory: one CTA per SM
constexpr size_t kAloneBytes = 116 << 10;
template <typename T>
void launch_sweep_batched(const SweepSlot<T> *slots, const BatchIndex &idx, int s, int c0, int N_max, cudaStream_t st,
                          Piece piece, bool spread) {
    if (idx.total() == 0) return;
    const size_t need = fs3::smem_bytes_n<T>(N_max);
    k_sweep_batched<T><<<idx.total(), fs3::NT, spread && need < kAloneBytes ? kAloneBytes : need, st>>>(slots, idx, s, c0, piece);
}
int sweep_tiles_x(int L) { return (L + fs3::TX - 1) / fs3::TX; }
int sweep_tiles_y(int M, int rows) { return (M + rows - 1) / rows; }

template <typename T> cudaError_t sweep_configure(int N) {
    const size_t sm = fs3::smem_bytes_n<T>(N);
    const cudaError_t e = allow_shared(k_sweep<T>, sm);
    return e != cudaSuccess ? e : allow_shared(k_sweep_batched<T>, sm);
}
template <typename T> size_t sweep_smem_bytes(int N) { return fs3::smem_bytes_n<T>(N); }
template <typename T> int sweep_blocks_per_sm(int N) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_sweep<T>, fs3::NT, fs3::smem_bytes_n<T>(N)) != cudaSuccess)
        return 1;
    return nb > 0 ? nb : 1;
}
int sweep_box_x() { return fs3::BXW; }
int sweep_box_y() { return fs3::BYH; }
int sweep_tile_x() { return fs3::TX; }
int sweep_table_planes() { return fs3::ZWIN - 3; }

// Materialise Bz = P + O_c in place; the caller clears the chunk totals.  Bound by latency on the grids that a host
// steps stage by stage: one thread per column and chunk, eight planes in flight (64 x 64 x 48 with six chunks:
// 20 us as one thread per column through all planes, 8.3 us cold).
template <typename T>
__global__ void k_bz_consolidate(Geom g, T *__restrict__ bz, const T *__restrict__ tot, ZChunks zc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, c = blockIdx.z;
    if (i > g.L || j > g.M) return;
    const int XP = g.XP, PS = (int)g.PS, plane = (g.M + 2) * XP;
    const int col = (j + 1) * XP + (i + 4);
    T o = T(0);
    for (int q = zc.n - 1; q > c; q--) o += tot[q * plane + col];
    T *p = bz + col + (zc.plane(c) + 1) * PS;
#pragma unroll 8
    for (int k = zc.plane(c + 1) - zc.plane(c); k > 0; k--, p += PS) *p += o;
}

// the last chunk has nothing below it
template <typename T> void launch_bz_consolidate(const Geom &g, T *bz, T *tot, const ZChunks &zc, cudaStream_t st) {
    if (zc.n <= 1) return;
    dim3 blk(32, 4), grd((g.L + 1 + 31) / 32, (g.M + 1 + 3) / 4, zc.n - 1);
    k_bz_consolidate<T><<<grd, blk, 0, st>>>(g, bz, tot, zc);
    cudaMemsetAsync(tot, 0, (size_t)zc.n * g.PS * sizeof(T), st);
}

// ------------------------------------------------------------------ exchange with the host

// One block per row, neighbouring threads on neighbouring cells.  (128 x 128 x 96, one component to the host's
// array: 0.80 ms with the whole volume copied and converted on the host, 0.33 ms.)
template <typename T>
__global__ void k_crop(Geom g, const T *__restrict__ v, double *__restrict__ out, int nx, int ny, int k) {
    const T *src = v + g.at(0, blockIdx.x, k + (int)blockIdx.y);
    double *dst = out + ((size_t)blockIdx.y * ny + blockIdx.x) * nx;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) dst[i] = (double)src[i];
}
template <typename T>
__global__ void k_place(Geom g, const double *__restrict__ in, T *__restrict__ v, int nx, int ny, int k) {
    const double *src = in + ((size_t)blockIdx.y * ny + blockIdx.x) * nx;
    T *dst = v + g.at(0, blockIdx.x, k + (int)blockIdx.y);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) dst[i] = (T)src[i];
}
template <typename T> void launch_crop(const Geom &g, const T *v, double *out, int nx, int ny, int k, int n, cudaStream_t st) {
    k_crop<T><<<dim3(ny, n), 128, 0, st>>>(g, v, out, nx, ny, k);
}
template <typename T> void launch_place(const Geom &g, const double *in, T *v, int nx, int ny, int k, int n, cudaStream_t st) {
    k_place<T><<<dim3(ny, n), 128, 0, st>>>(g, in, v, nx, ny, k);
}

#define INST(T)                                                                                                    \
    template void launch_crop<T>(const Geom &, const T *, double *, int, int, int, int, cudaStream_t);             \
    template void launch_place<T>(const Geom &, const double *, T *, int, int, int, int, cudaStream_t);            \
    template void launch_update_e<T>(const Geom &, FieldSet<T>, const T *, const Axis<T> &, StepScalars<T>,        \
                                     const SourceTable<T> &, int *, cudaStream_t);                                 \
    template void launch_bderivate<T>(const Geom &, FieldSet<T>, const Axis<T> &, T, int *, cudaStream_t);         \
    template void launch_fused_sweep<T>(const SweepMaps &, const Geom &, const T *, T *,                          \
                                        const Axis<T> &, StepScalars<T>, const StepScalars<T> *, StepGate,         \
                                        const SourceTable<T> &, const ZChunks &, int, int, bool, int *, cudaStream_t,  \
                                        bool);                                                                     \
    template cudaError_t sweep_configure<T>(int);                                                                  \
    template size_t sweep_smem_bytes<T>(int);                                                                      \
    template int sweep_blocks_per_sm<T>(int);                                                                      \
    template void launch_bz_consolidate<T>(const Geom &, T *, T *, const ZChunks &, cudaStream_t);             \
    template void launch_sweep_batched<T>(const SweepSlot<T> *, const BatchIndex &, int, int, int, cudaStream_t, Piece, bool);
INST(float)
INST(double)
#undef INST

}  // namespace tcsem
