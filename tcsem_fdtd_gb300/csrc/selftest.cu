// The sweep with copies that do not arrive: what its bounded waits do then, without a GPU fault.
#include "selftest.cuh"
#include "sweep.cuh"

namespace tcsem {

namespace {
// every wait of the march gives up at once; counts the tiles that loaded their last stage (plane 0) all the same
struct NoPatience {
    static constexpr int kPolls = 0;
    int *loaded;
    __device__ __forceinline__ void operator()() const { atomicAdd(loaded, 1); }
};
}  // namespace

template <typename T>
__global__ void __launch_bounds__(fs3::NT, sizeof(T) == 4 ? 2 : 1)
    k_sweep_lost(const __grid_constant__ SweepMaps maps, Geom g, const T *__restrict__ tin, T *__restrict__ tout, Axis<T> ax,
                 StepScalars<T> s, SourceTable<T> src, ZChunks zc, int *err, int *loaded) {
    sweep_cta<T, false, 2, true>(maps, g, tin, tout, ax, s, src, zc, blockIdx.x, blockIdx.y, 0, err, NoPatience{loaded});
}

template <typename T>
cudaError_t launch_sweep_lost(const SweepMaps &maps, const Geom &g, const T *tin, T *tout, const Axis<T> &ax, StepScalars<T> s,
                              const SourceTable<T> &src, int rows, int *err, int *loaded, cudaStream_t st) {
    ZChunks zc{1, rows, {0, g.N}};
    const size_t sm = sweep_smem_bytes<T>(g.N);
    const cudaError_t e = allow_shared(k_sweep_lost<T>, sm);
    if (e != cudaSuccess) return e;
    k_sweep_lost<T><<<dim3(sweep_tiles_x(g.L), sweep_tiles_y(g.M, rows)), fs3::NT, sm, st>>>(maps, g, tin, tout, ax, s, src,
                                                                                           zc, err, loaded);
    return cudaGetLastError();
}

#define INST(T)                                                                                                     \
    template cudaError_t launch_sweep_lost<T>(const SweepMaps &, const Geom &, const T *, T *, const Axis<T> &,      \
                                              StepScalars<T>, const SourceTable<T> &, int, int *, int *, cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace tcsem
