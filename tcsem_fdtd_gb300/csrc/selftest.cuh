// Kernels of the self-tests (selftest.cu).
#pragma once
#include "kernels.cuh"

namespace tcsem {

// One sweep in whole columns whose waits for a copy give up at once; *loaded += the tiles that went on to load plane 0.
// Columns have more planes than a march loads ahead.
template <typename T>
cudaError_t launch_sweep_lost(const SweepMaps &maps, const Geom &g, const T *tin, T *tout, const Axis<T> &ax, StepScalars<T> s,
                              const SourceTable<T> &src, int rows, int *err, int *loaded, cudaStream_t st);

}  // namespace tcsem
