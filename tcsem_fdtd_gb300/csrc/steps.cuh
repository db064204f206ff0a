// The time loop of one survey as one cooperative launch for many steps (see steps.cu).
#pragma once
#include "kernels.cuh"
#include "rx.cuh"
#include "steps_boundary.cuh"

namespace tcsem {

// control words, each on a line of its own: arrivals at the end of a step (all CTAs), after each of the
// boundary's three products (its CTAs; the last one has written the air plane), and the abort flag
enum { kStArrive = 0, kStProduct = 32, kStAir = kStProduct + 2 * 32, kStAbort = kStAir + 32, kStWords = kStAbort + 32 };

template <typename T> struct StepsArgs {
    SweepMaps maps[2];  // of the sweep that reads each field set
    FieldSet<T> f[2];
    T *tot[2];
    Geom g;
    Axis<T> ax;
    const StepScalars<T> *table;
    SourceTable<T> src;
    ZChunks zc;
    Products<T> pd;
    RxDev<T> rd;
    int *ctl;
    int *err;
    int tiles_x, tiles;   // sweep CTAs: tiles x (march + own), then nbnd boundary CTAs, then nrx receiver CTAs
    int nsweep, nbnd, nrx;
    int march, own;       // CTAs of a tile that take the lower chunks in turn; 1: another one takes the top chunk
    int nfwd, ncol, ninv; // tiles of the first product, frequencies per CTA of the second, tiles of the third
    long step0;           // first step of this launch
    int n;                // steps of this launch
    int cur;              // field set that holds the state before the first step
    long long wait_ns;    // a wait for another CTA gives up after this long
};

template <typename T> size_t steps_smem(const Products<T> &d, int N);
template <typename T> cudaError_t steps_configure(size_t smem);
template <typename T> int steps_blocks(size_t smem);  // co-resident CTAs on the device
template <typename T> cudaError_t launch_steps(const StepsArgs<T> &a, size_t smem, cudaStream_t st);

}  // namespace tcsem
