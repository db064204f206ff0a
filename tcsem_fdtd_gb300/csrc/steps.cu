// The time loop of one survey as one cooperative launch for many steps.
//
// On small grids a step is a chain of short kernels -- the four stages of the boundary and the sweep's top
// plane, each a few microseconds of which most is launch, start-up and the wait for the last block of the
// kernel before -- beside a sweep that is done much earlier.  Here every CTA is resident for the whole launch
// and has one role: a tile of one z-chunk of the sweep, a share of the boundary, or the receivers.
//   * The boundary is three products with constant matrices (steps_boundary.cuh), with the next one's table
//     on its way into shared memory while its CTAs wait for the one before.
//   * The sweep keeps the chunks of the captured graph, so that the fields differ by the boundary's rounding
//     alone (another chunk layout changes the last bits of Bz: early in a marine survey, where Bx at the
//     surface is a cancelling sum, by 3e-5 of Bx).  Only the top chunk's one plane needs the air plane: its CTAs
//     wait for the boundary there (AirFlag).
//   * One barrier of all CTAs ends a step.  The receivers of step s run beside step s + 1, which only
//     reads the field set step s wrote.
// What bounds it: the chain boundary -> top plane -> barrier, and where a chunk is deep the march of its planes
// (0.8 us each with one CTA on an SM).  64 x 64 x 48 with a 260 x 260 plane, us per step: about 3 from the barrier to
// the columns of F, 4 through y, 4 to the air plane, 4.5 for the top plane, 1.3 for the barrier; 18.9 in all, 25.8
// as a captured graph, whose four boundary kernels alone take 20.7.
// Every wait is bounded in time: a CTA that gives up sets the abort flag and the error word, and every
// CTA leaves at its next wait.
//
// Memory ordering.  A CTA's writes are ordered by a CTA barrier before thread 0's release; a waiting CTA's
// thread 0 acquires the count and releases its threads with a CTA barrier.  Values another CTA wrote are
// read from L2 (F, V, chunk totals, Bz) or by bulk-tensor copies, which the proxy fences on both sides order
// (the sweep's own bulk-tensor stores have completed before its CTA arrives).
#include "rx_body.cuh"
#include "steps.cuh"
#include "sweep.cuh"

namespace tcsem {

namespace {

template <typename T> struct Sync {
    const StepsArgs<T> &a;
    // thread 0: until *word >= target; false (abort flag and error word set) if it gave up
    __device__ __forceinline__ bool until(const int *word, int target) const {
        if (ld_acquire(word) >= target) return true;
        const unsigned long long t0 = globaltimer_ns();
        for (int polls = 1; ld_acquire(word) < target; polls++)
            if ((polls & 63) == 0 &&
                (ld_acquire(a.ctl + kStAbort) || globaltimer_ns() - t0 > (unsigned long long)a.wait_ns)) {
                atomicExch(a.ctl + kStAbort, 1);
                atomicExch(a.err, 1);
                return false;
            }
        return true;
    }
    // all threads, after a CTA barrier behind the writes (ASYNC: read by bulk-tensor copies): count this CTA in
    template <bool ASYNC> __device__ __forceinline__ void arrive(int *word) const {
        if (threadIdx.x != 0) return;
        if (ASYNC) fence_proxy_async_global();
        red_release(word, 1);
    }
    // all threads; false: the launch was given up
    template <bool ASYNC> __device__ __forceinline__ bool wait(const int *word, int target) const {
        bool ok = true;
        if (threadIdx.x == 0) {
            ok = until(word, target);
            if (ASYNC) fence_proxy_async_global();
        }
        return !__syncthreads_or(!ok);
    }
    // all threads, a copy did not arrive (err is set): the other CTAs leave at their next wait
    __device__ __forceinline__ void give_up() const {
        if (threadIdx.x == 0) atomicExch(a.ctl + kStAbort, 1);
    }
    // all threads: the end of step s of this launch
    __device__ __forceinline__ bool step_end(int s) const {
        arrive<true>(a.ctl + kStArrive);
        return wait<true>(a.ctl + kStArrive, (s + 1) * (int)gridDim.x);
    }
};

// the sweep's copying thread before the air plane; when it gives up the sweep finishes on the old
// plane and its CTA leaves at the next wait
template <typename T> struct AirFlag {
    static constexpr int kPolls = AirAfterKernel::kPolls;
    Sync<T> s;
    int target;
    __device__ __forceinline__ void operator()() const {
        s.until(s.a.ctl + kStAir, target);
        fence_proxy_async_global();
    }
};
// a product before it reads the one before (word; nothing to wait for without one); ok: the CTA goes on
template <typename T> struct After {
    Sync<T> s;
    const int *word;
    int target;
    bool *ok;
    __device__ __forceinline__ void operator()() const {
        if (word) *ok = s.template wait<false>(word, target) && *ok;
    }
    // a copy did not arrive: the CTA leaves at the end of the step, the others at a wait
    __device__ __forceinline__ void lost() const {
        *ok = false;
        s.give_up();
    }
};

}  // namespace

template <typename T>
__global__ void __launch_bounds__(fs3::NT, 2) k_steps(const __grid_constant__ StepsArgs<T> a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    static_assert(fs3::NT == 32 * products::NWARP, "every warp sums a share of the products");
    const Sync<T> sy{a};
    const int cta = blockIdx.x;
    if (cta < a.nsweep) {
        const int tile = cta % a.tiles, r = cta / a.tiles;
        for (int s = 0; s < a.n; s++) {
            const int b = (a.cur + s) & 1;  // the field set this step reads
            // lower chunks r + 1, r + 1 + march, ..., then the top one
            for (int c = r < a.march ? r + 1 : a.zc.n;; c += a.march) {
                const bool top = c >= a.zc.n;
                if (top && r != a.march - 1 + a.own) break;
                const bool ok = sweep_cta<T, true, fs3::ring<T>(), false>(a.maps[b], a.g, a.tot[b], a.tot[b ^ 1], a.ax, a.table[a.step0 + s], a.src,
                                                   a.zc, tile % a.tiles_x, tile / a.tiles_x, top ? 0 : c, a.err,
                                                   AirFlag<T>{sy, (s + 1) * a.nbnd});
                if (!ok) return sy.give_up();
                __syncthreads();
                if (threadIdx.x == 0) {
                    uint64_t *ring = reinterpret_cast<uint64_t *>(smem_raw + fs3::bars_offset<T>());
                    for (int q = 0; q < fs3::ring<T>(); q++) mbar_inval(ring + q);
                }
                if (top) break;
                __syncthreads();
            }
            if (!sy.step_end(s)) return;
        }
    } else if (cta < a.nsweep + a.nbnd) {
        const int own = cta - a.nsweep;
        int *word = a.ctl + kStProduct;
        for (int s = 0; s < a.n; s++) {
            const int b = (a.cur + s) & 1, target = (s + 1) * a.nbnd;
            bool ok = true;
            for (int i = own; i < a.nfwd; i += a.nbnd)
                products::forward_x<T>(a.pd, a.f[b].bz, a.tot[b], a.zc.n, a.g, i, After<T>{sy, nullptr, 0, &ok});
            sy.template arrive<false>(word);
            const int *first = word;
            for (int i = own; i * a.ncol * 2 < a.pd.nc; i += a.nbnd, first = nullptr) {
                if (a.ncol == 1) products::through_y<T, 1>(a.pd, i, After<T>{sy, first, target, &ok});
                else products::through_y<T, 2>(a.pd, i, After<T>{sy, first, target, &ok});
            }
            sy.template arrive<false>(word + 32);
            first = word + 32;
            for (int i = own; i < a.ninv; i += a.nbnd, first = nullptr)
                products::inverse_x<T>(a.pd, a.f[b].bx, a.f[b].by, a.g, i, After<T>{sy, first, target, &ok});
            sy.template arrive<true>(a.ctl + kStAir);
            if (!ok || !sy.step_end(s)) return;
        }
    } else {
        for (int s = 0; s <= a.n; s++) {
            if (s > 0) {  // the receivers of the step before, on the set it wrote
                const int b = (a.cur + s) & 1;
                const RxAction act = step_action(a.rd, a.step0 + s - 1);
                if (act.e_slot >= 0 || act.b_slot >= 0)
                    for (int i = (cta - a.nsweep - a.nbnd) * blockDim.x + threadIdx.x; i < a.rd.NComp * a.rd.nr;
                         i += a.nrx * blockDim.x)
                        rx_thread(a.rd, a.f[b], a.tot[b], a.zc, a.g, act, i);
            }
            __syncthreads();
            if (s == a.n || !sy.step_end(s)) return;
        }
    }
}

template <typename T> size_t steps_smem(const Products<T> &d, int N) {
    const size_t need[4] = {fs3::smem_bytes_n<T>(N), products::tile_layout<T>(d.L, kFwdJ).total, products::tile_layout<T>(d.nc, kInvJ).total,
                            products::spec_layout(d, 2, fs3::NT).total};
    size_t m = 0;
    for (size_t v : need) m = v > m ? v : m;
    return m;
}

template <typename T> cudaError_t steps_configure(size_t smem) {
    return allow_shared(k_steps<T>, smem);
}

template <typename T> int steps_blocks(size_t smem) {
    int nb = 0, dev = 0, sms = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_steps<T>, fs3::NT, smem) != cudaSuccess)
        return 0;
    return nb * sms;
}

template <typename T> cudaError_t launch_steps(const StepsArgs<T> &a, size_t smem, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(a.ctl, 0, kStWords * sizeof(int), st);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.nsweep + a.nbnd + a.nrx);
    cfg.blockDim = dim3(fs3::NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // every CTA resident: they wait for one another
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_steps<T>, a);
}

// ------------------------------------------------------------------ the products' tables

// cosine and sine of pi r / L1, r < 2 L1, then of pi r / M1, r < 2 M1
__global__ void k_trig(double2 *t, int L1, int M1) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, y = r >= 2 * L1;
    if (r >= 2 * (L1 + M1)) return;
    sincospi((double)(r - y * 2 * L1) / (double)(y ? M1 : L1), &t[r].y, &t[r].x);
}
// r modulo 2 n, for any r
__device__ __forceinline__ int turn(int r, int n) {
    r %= 2 * n;
    return r < 0 ? r + 2 * n : r;
}
// element (k, n) of a table of K rows
template <typename T> __device__ __forceinline__ T &entry(T *tab, int K, int k, int n) {
    return tab[((size_t)(n / kTabN) * K + k) * kTabN + n % kTabN];
}
// sum of the weights of grid cell i times the functions of angle a0 + a p (modulo 2 n) at their points p
__device__ __forceinline__ double2 through(const LineRemap &m, int i, const double2 *t, int a0, int a, int n) {
    double2 s{0, 0};
    const int q1 = m.off[i + 1];
    int q = m.off[i], r = turn(a0 + a * m.lo[i], n);
    a = turn(a, n);
    for (; q < q1; q++) {
        const double w = m.w[q];
        const double2 v = t[r];
        s.x += w * v.x;
        s.y += w * v.y;
        r += a;
        if (r >= 2 * n) r -= 2 * n;
    }
    return s;
}

template <typename T> __global__ void k_table_a(Products<T> d, T *A, int L1, LineRemap px, const double2 *t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, kx = blockIdx.y;
    if (i >= d.L) return;
    const double2 v = through(px, i, t, 0, 2 * kx, L1);
    entry(A, d.L, i, 2 * kx) = (T)v.x;
    entry(A, d.L, i, 2 * kx + 1) = (T)-v.y;
}

// Functions of y: the cosine and the sine of ky at the angle pi ky (2m - M1 + 1) / M1 of point m, measured from
// the middle of the line (the sine of ky = 0 and, for an even M1, the cosine of ky = M1/2 are zero).
template <typename T> __global__ void k_table_w(Products<T> d, T *Wc, T *Ws, LineRemap py, const double2 *t) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, ky = blockIdx.y;
    if (j >= d.Mh) return;
    double2 v = through(py, j, t, ky * (1 - d.M1), 2 * ky, d.M1);
    if (d.fold) {  // the mean of the row and its mirror image
        const double2 m = through(py, d.M - 1 - j, t, ky * (1 - d.M1), 2 * ky, d.M1);
        v = {0.5 * (v.x + m.x), 0.5 * (v.y - m.y)};
    }
    entry(Wc, d.Mh, j, ky) = (T)v.x;
    entry(Ws, d.Mh, j, ky) = (T)v.y;
}

template <typename T>
__global__ void k_table_c(Products<T> d, T *Cc, T *Cs, int rows, int R, const int *__restrict__ at,
                          const double *__restrict__ wt, const double2 *t) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, ky = blockIdx.y;
    if (r >= R) return;
    auto value = [&](int q) {
        const double2 v0 = t[turn(ky * (2 * at[q] - d.M1 + 1), d.M1)], v1 = t[turn(ky * (2 * at[q] - d.M1 + 3), d.M1)];
        return double2{(1.0 - wt[q]) * v0.x + wt[q] * v1.x, (1.0 - wt[q]) * v0.y + wt[q] * v1.y};
    };
    double2 v = value(r);
    if (d.fold) {
        const double2 m = value(rows - 1 - r);
        v = {0.5 * (v.x + m.x), 0.5 * (v.y - m.y)};
    }
    entry(Cc, d.K, ky, r) = (T)v.x;
    entry(Cs, d.K, ky, r) = (T)v.y;
}

template <typename T>
__global__ void k_table_d(Products<T> d, T *D, int n, int L1, const int *__restrict__ at, const double *__restrict__ wt,
                          const double2 *t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, kx = blockIdx.y;
    if (i >= n) return;
    const double2 v0 = t[turn(2 * kx * at[i], L1)], v1 = t[turn(2 * kx * (at[i] + 1), L1)];
    // the two self-conjugate frequencies count once, with their real parts alone
    const bool self = kx == 0 || 2 * kx == L1;
    const double f = self ? 1.0 : 2.0;
    entry(D, d.nc, 2 * kx, i) = (T)(f * ((1.0 - wt[i]) * v0.x + wt[i] * v1.x));
    entry(D, d.nc, 2 * kx + 1, i) = self ? T(0) : (T)(-f * ((1.0 - wt[i]) * v0.y + wt[i] * v1.y));
}

template <typename T>
cudaError_t products_tables(const Products<T> &d, int L1, const LineRemap &px, const LineRemap &py,
                            const LineSampling &s, double2 *trig, cudaStream_t st) {
    const int H = d.nc / 2, t = 64;
    auto grid = [&](int n, int k) { return dim3((n + t - 1) / t, k); };
    auto out = [](const T *p) { return const_cast<T *>(p); };
    const double2 *tx = trig, *ty = trig + 2 * L1;
    k_trig<<<(2 * (L1 + d.M1) + t - 1) / t, t, 0, st>>>(trig, L1, d.M1);
    k_table_a<T><<<grid(d.L, H), t, 0, st>>>(d, out(d.A), L1, px, tx);
    k_table_w<T><<<grid(d.Mh, d.K), t, 0, st>>>(d, out(d.Wc), out(d.Ws), py, ty);
    k_table_c<T><<<grid(d.Rx, d.K), t, 0, st>>>(d, out(d.Cxc), out(d.Cxs), d.M, d.Rx, s.bx_j, s.bx_v, ty);
    k_table_c<T><<<grid(d.Ry, d.K), t, 0, st>>>(d, out(d.Cyc), out(d.Cys), d.M + 1, d.Ry, s.by_j, s.by_v, ty);
    k_table_d<T><<<grid(d.L + 1, H), t, 0, st>>>(d, out(d.Dx), d.L + 1, L1, s.bx_i, s.bx_u, tx);
    k_table_d<T><<<grid(d.L, H), t, 0, st>>>(d, out(d.Dy), d.L, L1, s.by_i, s.by_u, tx);
    return cudaGetLastError();
}

#define INST(T)                                                                                              \
    template size_t steps_smem<T>(const Products<T> &, int);                                                \
    template cudaError_t steps_configure<T>(size_t);                                                        \
    template int steps_blocks<T>(size_t);                                                                   \
    template cudaError_t launch_steps<T>(const StepsArgs<T> &, size_t, cudaStream_t);                       \
    template cudaError_t products_tables<T>(const Products<T> &, int, const LineRemap &, const LineRemap &,  \
                                            const LineSampling &, double2 *, cudaStream_t);
INST(float)
#undef INST

}  // namespace tcsem
