// The boundary step as three products with constant matrices, for the launches that keep every CTA
// resident (steps.cu).
//
// The chain Bz plane -> spline remap -> 2-D transform -> continuation filters -> inverse transform ->
// bilinear sampling (UpContinuation_gpu.cu:166-274) is linear, and everything but the filters is
// separable.  Composing remap and transform (sampling and inverse transform) of each axis into one
// constant matrix leaves
//     F = A Bz^T             L      -> 2 H columns (real and imaginary parts of the kept x-frequencies)
//     V = C (g (W F))        M      -> M1 cosine and sine parts in y, filtered -> the M rows of Bx and
//                                      the M + 1 rows of By; every column by itself
//     out = V D              2 H    -> the L + 1 (L) points of each row
// The y line is symmetric about its middle, so even and odd parts use half of W and C.  More operations
// than the transforms (boundary_body.cuh), but three phases without a barrier in their sums in place of
// a chain of some thirty barrier-separated stages.
#pragma once
#include "async.cuh"
#include "check.cuh"
#include "kernels.cuh"
#include "pair.cuh"

namespace tcsem {

// "Columns" are the 2 H real and imaginary parts, column 2 kx the real and 2 kx + 1 the imaginary one.
// A table of K rows and n columns is stored in blocks of 32 columns, [n / 32][K][32], so that the part
// of it a tile needs is contiguous.
template <typename T> struct Products {
    int fold;       // the y line is symmetric about its middle: rows j and M-1-j share their weights
    int L, M, M1;   // grid rows and columns; length of the transform line in y
    int nc;         // 2 H columns
    int Mh;         // summed rows of the forward y product: ceil(M / 2) folded, else M
    int Rx, Ry;     // output rows of the inverse y product: ceil(M / 2), ceil((M + 1) / 2) folded, else M, M + 1
    int K;          // frequencies ky = 0 .. M1/2 of y, a cosine and a sine function each
    int ldF, ldV, ldG;   // row pitches
    int oFo;             // F: the even parts at 0, the odd parts here (0 when not folded)
    int oVy;             // V: the M rows of Bx at 0, the M + 1 rows of By here
    const T *A;          // K = L,  n = nc: grid row of Bz to the columns (spline remap and transform in x)
    const T *Wc, *Ws;    // K = Mh, n = K: y remap and transform, cosine and sine parts
    const T *gx, *gy;    // [H][ldG]: continuation filters for ky = 0 .. M1/2, with the pair factor and 1/(L1 M1)
    const T *Cxc, *Cxs;  // K = K, n = Rx: inverse in y and sampling to the rows of Bx
    const T *Cyc, *Cys;  // ... n = Ry: to the rows of By
    const T *Dx, *Dy;    // K = nc, n = L + 1 (L): inverse in x and sampling to the points of Bx (By)
    T *F;                // [nc][ldF]
    T *V;                // [nc][ldV]
    int *err;
};
// the arrays in the order A Wc Ws gx gy Cxc Cxs Cyc Cys Dx Dy F V
constexpr int kProductArrays = 13;

constexpr int kTabN = 32;    // columns of a table block and of an output tile
constexpr int kFwdJ = 16;    // rows of an output tile of the first product ...
constexpr int kInvJ = 8;     // ... and of the third, whose sums are the longest

__host__ __device__ inline int up(int n, int m) { return (n + m - 1) / m; }

// sizes and pitches (pointers unset), elements of each array, and the arrays' pointers
template <typename T> inline void products_shape(Products<T> &d, int L, int M, int L1, int M1, bool fold) {
    d = Products<T>{};
    d.fold = fold;
    d.L = L; d.M = M; d.M1 = M1;
    d.nc = 2 * (L1 / 2 + 1);
    d.Mh = fold ? (M + 1) / 2 : M;
    d.Rx = fold ? (M + 1) / 2 : M;
    d.Ry = fold ? (M + 2) / 2 : M + 1;
    d.K = M1 / 2 + 1;
    d.ldG = up(d.K, 4) * 4;
    d.oFo = fold ? up(d.Mh, 4) * 4 : 0;
    d.ldF = fold ? 2 * d.oFo : up(d.Mh, 4) * 4;
    d.oVy = up(M, kInvJ) * kInvJ;  // both lists in whole tiles
    d.ldV = d.oVy + up(M + 1, kInvJ) * kInvJ;
}
template <typename T> inline void products_sizes(const Products<T> &d, size_t n[kProductArrays]) {
    auto table = [](int K, int cols) { return (size_t)K * up(cols, kTabN) * kTabN; };
    const size_t H = d.nc / 2;
    n[0] = table(d.L, d.nc);
    n[1] = n[2] = table(d.Mh, d.K);
    n[3] = n[4] = H * d.ldG;
    n[5] = n[6] = table(d.K, d.Rx);
    n[7] = n[8] = table(d.K, d.Ry);
    n[9] = table(d.nc, d.L + 1);
    n[10] = table(d.nc, d.L);
    n[11] = (size_t)d.nc * d.ldF;
    n[12] = (size_t)d.nc * d.ldV;
}
template <typename T> inline void products_bind(Products<T> &d, T *const p[kProductArrays]) {
    d.A = p[0]; d.Wc = p[1]; d.Ws = p[2]; d.gx = p[3]; d.gy = p[4];
    d.Cxc = p[5]; d.Cxs = p[6]; d.Cyc = p[7]; d.Cys = p[8]; d.Dx = p[9]; d.Dy = p[10];
    d.F = p[11]; d.V = p[12];
}
template <typename T> inline int tiles_fwd(const Products<T> &d) {
    return up(d.nc, kTabN) * (d.fold ? up(d.Mh, kFwdJ / 2) : up(d.M, kFwdJ));
}
template <typename T> inline int tiles_inv(const Products<T> &d) {
    return up(d.L + 1, kTabN) * up(d.M, kInvJ) + up(d.L, kTabN) * up(d.M + 1, kInvJ);
}

// The tables A, W, C, D are filled on the device, in 64 bits, from the remaps of both axes (weights of grid cell
// i at the points lo[i] ... of the transform line: w[off[i]] .. w[off[i + 1]]) and the two-point sampling of the
// lines (first point and second point's weight); trig takes 2 (L1 + M1) cosine and sine pairs.
struct LineRemap {
    const int *off, *lo;
    const double *w;
};
struct LineSampling {
    const int *bx_i, *bx_j, *by_i, *by_j;      // first point on the transform line: Bx at L+1, M; By at L, M+1
    const double *bx_u, *bx_v, *by_u, *by_v;   // weight of the second point
};
template <typename T>
cudaError_t products_tables(const Products<T> &d, int L1, const LineRemap &px, const LineRemap &py,
                            const LineSampling &s, double2 *trig, cudaStream_t st);

namespace products {

template <typename T> struct alignas(16) Vec4 { T v[4]; };

// four neighbouring values another CTA of this launch may have written (L2), or constant ones
template <bool FRESH> __device__ __forceinline__ Vec4<float> ld4(const float *p) {
    const float4 *q = reinterpret_cast<const float4 *>(p);
    const float4 r = FRESH ? __ldcg(q) : __ldg(q);
    return {{r.x, r.y, r.z, r.w}};
}

// Rounding.  A warp's chain of multiply-adds is put aside after 16 rows, and the ten warps' (the second
// product's) shares are added as a tree.  Relative error of the air plane, geometric mean over 16 grids
// and three fields each: transforms in FP32 1.67e-7; whole chains, shares added one after the other 1.75e-7; as a
// tree 1.60e-7; put aside too 1.54e-7 (0.1 to 0.5 us per step).  Two chains side by side in a warp take 1 to 1.6 us.
// Of whole runs the errors are the same: traces of 22 surveys (470 to 1860 steps) against FP64, this form over the
// transforms, 0.23 to 1.9 in single ones; geometric mean 0.98 of the rms error and 1.00 of the largest.

// ---- first and third product: Out[j][n] = sum_k X[j][k] Tab[k][n], one tile of J j by 32 n per CTA.
// The table's block streams through shared memory by bulk copies that are issued before the CTA waits for
// the phase before; each of the 10 warps sums a share of k for the whole tile (J/4 j by 4 n per lane) and
// the shares are added in a fixed order.
constexpr int NWARP = 10;
constexpr int SH = 8;                   // rows of a chunk per warp
constexpr int CHUNK = NWARP * SH;       // rows of the table per bulk copy
constexpr int NSLOT = 6;                // copies in flight; longer sums reuse the slots
constexpr int FLUSH = 2;                // chunks after which a warp's chains are put aside
// pitch of X's rows: whole 16-byte pieces, neighbouring rows on different banks
__host__ __device__ inline int x_pitch(int K) { return (K + 3) / 8 * 8 + 4; }
template <typename T> struct TileLayout {
    size_t x, slots, aside, total;
    int nchunk, nslot;
};
template <typename T> __host__ __device__ inline TileLayout<T> tile_layout(int K, int J) {
    TileLayout<T> l;
    l.nchunk = up(K, CHUNK);
    l.nslot = l.nchunk < NSLOT ? l.nchunk : NSLOT;
    l.x = 64;
    l.slots = l.x + rnd16((size_t)J * x_pitch(K) * sizeof(T));
    const size_t s = (size_t)l.nslot * CHUNK * kTabN * sizeof(T), r = (size_t)NWARP * J * kTabN * sizeof(T);
    l.aside = l.slots + (s > r ? s : r);
    l.total = l.aside + (l.nchunk > FLUSH ? r : 0);
    return l;
}
template <typename T, int J> struct Tile {
    static constexpr int NJ = J / 4;
    TileLayout<T> l;
    int K;
    const T *tab;  // the block [K][32]
    uint64_t *bars;
    T *xs, *slots, *aside;

    __device__ __forceinline__ Tile(unsigned char *smem, int k, const T *block) : l(tile_layout<T>(k, J)), K(k), tab(block) {
        bars = reinterpret_cast<uint64_t *>(smem);
        xs = reinterpret_cast<T *>(smem + l.x);
        slots = reinterpret_cast<T *>(smem + l.slots);
        aside = reinterpret_cast<T *>(smem + l.aside);
    }
    __device__ __forceinline__ T *xrow(int j) const { return xs + (size_t)j * x_pitch(K); }
    __device__ __forceinline__ void load_chunk(int c) const {
        uint64_t *b = bars + c % l.nslot;
        const unsigned bytes = (unsigned)(min(CHUNK, K - c * CHUNK) * kTabN * sizeof(T));
        mbar_expect_tx(b, bytes);
        bulk_load(slots + (size_t)(c % l.nslot) * CHUNK * kTabN, tab + (size_t)c * CHUNK * kTabN, bytes, b);
    }
    // a barrier has to follow before run
    __device__ __forceinline__ void start() const {
        if (threadIdx.x != 0) return;
        for (int q = 0; q < l.nslot; q++) mbar_init(bars + q, 1);
        mbar_init_fence();
        async_shared_fence();  // the product before left ordinary stores where the copies land
        for (int c = 0; c < l.nslot; c++) load_chunk(c);
    }
    // all threads: the sums of this lane's share, into slots[warp][J][32]; false: a copy did not arrive
    __device__ __forceinline__ bool run(int *err) const {
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nq = lane & 7, jq = lane >> 3;
        const int pitch = x_pitch(K);
        Pair<T> acc[2][NJ];
#pragma unroll
        for (int j = 0; j < NJ; j++) acc[0][j] = acc[1][j] = dup<T>(T(0));
        // this thread's sums in a buffer of [warp][J][32]; put aside, and the sum of what was put aside
        const int own = (w * J + jq) * kTabN + 4 * nq;
        auto store = [&](T *to) {
#pragma unroll
            for (int j = 0; j < NJ; j++)
                *reinterpret_cast<Vec4<T> *>(to + own + 4 * j * kTabN) = {{acc[0][j].a, acc[0][j].b, acc[1][j].a, acc[1][j].b}};
        };
        auto add = [&]() {
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const Vec4<T> v = *reinterpret_cast<const Vec4<T> *>(aside + own + 4 * j * kTabN);
                acc[0][j] = acc[0][j] + pair<T>(v.v[0], v.v[1]);
                acc[1][j] = acc[1][j] + pair<T>(v.v[2], v.v[3]);
            }
        };
        const T *x0 = xrow(jq) + w * SH;
        bool ok = true;
        int loaded = l.nslot;  // chunks thread 0 has asked for
        for (int c = 0; c < l.nchunk; c++) {
            ok = mbar_wait_bounded(bars + c % l.nslot, (unsigned)(c / l.nslot) & 1u) && ok;
            const T *t = slots + ((size_t)(c % l.nslot) * CHUNK + w * SH) * kTabN + 4 * nq;
            const T *x = x0 + c * CHUNK;
            const int n = min(SH, K - c * CHUNK - w * SH);
            // rows of X are read four k at a time; beyond K they hold anything finite, and the table's rows are not used
            for (int k = 0; k < n; k += 4) {
                Vec4<T> xv[NJ];
#pragma unroll
                for (int j = 0; j < NJ; j++) xv[j] = *reinterpret_cast<const Vec4<T> *>(x + 4 * j * pitch + k);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (k + q < n) {
                        const Vec4<T> tv = *reinterpret_cast<const Vec4<T> *>(t + (k + q) * kTabN);
#pragma unroll
                        for (int j = 0; j < NJ; j++) {
                            const Pair<T> d = dup<T>(xv[j].v[q]);
                            acc[0][j] = fma(pair<T>(tv.v[0], tv.v[1]), d, acc[0][j]);
                            acc[1][j] = fma(pair<T>(tv.v[2], tv.v[3]), d, acc[1][j]);
                        }
                    }
                }
            }
            if (c % FLUSH == FLUSH - 1 && c + 1 < l.nchunk) {
                if (c > FLUSH) add();
                store(aside);
#pragma unroll
                for (int j = 0; j < NJ; j++) acc[0][j] = acc[1][j] = dup<T>(T(0));
            }
            if (c + l.nslot < l.nchunk) {  // the slot takes its next chunk, once the loading thread has seen it filled
                __syncthreads();
                if (threadIdx.x == 0 && ok) {
                    async_shared_fence();
                    load_chunk(loaded++);
                }
            }
        }
        if (__syncthreads_or(!ok)) {  // record it, let the copies land, leave together
            if (threadIdx.x == 0) {
                atomicExch(err, 1);
                for (int c = loaded - l.nslot; c < loaded; c++)
                    mbar_wait_bounded(bars + c % l.nslot, (unsigned)(c / l.nslot) & 1u);
            }
            __syncthreads();
            return false;
        }
        if (l.nchunk > FLUSH) add();
        store(slots);
        __syncthreads();
        return true;
    }
    template <typename V, typename Load> static __device__ __forceinline__ V tree(const Load &at) {
        static_assert(NWARP == 10, "the tree of ten shares");
        return (((at(0) + at(1)) + (at(2) + at(3))) + ((at(4) + at(5)) + (at(6) + at(7)))) + (at(8) + at(9));
    }
    __device__ __forceinline__ T sum(int j, int n) const {
        const T *red = slots + j * kTabN + n;
        return tree<T>([&](int w) { return red[w * J * kTabN]; });
    }
    __device__ __forceinline__ Vec4<T> sum4(int j, int n) const {
        const T *red = slots + j * kTabN + n;
        const Pair<T> a = tree<Pair<T>>([&](int w) { return *reinterpret_cast<const Pair<T> *>(red + w * J * kTabN); }),
                      b = tree<Pair<T>>([&](int w) { return *reinterpret_cast<const Pair<T> *>(red + w * J * kTabN + 2); });
        return {{a.a, a.b, b.a, b.b}};
    }
    // thread 0, after the CTA is done with the tile: its barriers may become other data
    __device__ __forceinline__ void retire() const {
        for (int q = 0; q < l.nslot; q++) mbar_inval(bars + q);
    }
};

// columns of every grid row, as even and odd parts in y.  Plane 0 of Bz is chunk-partial: the totals of the
// chunks below are added as it is loaded.  wait(): before the fields of the step before are read;
// wait.lost(): a copy of the table did not arrive.
template <typename T, typename Wait>
__device__ __forceinline__ void forward_x(const Products<T> &d, const T *__restrict__ bz, const T *__restrict__ tot, int nch,
                                          const Geom &g, int blk, const Wait &wait) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int nt = up(d.nc, kTabN), nb = blk % nt, n0 = nb * kTabN;
    const int rows = d.fold ? kFwdJ / 2 : kFwdJ, j0 = (blk / nt) * rows;
    const Tile<T, kFwdJ> t(smem_raw, d.L, d.A + (size_t)nb * d.L * kTabN);
    t.start();
    wait();
    const long long plane = (long long)(g.M + 2) * g.XP;
    const int nq = up(d.L, 4);
    for (int e = threadIdx.x; e < kFwdJ * nq; e += blockDim.x) {
        const int r = e / nq, i = 4 * (e - r * nq);
        // folded: 8 rows and their mirror images
        const int j = !d.fold || r < rows ? j0 + r : d.M - 1 - (j0 + r - rows);
        const bool in = d.fold ? (r < rows ? j < d.Mh : j >= d.Mh) : j < d.M;
        Vec4<T> v{};
        const long long o = (long long)(j + 1) * g.XP + 4 + i;
        if (in && TCSEM_IN(plane + o + 3, g.total(), d.err) &&
            TCSEM_IN((long long)(nch - 1) * plane + o + 3, (long long)nch * plane, d.err)) {
            v = ld4<true>(bz + plane + o);
            for (int c0 = 1; c0 < nch; c0 += 5) {  // five totals in flight
                Vec4<T> p[5];
#pragma unroll
                for (int c = 0; c < 5; c++) p[c] = c0 + c < nch ? ld4<true>(tot + (c0 + c) * plane + o) : Vec4<T>{};
#pragma unroll
                for (int c = 0; c < 5; c++)
#pragma unroll
                    for (int q = 0; q < 4; q++) v.v[q] += p[c].v[q];
            }
        }
        *reinterpret_cast<Vec4<T> *>(t.xrow(r) + i) = v;
    }
    __syncthreads();
    if (t.run(d.err)) {
        const int parts = d.fold ? 2 : 1, quads = rows / 4;
        for (int e = threadIdx.x; e < 4 * kTabN; e += blockDim.x) {  // four rows of one column
            const int n = e % kTabN, q = e / kTabN, odd = q / quads, r = 4 * (q % quads), c = n0 + n, j = j0 + r;
            if (c >= d.nc || odd >= parts || j >= d.Mh ||
                !TCSEM_IN((long long)c * d.ldF + odd * d.oFo + j + 3, (long long)d.nc * d.ldF, d.err))
                continue;
            Vec4<T> o;
#pragma unroll
            for (int a = 0; a < 4; a++) {
                o.v[a] = t.sum(r + a, n);
                if (d.fold) {
                    const T m = t.sum(rows + r + a, n);
                    o.v[a] = odd ? o.v[a] - m : o.v[a] + m;
                }
            }
            *reinterpret_cast<Vec4<T> *>(d.F + (size_t)c * d.ldF + odd * d.oFo + j) = o;
        }
    } else {
        wait.lost();
    }
    __syncthreads();
    if (threadIdx.x == 0) t.retire();
}

// the inverse along x and the sampling to the points of Bx (By), into plane -1
template <typename T, typename Wait>
__device__ __forceinline__ void inverse_x(const Products<T> &d, T *bx, T *by, const Geom &g, int blk, const Wait &wait) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tnx = up(d.L + 1, kTabN), tjx = up(d.M, kInvJ);
    const bool isy = blk >= tnx * tjx;
    const int b = isy ? blk - tnx * tjx : blk, nt = isy ? up(d.L, kTabN) : tnx;
    const int n0 = (b % nt) * kTabN, j0 = (b / nt) * kInvJ;
    const int rows = isy ? d.M + 1 : d.M, nn = isy ? d.L : d.L + 1;
    const Tile<T, kInvJ> t(smem_raw, d.nc, (isy ? d.Dy : d.Dx) + (size_t)(b % nt) * d.nc * kTabN);
    t.start();
    wait();
    // the rows of V from its columns: 16 columns by two row quads per warp, four loads in flight
    const T *src = d.V + (isy ? d.oVy : 0) + j0;
    for (int e0 = threadIdx.x; e0 < up(d.nc, 16) * 32; e0 += 4 * blockDim.x) {
        Vec4<T> v[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const int e = e0 + h * blockDim.x, c = e >> 1, q = e & 1;
            v[h] = c < d.nc && TCSEM_IN((long long)c * d.ldV + (isy ? d.oVy : 0) + j0 + 4 * q + 3, (long long)d.nc * d.ldV, d.err)
                       ? ld4<true>(src + (size_t)c * d.ldV + 4 * q) : Vec4<T>{};
        }
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const int e = e0 + h * blockDim.x, c = e >> 1, q = e & 1;
            if (c < d.nc)
#pragma unroll
                for (int a = 0; a < 4; a++) t.xrow(4 * q + a)[c] = v[h].v[a];
        }
    }
    __syncthreads();
    if (t.run(d.err)) {
        T *out = isy ? by : bx;
        for (int e = threadIdx.x; e < kInvJ * kTabN / 4; e += blockDim.x) {
            const int n = 4 * (e % (kTabN / 4)), j = e / (kTabN / 4), i = n0 + n;
            if (j0 + j >= rows || i >= nn || !TCSEM_IN(g.at(min(i + 3, nn - 1), j0 + j, -1), g.total(), d.err)) continue;
            const Vec4<T> o = t.sum4(j, n);
            T *dst = out + g.at(i, j0 + j, -1);
            if (i + 3 < nn) *reinterpret_cast<Vec4<T> *>(dst) = o;
            else
                for (int q = 0; q < nn - i; q++) dst[q] = o.v[q];
        }
    } else {
        wait.lost();
    }
    __syncthreads();
    if (threadIdx.x == 0) t.retire();
}

// ---- second product, NCOL frequencies kx per CTA: along y forward, the two continuation filters, and
// the inverse along y with the sampling to the rows of Bx and By.  With P and Q the cosine and sine
// parts of a column, F = P -+ iQ for ky and -ky; gx is even and gy odd in ky, so a pair contributes, with C
// and S the cosine and sine at the sampled row,
//   to Bx: i 2gx (C P + S Q),   to By: 2gy (C Q - S P);
// the unpaired ky = 0 and M1/2 give i gx C P (i gx S Q) and, at M1/2, i gy S Q.  Both sums have one thread
// per four outputs and share of k, the table straight from L2 (each element is used once per CTA) and the
// real and imaginary part as a pair.
template <typename T> struct SpecLayout {
    size_t f, u, part, total;
    int s1, s2;   // shares of k in the two sums
    int q1, qx, qy;  // quads of outputs: of one list of W, of C for Bx, for By
};
template <typename T> __host__ __device__ inline SpecLayout<T> spec_layout(const Products<T> &d, int ncol, int threads) {
    SpecLayout<T> l;
    l.q1 = up(d.K, 4);
    l.qx = up(d.Rx, 4);
    l.qy = up(d.Ry, 4);
    const int q2 = 2 * (l.qx + l.qy);
    l.s1 = threads / (2 * l.q1) > 1 ? threads / (2 * l.q1) : 1;
    l.s2 = threads / q2 > 1 ? threads / q2 : 1;
    if (l.s1 > 8) l.s1 = 8;
    if (l.s2 > 16) l.s2 = 16;
    const size_t c = (size_t)2 * ncol * sizeof(T);
    l.f = 0;                                               // [2 lists][Mh][ncol] pairs
    l.u = l.f + rnd16(2 * d.Mh * c);                       // [4 lists][K]
    l.part = l.u + rnd16(4 * (size_t)d.K * c);             // [shares][outputs]
    const size_t a = (size_t)l.s1 * 2 * l.q1 * 4 * c, b = (size_t)l.s2 * q2 * 4 * c;
    l.total = l.part + (a > b ? a : b);
    return l;
}
template <typename T, int NCOL, typename Wait>
__device__ __forceinline__ void through_y(const Products<T> &d, int blk, const Wait &wait) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    typedef Pair<T> P;
    const SpecLayout<T> l = spec_layout(d, NCOL, (int)blockDim.x);
    P *f = reinterpret_cast<P *>(smem_raw + l.f), *u = reinterpret_cast<P *>(smem_raw + l.u),
      *part = reinterpret_cast<P *>(smem_raw + l.part);
    const int kx0 = blk * NCOL, tid = threadIdx.x;
    // One item of a sum: the quad at column n of a table of K rows, k in [k0, k1); its first PRE rows are fetched
    // before the operand is there.
    constexpr int PRE = 4;
    struct Item {
        const T *t;
        int k0, k1;
    };
    auto prefetch = [](const Item &i, Vec4<T> (&pre)[PRE]) {
#pragma unroll
        for (int k = 0; k < PRE; k++)
            if (i.k0 + k < i.k1) pre[k] = ld4<false>(i.t + (size_t)(i.k0 + k) * kTabN);
    };
    auto dot = [](const Item &i, const Vec4<T> (&pre)[PRE], const P *x, P *out) {  // x: [k][NCOL]
        P acc[4][NCOL];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < NCOL; q++) acc[r][q] = dup<T>(T(0));
        auto row = [&](const Vec4<T> &w, int k) {
#pragma unroll
            for (int q = 0; q < NCOL; q++) {
                const P v = x[k * NCOL + q];
#pragma unroll
                for (int r = 0; r < 4; r++) acc[r][q] = fma(dup<T>(w.v[r]), v, acc[r][q]);
            }
        };
#pragma unroll
        for (int k = 0; k < PRE; k++)
            if (i.k0 + k < i.k1) row(pre[k], i.k0 + k);
#pragma unroll 4
        for (int k = i.k0 + PRE; k < i.k1; k++) row(ld4<false>(i.t + (size_t)k * kTabN), k);
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int q = 0; q < NCOL; q++) out[r * NCOL + q] = acc[r][q];
    };
    // the shares of one output, `pitch` apart, as four sums
    auto shares = [](const P *p, int n, int pitch) {
        const P none = dup<T>(T(0));
        auto at = [&](int k) { return k < n ? p[(size_t)k * pitch] : none; };
        P s0 = p[0], s1 = at(1), s2 = at(2), s3 = at(3);
        for (int k = 4; k < n; k += 4) {
            s0 = s0 + at(k);
            s1 = s1 + at(k + 1);
            s2 = s2 + at(k + 2);
            s3 = s3 + at(k + 3);
        }
        return (s0 + s1) + (s2 + s3);
    };
    auto column = [](const T *tab, int K, int n) { return tab + ((size_t)(n / kTabN) * K) * kTabN + n % kTabN; };
    const int n1 = 2 * l.q1, n2 = 2 * (l.qx + l.qy);
    auto item1 = [&](int e, int &o, int &list) {
        const int s = e / n1;
        o = e - s * n1;
        list = o >= l.q1;
        return Item{column(list ? d.Ws : d.Wc, d.Mh, 4 * (o - list * l.q1)), d.Mh * s / l.s1, d.Mh * (s + 1) / l.s1};
    };
    auto item2 = [&](int e, int &o, int &list) {  // list: of u
        const int s = e / n2;
        o = e - s * n2;
        const int isy = o >= 2 * l.qx, p = isy ? o - 2 * l.qx : o, nq = isy ? l.qy : l.qx, sine = p >= nq;
        list = 2 * isy + sine;
        return Item{column(isy ? (sine ? d.Cys : d.Cyc) : (sine ? d.Cxs : d.Cxc), d.K, 4 * (p - sine * nq)), d.K * s / l.s2,
                    d.K * (s + 1) / l.s2};
    };
    int o = 0, list = 0;
    Vec4<T> pre[PRE];
    Item it{};
    if (tid < n1 * l.s1) {
        it = item1(tid, o, list);
        prefetch(it, pre);
    }
    wait();
    for (int e = tid; e < 2 * d.Mh * NCOL; e += blockDim.x) {
        const int k = e % d.Mh, r = e / d.Mh, lf = r / NCOL, q = r % NCOL, c = 2 * (kx0 + q);
        P v = dup<T>(T(0));
        if (c < d.nc && TCSEM_IN((long long)(c + 1) * d.ldF + lf * d.oFo + k, (long long)d.nc * d.ldF, d.err)) {
            const T *p = d.F + (size_t)c * d.ldF + lf * d.oFo + k;
            v = pair<T>(__ldcg(p), __ldcg(p + d.ldF));
        }
        f[(lf * d.Mh + k) * NCOL + q] = v;
    }
    __syncthreads();
    for (int e = tid; e < n1 * l.s1; e += blockDim.x) {
        if (e != tid) {
            it = item1(e, o, list);
            prefetch(it, pre);
        }
        dot(it, pre, f + list * d.Mh * NCOL, part + (size_t)e * 4 * NCOL);
    }
    if (tid < n2 * l.s2) {
        it = item2(tid, o, list);
        prefetch(it, pre);
    }
    // filters: u = factors of C, S for Bx, then for By
    const int nyq = (d.M1 & 1) ? -1 : d.M1 / 2;
    auto filter = [&](int e, T &gx, T &gy) {
        const int q = e % NCOL, r = e / NCOL, ky = r % d.K, kx = kx0 + q;
        gx = gy = T(0);
        if (2 * kx < d.nc) {
            gx = __ldg(d.gx + (size_t)kx * d.ldG + ky);
            gy = __ldg(d.gy + (size_t)kx * d.ldG + ky);
        }
    };
    T gx = T(0), gy = T(0);
    if (tid < 2 * d.K * NCOL) filter(tid, gx, gy);
    __syncthreads();
    for (int e = tid; e < 2 * d.K * NCOL; e += blockDim.x) {
        if (e != tid) filter(e, gx, gy);
        const int q = e % NCOL, r = e / NCOL, sine = r >= d.K, ky = r - sine * d.K;
        const P *p = part + (size_t)((sine * l.q1 * 4 + ky) * NCOL + q);
        const P v = shares(p, l.s1, n1 * 4 * NCOL);
        u[(sine * d.K + ky) * NCOL + q] = pair<T>(-gx * v.b, gx * v.a);  // i gx
        P *yc = u + (2 * d.K + ky) * NCOL + q, *ys = u + (3 * d.K + ky) * NCOL + q;
        if (sine) {
            *yc = ky == nyq ? dup<T>(T(0)) : pair<T>(gy * v.a, gy * v.b);
            if (ky == nyq) *ys = pair<T>(-gy * v.b, gy * v.a);
        } else if (ky != nyq) {
            *ys = pair<T>(-gy * v.a, -gy * v.b);
        }
    }
    __syncthreads();
    for (int e = tid; e < n2 * l.s2; e += blockDim.x) {
        if (e != tid) {
            it = item2(e, o, list);
            prefetch(it, pre);
        }
        dot(it, pre, u + list * d.K * NCOL, part + (size_t)e * 4 * NCOL);
    }
    __syncthreads();
    // rows and their mirror images: sum and difference of the cosine and the sine part
    const int nr = d.Rx + d.Ry;
    for (int e = tid; e < nr * NCOL; e += blockDim.x) {
        const int r0 = e % nr, q = e / nr, isy = r0 >= d.Rx, r = isy ? r0 - d.Rx : r0, rows = isy ? d.M + 1 : d.M;
        const int oc = (isy ? 2 * l.qx : 0) * 4 + r, os = oc + (isy ? l.qy : l.qx) * 4, c = 2 * (kx0 + q);
        const P a = shares(part + (size_t)oc * NCOL + q, l.s2, n2 * 4 * NCOL),
                b = shares(part + (size_t)os * NCOL + q, l.s2, n2 * 4 * NCOL);
        if (c >= d.nc || !TCSEM_IN((long long)(c + 1) * d.ldV + (isy ? d.oVy : 0) + rows - 1, (long long)d.nc * d.ldV, d.err)) continue;
        T *v = d.V + (size_t)c * d.ldV + (isy ? d.oVy : 0);
        const P x = a + b, y = a - b;
        v[r] = x.a;
        v[d.ldV + r] = x.b;
        if (d.fold && 2 * r != rows - 1) {
            v[rows - 1 - r] = y.a;
            v[d.ldV + rows - 1 - r] = y.b;
        }
    }
    __syncthreads();
}

}  // namespace products
}  // namespace tcsem
