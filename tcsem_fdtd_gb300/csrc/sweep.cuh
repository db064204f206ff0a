// The fused E/B sweep as a per-CTA body, shared by the single-survey kernel,
// the batched kernel and the persistent batch scheduler.
#pragma once
#include "async.cuh"
#include "check.cuh"
#include "kernels.cuh"
#include "pair.cuh"

namespace tcsem {

// ------------------------------------------------------------- fused sweep
//
// One pass per time step over the volume: old E/B/sigma planes stream into a
// shared-memory ring through TMA bulk-tensor copies (cp.async.bulk.tensor,
// mbarrier completion): stage k of the ring is what the iteration of plane k reads,
// E and Bz of plane k and Bx, By and sigma of plane k-1 (those of plane k are in
// registers from the iteration before), so a slot is free after its iteration
// and every copy has three iterations to arrive.  The new E and B go to the other buffer of the
// ping-pong pair through shared-memory planes that the TMA stores.  Tiles are
// 64 x 8 columns, aligned so every TMA box starts on a 16-byte boundary; each
// thread owns two columns of a row (x = lane and lane + 32) and marches them z
// bottom-up through one z-chunk, the two cells side by side in packed FP32
// arithmetic (pair.cuh).  Warps 0..7 own the tile rows, warp 8 recomputes the +y
// halo row and warp 9 the +x halo column (E and the B components the tile's Bz
// needs), so no CTA waits for another; the -x/-y halo is plain old data in the
// TMA box.  Neighbour values of the new fields go through the same shared
// planes that are stored, double-buffered, with one __syncthreads per z-plane:
//   iteration k:  B(k+1)  ->  E(k)  ->  publish E(k), B(k+1)  ->  sync
//                 ->  TMA store of E(k), B(k+1), Bz(k+2); TMA load of stage k-4 into the freed slot
//                 ->  Bz(k+1)
//
// What bounds it: memory.  256 x 256 x 160 in FP32 (545 MB of algorithmic traffic, 80 us at the copy rate)
// takes 110 to 112 us, with DRAM busy 67 % of the time, issue slots 43 % and 51 million warp-instructions; with
// register stores, scalar arithmetic and two iterations of lead for the copies it was 119 us and 74 million.
// The pieces, measured one after the other: TMA stores and packed arithmetic 115.8 us (and 17 -> 14.5 us on
// 64 x 64 x 48, which stays in L2), the third iteration of lead 111.1 us.
//
// Bz within a chunk is the partial sum P(k) = sum_{k'=k}^{k1-1} dz div_xy B(k');
// the true Bz(k) = P(k) + O_c with O_c = sum of the chunk totals T_c' of the
// chunks below (c' > c).  Readers add O_c; T has one plane per chunk.

namespace fs3 {
constexpr int TX = 64, BY = 8;         // owned tile 64 x 8, two cells per thread: x = lane and lane + 32
constexpr int NW = 10;                 // warps 0..7 own the tile rows, 8: +y halo row, 9: +x halo column
constexpr int NT = 32 * NW;
constexpr int BXW = TX + 8, BYH = BY + 2;  // TMA box 72 x 10: x in [i0-4, i0+68), y in [j0-1, j0+9)
constexpr int BOX = BXW * BYH;
constexpr int NARR = 7;                // ex ey ez bx by bz sigma
// ring stride of one box: rounded up to 128 bytes so every TMA destination is 128-byte aligned
template <typename T> __host__ __device__ constexpr int boxs() { return (int)(((BOX * sizeof(T) + 127) / 128) * 128 / sizeof(T)); }
// stages in flight: four in FP32, where two CTAs share an SM and memory is the bound; two in FP64, where a
// plane takes several times a copy's latency on the FP64 pipe, which leaves room for boundary blocks beside
// the one CTA of an SM
template <typename T> __host__ __device__ constexpr int ring() { return sizeof(T) == 4 ? 4 : 2; }
enum { AEX = 0, AEY, AEZ, ABX, ABY, ABZ, ASG };
// New planes in shared memory, two buffers each.  Those that neighbours read (Ez, Bx, By): nine dense rows
// of 64 (the ninth is the +y halo row), then the +x halo column, then cells nobody reads for idle
// lanes.  Those that are only stored (Ex, Ey, Bz): eight dense rows.
constexpr int XCOL = 9 * TX, XBUF = 10 * TX, SBUF = BY * TX;
enum { XEZ = 0, XBX, XBY };
enum { SEX = 0, SEY, SBZ };
constexpr int kLost = 1 << 30;  // above every plane's number
template <typename T> __host__ __device__ constexpr int xoff(int a, int q) { return ring<T>() * NARR * boxs<T>() + (2 * a + q) * XBUF; }
template <typename T> __host__ __device__ constexpr int soff(int a, int q) { return xoff<T>(3, 0) + (3 * q + a) * SBUF; }
// What the z table is made from: its values dtb/dz, 1/(dz[k-1]+dz[k]) and dz of a plane, the first two times a factor
template <typename T> struct ZSource {
    const T *rdz, *rdzs, *dzk;
    T dtb, cf;
};
// byte offset of the ring's mbarriers, the source planes and the z table's source; then the z table
template <typename T> __host__ __device__ constexpr size_t bars_offset() { return (size_t)soff<T>(0, 2) * sizeof(T); }
template <typename T> __host__ __device__ constexpr size_t zsource_offset() { return bars_offset<T>() + ring<T>() * 8 + 16; }
template <typename T> __host__ __device__ constexpr size_t smem_bytes() { return zsource_offset<T>() + (sizeof(ZSource<T>) + 15) / 16 * 16; }
// Planes of the z table.  A deeper march fills it again on its way (two barriers every 220 planes), so that two CTAs
// share an SM in FP32 whatever the depth of the grid: with a table of all planes, each value twice, it was one
// CTA from 230 planes on.
constexpr int ZWIN = 224;
template <typename T> size_t smem_bytes_n(int N) {  // plus the z table
    return smem_bytes<T>() + 3 * (size_t)(N + 3 < ZWIN ? N + 3 : ZWIN) * 2 * sizeof(T);
}
// 228 KB of an SM, of which each CTA takes one more
static_assert(2 * (smem_bytes<float>() + 3 * (size_t)ZWIN * 2 * sizeof(float) + 1024) <= (228 << 10), "two CTAs per SM in FP32");
// the chunk offsets of Bz over the box, for the planes below k1 and for k1 itself, lie in the first
// buffers of the stored planes: they are in registers before the third plane of the march writes there
static_assert(2 * BOX <= 3 * SBUF, "the offset boxes fit the first store buffers");
}  // namespace fs3

// reciprocals of the E update: one MUFU op in FP32 (about 1 ulp)
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// In FP64 the hardware's approximation r0 of 1/x (a MUFU op, about 20 bits) and one third-order step of
// Householder's iteration, 1/x = r0 / (1 - e) = r0 (1 + e + e^2 + ...) with e = 1 - x r0: what is left out is
// e^3, and three FP64 operations take the place of a division's.  For normal x with a normal reciprocal: here
// x = 2 gamma + sigma dt with gamma > 0.  IEEE division's result or a neighbour of it (tests/test_gpu_reciprocal.py).
__device__ __forceinline__ double rcp64(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = ::fma(-x, r, 1.0);
    return ::fma(r, ::fma(e, e, e), r);
}
__device__ __forceinline__ Pair<double> rcp64(Pair<double> x) { return {rcp64(x.a), rcp64(x.b)}; }

// per-thread state of the sweep; sweep_plane() advances one z-plane: plane ktop - n reads the stage in slot n mod RING,
// round n / RING, and the buffers of parity PAR = n mod 2
template <typename T> struct SweepThread {
    T *sm;  // ring, then the new planes
    uint64_t *bars;
    int *s_src;  // first and last plane with a source segment in the tile
    const SweepMaps *maps;
    int j, N, k0, klow, ktop, i0, j0;  // planes k0 .. ktop - 1; klow: first plane of the z table
    int kend;     // last plane whose stage the thread waits for, or loads: k0, or kLost + the stage at which it gave up
    int role;     // 0: a row of the tile, 1: the +y halo row, 2: the +x halo column, 3: none (warp-uniform)
    int duty;     // 1: the thread issues the loads (a lane of warp 8), 2: the stores (of the +x warp)
    bool src;     // a source segment touches the tile in this step
    int so, xo, xd, xr, i;         // first cell: in the box, in the new planes; its +y and the second one's +x neighbour; x index
    // which components of the cells are updated: bits 0, 1 Ex and By, bits 2, 3 Ey and Bx (both: Ez too);
    // edge: not all of them in some lane of the warp, which then keeps old values where they are not
    unsigned upd;
    bool edge;
    Pair<T> rdy2, rdy, fy;         // per row: 1/(dy[j-1]+dy[j]), 1/dy[j], dtb/dy[j]
    // 2 lambda, dt/4 (the sweep forms sigma sums of four cells), c4.  FP64: c4 is in rdx2, rdy2 and the z
    // table's 1/(dz[k-1]+dz[k]), and t.c4 is 4 lambda
    Pair<T> lam, dt, c4;
    Pair<T> rdx2, rdx, fx;
    // Bz chunk offsets of the plane being updated: at, left of, below the cells (FP64: left minus at, at minus
    // below, and whether there are any)
    Pair<T> oc0, oci, ocj;
    bool offsets;
    Pair<T> ex1, ey1, exn, eyn, ezn;
    Pair<T> bxo1, byo1, bxn, byn, acc;
    Pair<T> sxk, syk, szk, bxk, byk, bxj, byi;  // of plane k: sigma sums, own B, Bx below and By left of the cell
};

// the old value of the cells whose bit of m (bits 0, 1) is not set
template <typename T> __device__ __forceinline__ void keep(Pair<T> &v, Pair<T> old, unsigned m) {
    if (!(m & 1u)) v.a = old.a;
    if (!(m & 2u)) v.b = old.b;
}
// the thread's two cells at offset o
template <typename T> __device__ __forceinline__ Pair<T> cells(const T *p, int o) { return pair<T>(p[o], p[o + 32]); }
template <typename T> __device__ __forceinline__ void put_cells(T *p, int o, Pair<T> v) { p[o] = v.a; p[o + 32] = v.b; }
// ... of which the +x halo column has one (ROLE 2: the second one's arithmetic is dead code)
template <int ROLE, typename T> __device__ __forceinline__ Pair<T> rcells(const T *p, int o) {
    if constexpr (ROLE == 2) return pair<T>(p[o], T(0));
    else return cells(p, o);
}
template <int ROLE, typename T> __device__ __forceinline__ void rput(T *p, int o, Pair<T> v) {
    if constexpr (ROLE == 2) p[o] = v.a;
    else put_cells(p, o, v);
}

// sigma sums and B of the plane in the B and sigma boxes p
template <int ROLE, typename T> __device__ __forceinline__ void carry_plane(SweepThread<T> &t, const T *p) {
    using namespace fs3;
    constexpr int BS = boxs<T>();
    const T *sg = p + ASG * BS;
    const int so = t.so;
    const Pair<T> a = rcells<ROLE>(sg, so), b = rcells<ROLE>(sg, so - 1), c = rcells<ROLE>(sg, so - BXW), d = rcells<ROLE>(sg, so - BXW - 1);
    t.sxk = a + c;
    t.syk = a + b;
    t.szk = t.sxk + b + d;
    t.bxk = rcells<ROLE>(p + ABX * BS, so);
    t.byk = rcells<ROLE>(p + ABY * BS, so);
    t.bxj = rcells<ROLE>(p + ABX * BS, so - BXW);
    t.byi = rcells<ROLE>(p + ABY * BS, so - 1);
}
// What the loading thread does before it loads the air plane (k = -1), the boundary's output: wait for the
// previous kernel on the stream (a top chunk launched early, programmatic dependent launch after the
// boundary's last stage, waits for it there and not before; no-op without the launch attribute).
struct AirAfterKernel {
    static constexpr int kPolls = 1 << 20;  // of a copy, before the wait for it gives up
    __device__ __forceinline__ void operator()() const { pdl_wait_prev(); }
};
// the loading thread: stage k into slot q
template <typename T, typename Air>
__device__ __forceinline__ void load_stage(const SweepThread<T> &t, int k, int q, const Air &air) {
    using namespace fs3;
    uint64_t *b = t.bars + q;
    T *dst = t.sm + q * NARR * boxs<T>();
    auto box = [&](int a, int z) { tma_load_3d(dst + a * boxs<T>(), t.maps->m + a, t.i0, t.j0, z + 1, b); };
    mbar_expect_tx(b, (unsigned)(NARR * BOX * sizeof(T)));
    box(AEX, k);
    box(AEY, k);
    box(AEZ, k);
    box(ABZ, k);
    box(ASG, k - 1);
    if (k == 0) air();
    box(ABX, k - 1);
    box(ABY, k - 1);
}

// Planes of a march: the first one (k = ktop: E of the halo plane, or the zero bottom; nothing stored), the
// second (no B below it in the chunk), the inner ones, and k0 - 1 (only B(k0)).  Compiled apart: the inner
// planes' code has no condition on k but the two at the end of the ring.
enum { FIRST, SECOND, INNER, LAST };

template <typename T, int PAR, int KIND, int ROLE, typename Air>
__device__ __forceinline__ void sweep_plane(SweepThread<T> &t, int k, int slot, int round, const StepScalars<T> &s,
                                            const Pair<T> *zt, const SourceTable<T> &src, const Air &air) {
    using namespace fs3;
    typedef Pair<T> P;
    constexpr int BS = boxs<T>(), RING = ring<T>();
    constexpr int QE = PAR, QB = PAR ^ 1;
    constexpr bool doB = (KIND == INNER || KIND == LAST) && ROLE != 3, doE = KIND != LAST && ROLE != 3;
    zt += 3 * (k - t.klow);  // dtb/dz, 1/(dz[k-1]+dz[k]), dz of plane k
    // Roles (one compiled copy each, FP64 only): the row warps update and store every component; the
    // +y halo row warp only produces what the tile's last row reads from it (Ex and Ez for By there,
    // By for Bz), the +x halo column warp what the tile's last column reads (Ey and Ez for Bx there,
    // Bx for Bz).  Every copy passes the one barrier per plane in the same order.
    constexpr bool rX = ROLE != 2, rY = ROLE != 1;
    const bool rows = sizeof(T) == 8 ? ROLE == 0 : t.role == 0;
    T *const sm = t.sm;
    // ---- B_new(k+1) from E_new(k+1) (own + neighbours) and E_new(k+2)
    if constexpr (doB) {
        const P fz = zt[3];
        const T *ez = sm + xoff<T>(XEZ, QB);
        if constexpr (rY) {
            const P ezj = rcells<ROLE>(ez, t.xd);
            t.bxn = fma(t.ezn - ezj, t.fy, fma(t.ey1 - t.eyn, fz, t.bxo1));
        }
        if constexpr (rX) {
            const P ezi = pair<T>(ez[t.xo + 1], ez[t.xr]);
            t.byn = fma(t.exn - t.ex1, fz, fma(ezi - t.ezn, t.fx, t.byo1));
        }
        if (t.edge) {
            keep(t.bxn, t.bxo1, t.upd >> 2);
            keep(t.byn, t.byo1, t.upd);
        }
    }
    // ---- E_new(k)
    if constexpr (doE) {
        t.ex1 = t.exn;
        t.ey1 = t.eyn;
        const T *p0 = sm + slot * (NARR * BS);
        const int so = t.so;
        const P sx0 = t.sxk, sy0 = t.syk, sz0 = t.szk, bx0 = t.bxk, by0 = t.byk, bxj = t.bxj, byi = t.byi;
        carry_plane<ROLE>(t, p0);  // plane k-1, the next one up
        const P ezo = rcells<ROLE>(p0 + AEZ * BS, so);
        P exo = dup<T>(T(0)), eyo = exo;
        if constexpr (rX) exo = rcells<ROLE>(p0 + AEX * BS, so);
        if constexpr (rY) eyo = rcells<ROLE>(p0 + AEY * BS, so);
        if (KIND != FIRST || k < t.N) {
            const P bz = rcells<ROLE>(p0 + ABZ * BS, so);
            // DuFort-Frankel update (ElectricalFiled.cu:89-345) of the three components, computed for
            // every cell and kept where the component is updated; s.dt carries the 1/4 of the sigma sums
            const P sx = sx0 + t.sxk, sy = sy0 + t.syk, lam = t.lam, dt = t.dt, c4 = t.c4, rdy2 = t.rdy2, rz2 = zt[1];
            if constexpr (sizeof(T) == 8) {
                // FP64, bound by the FP64 pipe (two lanes per clock and SM): with D = lam2 + sigma dt the
                // update (lam2 - sigma dt)/D E + c4/D curl is (2 lam2 E + c4 curl)/D - E, with c4 in the
                // cell sizes of the curl.  (In FP32, where 1/D is an approximate reciprocal, such a form
                // raised the trace error of a long whole run on 142 x 36 x 25 cells to 1.02 % of its peak.)
                const P rx = rcp64(fma(sx, dt, lam)), ry = rcp64(fma(sy, dt, lam)), rz = rcp64(fma(sz0, dt, lam));
                const P l2 = t.c4;
                if constexpr (rX) {
                    P db = bz - rcells<ROLE>(p0 + ABZ * BS, so - BXW);
                    if (t.offsets) db = db + t.ocj;
                    t.exn = fma(fma(db, rdy2, fma(t.byk - by0, rz2, l2 * exo)), rx, -exo);
                }
                if constexpr (rY) {
                    P db = rcells<ROLE>(p0 + ABZ * BS, so - 1) - bz;
                    if (t.offsets) db = db + t.oci;
                    t.eyn = fma(fma(db, t.rdx2, fma(bx0 - t.bxk, rz2, l2 * eyo)), ry, -eyo);
                }
                t.ezn = fma(fma(by0 - byi, t.rdx2, fma(bxj - bx0, rdy2, l2 * ezo)), rz, -ezo);
            } else {
                const P bzo = bz + t.oc0;
                const P cz = fma(by0 - byi, t.rdx2, -((bx0 - bxj) * rdy2));
                const P cx = fma(bzo - (rcells<ROLE>(p0 + ABZ * BS, so - BXW) + t.ocj), rdy2, -((by0 - t.byk) * rz2));
                const P cy = fma(bx0 - t.bxk, rz2, -((bzo - (rcells<ROLE>(p0 + ABZ * BS, so - 1) + t.oci)) * t.rdx2));
                auto rcp = [](P d) { return pair<T>(rcp_fast(d.a), rcp_fast(d.b)); };
                const P Dx = fma(sx, dt, lam), Dy = fma(sy, dt, lam), Dz = fma(sz0, dt, lam);
                const P rx = rcp(Dx), ry = rcp(Dy), rz = rcp(Dz), ndt = -dt;
                t.exn = fma(fma(sx, ndt, lam) * rx, exo, (c4 * rx) * cx);
                t.eyn = fma(fma(sy, ndt, lam) * ry, eyo, (c4 * ry) * cy);
                t.ezn = fma(fma(sz0, ndt, lam) * rz, ezo, (c4 * rz) * cz);
            }
            if (t.edge) {
                if constexpr (rX) keep(t.exn, exo, t.upd);
                if constexpr (rY) keep(t.eyn, eyo, t.upd >> 2);
                keep(t.ezn, ezo, t.upd & (t.upd >> 2));
            }
            // AddTx_*: subtracted after the update of the cell, on the planes where a segment meets the tile
            if (t.src && k >= t.s_src[0] && k <= t.s_src[1]) {
                T e[3][2] = {{t.exn.a, t.exn.b}, {t.eyn.a, t.eyn.b}, {t.ezn.a, t.ezn.b}};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    if (!(t.upd & (5u << c))) continue;
                    const int i = t.i + 32 * c;
                    for (int q = 0; q < src.nseg; q++) {
                        const int cp = src.comp[q];
                        int d;
                        if (cp == 0) { if (t.j != src.j[q] || k != src.k[q]) continue; d = i - src.i[q]; }
                        else if (cp == 1) { if (i != src.i[q] || k != src.k[q]) continue; d = t.j - src.j[q]; }
                        else { if (i != src.i[q] || t.j != src.j[q]) continue; d = k - src.k[q]; }
                        if (d < 0 || d >= src.count[q]) continue;
                        const T v = s.wave * src.coef[src.off[q] + d];
                        if (cp == 0) e[0][c] -= v; else if (cp == 1) e[1][c] -= v; else e[2][c] -= v;
                    }
                }
                t.exn = pair<T>(e[0][0], e[0][1]);
                t.eyn = pair<T>(e[1][0], e[1][1]);
                t.ezn = pair<T>(e[2][0], e[2][1]);
            }
        } else {
            t.exn = exo;
            t.eyn = eyo;
            t.ezn = ezo;
        }
        t.bxo1 = bx0;  // B_old(k) for the next plane's B update
        t.byo1 = by0;
        rput<ROLE>(sm + xoff<T>(XEZ, QE), t.xo, t.ezn);  // publish Ez_new(k)
        if (KIND != FIRST && rows) {
            rput<ROLE>(sm + soff<T>(SEX, QE), t.xo, t.exn);
            rput<ROLE>(sm + soff<T>(SEY, QE), t.xo, t.eyn);
        }
    }
    if constexpr (doB) {  // publish B_new(k+1): Bx where Bz reads it (rows, +x column), By likewise (rows, +y row)
        if constexpr (rY) rput<ROLE>(sm + xoff<T>(XBX, QB), t.xo, t.bxn);
        if constexpr (rX) rput<ROLE>(sm + xoff<T>(XBY, QB), t.xo, t.byn);
    }
    // stage k-1 is read by the next plane; a thread whose wait gave up waits for no other, and loads none.  The last
    // slot is one phase ahead: it carried plane ktop's B and sigma first.
    const int ns = (slot + 1) % RING;
    const unsigned parity = (unsigned)(round + (ns == 0) + (ns == RING - 1)) & 1u;
    if (KIND != LAST && k > t.kend && !mbar_wait_bounded(t.bars + ns, parity, Air::kPolls)) t.kend = kLost + k - 1;
    async_shared_fence();  // the new planes are read by the TMA
    if (t.duty == 2) bulk_wait_read();  // ... which is done with the buffers the next plane writes
    __syncthreads();
    if (t.duty) {
        if (t.duty == 2) {  // store E(k), B(k+1) and, summed after the barrier of plane k+1, Bz(k+2)
            if constexpr (KIND == SECOND || KIND == INNER) {
                tma_store_3d(t.maps->o + 0, sm + soff<T>(SEX, QE), t.i0, t.j0, k);
                tma_store_3d(t.maps->o + 1, sm + soff<T>(SEY, QE), t.i0, t.j0, k);
                tma_store_3d(t.maps->o + 2, sm + xoff<T>(XEZ, QE), t.i0, t.j0, k);
            }
            if constexpr (KIND == INNER || KIND == LAST) {
                tma_store_3d(t.maps->o + 3, sm + xoff<T>(XBX, QB), t.i0, t.j0, k + 1);
                tma_store_3d(t.maps->o + 4, sm + xoff<T>(XBY, QB), t.i0, t.j0, k + 1);
                if (k + 2 < t.ktop) tma_store_3d(t.maps->o + 5, sm + soff<T>(SBZ, QB), t.i0, t.j0, k + 2);
            }
            bulk_commit();
        } else if (KIND != LAST && k - RING >= t.kend) {  // the slot takes the stage RING planes up
            load_stage(t, k - RING, slot, air);
        }
    }
    // ---- Bz(k+1) = Bz(k+2) + dz (dBx/dx + dBy/dy), for the tile's own rows
    if (doB && rows) {
        const T *bx = sm + xoff<T>(XBX, QB), *by = sm + xoff<T>(XBY, QB);
        const P bxr = pair<T>(bx[t.xo + 1], bx[t.xr]), byu = rcells<ROLE>(by, t.xd);
        t.acc = fma(zt[5], fma(bxr - t.bxn, t.rdx, (byu - t.byn) * t.rdy), t.acc);
        rput<ROLE>(sm + soff<T>(SBZ, QE), t.xo, t.acc);
    }
}

// the cells' Bz chunk offsets from one of the two offset boxes
template <typename T> __device__ __forceinline__ void set_offsets(SweepThread<T> &t, const T *box) {
    t.oc0 = cells(box, t.so);
    t.oci = cells(box, t.so - 1);
    t.ocj = cells(box, t.so - fs3::BXW);
    if (sizeof(T) == 8) {
        t.oci = t.oci - t.oc0;
        t.ocj = t.oc0 - t.ocj;
    }
}

// all threads: the z table for the planes klow ..., as far as it goes or the march needs
template <typename T> __device__ __forceinline__ void fill_z(Pair<T> *s_z, const fs3::ZSource<T> &z, int klow, int ktop, int N) {
    const int n = min(fs3::ZWIN, ktop + 2 - klow);
    for (int e = threadIdx.x; e < n; e += fs3::NT) {
        const int k = klow + e;
        const bool in = k >= 0 && k < N;
        s_z[3 * e] = dup<T>(in ? z.rdz[k] * z.dtb : T(0));
        s_z[3 * e + 1] = dup<T>(in ? z.rdzs[k] * z.cf : T(0));
        s_z[3 * e + 2] = dup<T>(in ? z.dzk[k] : T(0));
    }
}
// all threads, between two planes: the table for the planes below k, down to k0 - 1 if they fit
template <typename T> __device__ __forceinline__ void refill_z(SweepThread<T> &t, Pair<T> *s_z, int k) {
    const fs3::ZSource<T> &z = *reinterpret_cast<const fs3::ZSource<T> *>(reinterpret_cast<const unsigned char *>(t.sm) + fs3::zsource_offset<T>());
    __syncthreads();  // the last plane's readers are done
    t.klow = max(t.k0 - 1, k + 1 - fs3::ZWIN);
    fill_z(s_z, z, t.klow, k - 1, t.N);
    __syncthreads();
}

// The z-march of one warp through the chunk, in the copy of the plane code for its role.  COPIES of the inner plane:
// RING with the slots as constants, or 2 with the slot in a register and half of the code (256 x 256 x 160
// 131.2 -> 128.7 us per step, in FP64 1348 -> 1336).  The batched and the cooperative kernel keep RING in FP32: there the
// register is one too many (8 surveys of up to 152 x 131 x 112 170 -> 174 us, 64 x 64 x 48 19.2 -> 19.3).
// DEEP: the march may have more planes than the z table.
template <typename T, int ROLE, int COPIES, bool DEEP, typename Air>
__device__ __forceinline__ void sweep_march(SweepThread<T> &t, const StepScalars<T> &s, Pair<T> *s_z,
                                            const SourceTable<T> &src, const T *s_oc, const Air &air) {
    using namespace fs3;
    constexpr int RING = ring<T>();
    static_assert(COPIES == 2 || (COPIES == 4 && RING == 4), "slots of the inner copies");
    const int k0 = t.k0;
    sweep_plane<T, 0, FIRST, ROLE>(t, t.ktop, 0, 0, s, s_z, src, air);
    set_offsets(t, s_oc);
    // the inner planes k = ktop - 2 .. k0
    int k = t.ktop - 1;
    sweep_plane<T, 1, SECOND, ROLE>(t, k, 1 % RING, 1 / RING, s, s_z, src, air);
    if constexpr (COPIES == 2) {
        int n = 2;  // planes done
        for (;;) {
            if (DEEP && t.klow >= k0 && k - 2 < t.klow) refill_z(t, s_z, k);
            if (--k < k0) break;
            sweep_plane<T, 0, INNER, ROLE>(t, k, n % RING, n / RING, s, s_z, src, air);
            n++;
            if (--k < k0) break;
            sweep_plane<T, 1, INNER, ROLE>(t, k, n % RING, n / RING, s, s_z, src, air);
            n++;
        }
        if (n & 1) sweep_plane<T, 1, LAST, ROLE>(t, k, n % RING, n / RING, s, s_z, src, air);
        else sweep_plane<T, 0, LAST, ROLE>(t, k, n % RING, n / RING, s, s_z, src, air);
    } else {
        int round = 0, left = 2;  // slot of the plane after the last inner one
        for (;;) {
            if (DEEP && t.klow >= k0 && k - 4 < t.klow) refill_z(t, s_z, k);
            if (--k < k0) break;
            sweep_plane<T, 0, INNER, ROLE>(t, k, 2, round, s, s_z, src, air);
            if (--k < k0) { left = 3; break; }
            sweep_plane<T, 1, INNER, ROLE>(t, k, 3, round, s, s_z, src, air);
            round ^= 1;
            if (--k < k0) { left = 0; break; }
            sweep_plane<T, 0, INNER, ROLE>(t, k, 0, round, s, s_z, src, air);
            if (--k < k0) { left = 1; break; }
            sweep_plane<T, 1, INNER, ROLE>(t, k, 1, round, s, s_z, src, air);
        }
        if (left == 0) sweep_plane<T, 0, LAST, ROLE>(t, k, 0, round, s, s_z, src, air);
        else if (left == 1) sweep_plane<T, 1, LAST, ROLE>(t, k, 1, round, s, s_z, src, air);
        else if (left == 2) sweep_plane<T, 0, LAST, ROLE>(t, k, 2, round, s, s_z, src, air);
        else sweep_plane<T, 1, LAST, ROLE>(t, k, 3, round, s, s_z, src, air);
    }
}

// one CTA of the sweep: tile (bx, by) of z-chunk c (or a piece of the only chunk) with the step scalars s.  FRESH: the chunk
// totals tin may have been written by another CTA of the same launch (persistent schedule).  False (for all threads): a
// copy did not arrive; it is recorded in err, and no copy is in flight.
template <typename T, bool FRESH = false, int COPIES = fs3::ring<T>(), bool DEEP = true, typename Air = AirAfterKernel>
__device__ __forceinline__ bool sweep_cta(const SweepMaps &maps, const Geom &g, const T *__restrict__ tin,
                                          T *__restrict__ tout, const Axis<T> &ax, StepScalars<T> s,
                                          const SourceTable<T> &src, const ZChunks &zc, int bx, int by, int c, int *err,
                                          const Air &air = Air(), Piece piece = Piece::WHOLE,
                                          const T *__restrict__ bz_new = nullptr) {
    using namespace fs3;
    constexpr int BS = boxs<T>(), RING = ring<T>();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SweepThread<T> t;
    t.sm = reinterpret_cast<T *>(smem_raw);
    T *s_oc = t.sm + soff<T>(0, 0);  // [BYH][BXW] chunk offsets of Bz for planes < k1
    T *s_oc1 = s_oc + BOX;           // ... for plane k1
    t.bars = reinterpret_cast<uint64_t *>(smem_raw + bars_offset<T>());
    static_assert(bars_offset<T>() % 128 == 0, "the new planes are whole 128-byte lines");
    t.s_src = reinterpret_cast<int *>(t.bars + RING);
    Pair<T> *s_z = reinterpret_cast<Pair<T> *>(smem_raw + smem_bytes<T>());  // [ZWIN][3] at most, each value twice
    t.maps = &maps;

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    t.i0 = bx * TX;
    t.j0 = by * zc.rows;
    const int L = g.L, M = g.M, N = g.N, XP = g.XP, PS = (int)g.PS;
    t.N = N;
    t.k0 = zc.plane(c) + (piece == Piece::LOWER ? 1 : 0);
    t.ktop = piece == Piece::TOP ? t.k0 + 1 : zc.plane(c + 1);  // first plane of the march: the halo plane of the chunk below, or the zero bottom
    // rows: cells x = lane, lane + 32 of row w; column warp: one cell per lane, x = 64 of row `lane`.  A tile
    // has zc.rows rows, warp zc.rows computes the halo row and the warps between it and the column's idle.
    const bool column = w == 9;
    const int ty = column ? lane : w;
    t.role = column ? 2 : w < zc.rows ? 0 : w == zc.rows ? 1 : 3;
    t.duty = lane == 0 ? (column ? 2 : w == 8 ? 1 : 0) : 0;
    t.j = t.j0 + ty;
    t.i = t.i0 + (column ? TX : lane);
    const bool rowok = column ? lane <= zc.rows : t.role != 3;
    t.so = rowok ? (ty + 1) * BXW + (column ? TX : lane) + 4 : BXW + 4;
    t.xo = column ? XCOL + lane : ty * TX + lane;  // the column's idle lanes and second cells: cells nobody reads
    t.xd = t.xo + (column ? 1 : TX);
    t.xr = column ? t.xo : lane < 31 ? t.xo + 33 : XCOL + ty;
    s.dt *= T(0.25);  // the sweep forms sigma sums of four cells: 0.25 * sum * dt
    const T cf = sizeof(T) == 4 ? T(1) : s.c4;  // in the cell sizes of the curl (FP64)
    t.lam = dup<T>(s.lam2);
    t.dt = dup<T>(s.dt);
    t.c4 = dup<T>(sizeof(T) == 4 ? s.c4 : s.lam2 + s.lam2);
    const T rdy = (rowok && t.j < M) ? ax.rdy[t.j] : T(0);
    t.rdy2 = dup<T>((rowok && t.j >= 1 && t.j < M) ? ax.rdy2[t.j] * cf : T(0));
    t.rdy = dup<T>(rdy);
    t.fy = dup<T>(rdy * s.dtb);
    T r2[2], r1[2];
    t.upd = 0;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const bool act = rowok && (q == 0 || !column);
        const int i = t.i + 32 * q;
        const bool ux = act && t.j >= 1 && t.j < M && i < L, uy = act && i >= 1 && i < L && t.j < M;
        t.upd |= (ux ? 1u << q : 0u) | (uy ? 4u << q : 0u);
        r2[q] = uy ? ax.rdx2[i] * cf : T(0);
        r1[q] = (act && i < L) ? ax.rdx[i] : T(0);
    }
    t.edge = __any_sync(0xffffffffu, t.upd != 15u);
    t.rdx2 = pair<T>(r2[0], r2[1]);
    t.rdx = pair<T>(r1[0], r1[1]);
    t.fx = pair<T>(r1[0] * s.dtb, r1[1] * s.dtb);
    const int ktop = t.ktop;
    t.klow = DEEP ? max(t.k0 - 1, ktop + 2 - ZWIN) : t.k0 - 1;  // entries of planes ktop and ktop + 1 among them
    const ZSource<T> zsrc{ax.rdz, ax.rdzs, ax.dzk, s.dtb, cf};
    fill_z(s_z, zsrc, t.klow, ktop, N);
    if (DEEP && tid == 0) *reinterpret_cast<ZSource<T> *>(smem_raw + zsource_offset<T>()) = zsrc;

    bool src_tile = false;  // tile-uniform: does any source segment touch this tile, and on which planes?
    int sk0 = N, sk1 = -1;
    for (int q = 0; q < src.nseg; q++) {
        int a0 = src.i[q], a1 = src.i[q], b0 = src.j[q], b1 = src.j[q], c1 = src.k[q];
        if (src.comp[q] == 0) a1 += src.count[q] - 1;
        if (src.comp[q] == 1) b1 += src.count[q] - 1;
        if (src.comp[q] == 2) c1 += src.count[q] - 1;
        if (a1 >= t.i0 && a0 <= t.i0 + TX && b1 >= t.j0 && b0 <= t.j0 + zc.rows) {
            src_tile = true;
            sk0 = min(sk0, src.k[q]);
            sk1 = max(sk1, c1);
        }
    }
    t.src = src_tile && s.wave != T(0);
    if (tid == 0) {
        for (int r = 0; r < RING; r++) mbar_init(t.bars + r, 1);
        mbar_init_fence();
        t.s_src[0] = sk0;  // read by the source epilogue, after the barrier below
        t.s_src[1] = sk1;
    }
    __syncthreads();
    if (t.duty == 1) {  // B and sigma of plane ktop through the last slot, the first stages into the others
        uint64_t *b = t.bars + RING - 1;
        async_shared_fence();  // another role's ordinary stores, where CTAs outlive one tile
        mbar_expect_tx(b, (unsigned)(3 * BOX * sizeof(T)));
        for (int a : {ABX, ABY, ASG})
            tma_load_3d(t.sm + ((RING - 1) * NARR + a) * BS, maps.m + a, t.i0, t.j0, ktop + 1, b);
        for (int q = 0; q < RING - 1 && ktop - q >= t.k0; q++) load_stage(t, ktop - q, q, air);
    }
    // chunk offsets of Bz over the box (zero without chunking)
    for (int e = tid; e < BOX; e += NT) {
        T o = T(0), o1 = T(0);
        if (zc.n > 1) {
            const int gy = t.j0 + e / BXW, gx = t.i0 + e % BXW;  // padded coordinates
            if (gy < g.YP && gx < XP) {
                const int pc = gy * XP + gx;
                T pv[kMaxChunks];  // all loads in flight together
#pragma unroll
                for (int q = 1; q < kMaxChunks; q++)
                    pv[q] = q > c && q < zc.n && TCSEM_IN(q * PS + pc, zc.n * PS, err) ? ld_in<FRESH>(tin + q * PS + pc) : T(0);
                const T first = c + 1 < zc.n ? ld_in<FRESH>(tin + (c + 1) * PS + pc) : T(0);
#pragma unroll
                for (int q = 1; q < kMaxChunks; q++)
                    if (q > c && q < zc.n) o += pv[q];
                o1 = c + 1 < zc.n ? o - first : T(0);
            }
        }
        s_oc[e] = o;
        s_oc1[e] = o1;
    }
    t.kend = mbar_wait_bounded(t.bars + RING - 1, 0u) && mbar_wait_bounded(t.bars + 0, 0u) ? t.k0 : kLost + ktop;
    carry_plane<0>(t, t.sm + (RING - 1) * NARR * BS);
    t.ex1 = t.ey1 = t.exn = t.eyn = t.ezn = dup<T>(T(0));
    t.bxo1 = t.byo1 = t.bxn = t.byn = t.acc = dup<T>(T(0));
    if (piece == Piece::TOP && t.role == 0 && t.j < M) {  // the sum up to the plane below
        const long long o = g.at(t.i, t.j, t.ktop);
        if (t.i < L && TCSEM_IN(o, g.total(), err)) t.acc.a = __ldcg(bz_new + o);
        if (t.i + 32 < L && TCSEM_IN(o + 32, g.total(), err)) t.acc.b = __ldcg(bz_new + o + 32);
    }
    async_shared_fence();
    __syncthreads();
    if (t.duty == 1 && ktop - (RING - 1) >= t.kend) load_stage(t, ktop - (RING - 1), RING - 1, air);

    // Bz offsets of the first plane: ktop is the halo plane k1 of the chunk below (its offsets) or the
    // zero bottom; every later plane lies in this chunk
    set_offsets(t, ktop < N ? s_oc1 : s_oc);
    t.offsets = c + 1 < zc.n;
    // FP64 (bound by the FP64 pipe): the halo warps run their reduced copies of the plane code
    // (5 % faster).  FP32 runs one copy in every warp: three copies of its loop made the sweep 40 %
    // slower (measured; presumably the larger loop no longer fits the instruction cache).
    if constexpr (sizeof(T) == 8) {
        if (t.role == 0) sweep_march<T, 0, COPIES, DEEP>(t, s, s_z, src, s_oc, air);
        else if (t.role == 1) sweep_march<T, 1, COPIES, DEEP>(t, s, s_z, src, s_oc, air);
        else if (t.role == 2) sweep_march<T, 2, COPIES, DEEP>(t, s, s_z, src, s_oc, air);
        else sweep_march<T, 3, COPIES, DEEP>(t, s, s_z, src, s_oc, air);
    } else {
        sweep_march<T, 0, COPIES, DEEP>(t, s, s_z, src, s_oc, air);
    }
    // the last plane's Bz, in the buffer of its parity
    async_shared_fence();
    const bool bad = __syncthreads_or(t.kend >= kLost);
    if (t.duty == 2) {
        tma_store_3d(maps.o + 5, t.sm + ((ktop - t.k0) & 1 ? soff<T>(SBZ, 0) : soff<T>(SBZ, 1)), t.i0, t.j0, t.k0);
        bulk_commit();
        bulk_wait_all();
    }
    if (bad) {  // a copy did not arrive: record it and let those in flight land
        if (t.duty == 1) {
            atomicExch(err, 1);
            // Unless this thread gave up, it has seen every stage land.  Having given up on stage `lost` it loaded no
            // more: the RING - 1 stages from that one on were under way (and at the first one, ktop's B and sigma).
            if (t.kend >= kLost) {
                const int lost = t.kend - kLost;
                if (lost == ktop) mbar_wait_bounded(t.bars + RING - 1, 0u);
                for (int k = lost; k > lost - (RING - 1) && k >= t.k0; k--) {
                    const int n = ktop - k;  // slot n % RING, round n / RING
                    mbar_wait_bounded(t.bars + n % RING, (unsigned)(n / RING + (n % RING == RING - 1)) & 1u);
                }
            }
        }
        __syncthreads();
        return false;
    }
    if (zc.n > 1 && t.role == 0) {
        const T a[2] = {t.acc.a, t.acc.b};
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int o = c * PS + (t.j + 1) * XP + t.i + 32 * q + 4;
            if (t.j < M && t.i + 32 * q < L && TCSEM_IN(o, zc.n * PS, err)) tout[o] = a[q];
        }
    }
    return true;
}

}  // namespace tcsem
