// rpy_kernels.cu -- pairwise RPY block products on the FP32 pipe.
//
// Replaces the reference kernels Mss_mult / Mbb_mult / Msb_mult / Mbs_mult
// (src/cilia/cuda_functions.cu:362-757).  Those use one thread per target,
// 64-thread blocks and AoS global loads; here a CTA of 128 threads owns
// 128*TI targets and one split of the sources, staged by a single bulk async
// copy per array into shared memory, so that the grid covers every SM even
// for a few thousand particles.  Partial sums are reduced in FP64 by a second
// small kernel in a fixed order.
#include "common.cuh"
#include "rpy_kernels.cuh"
#include "rpy_pairs.cuh"
#include "rpy_sym6.cuh"
#include "tma.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace cufil {

namespace {

constexpr int kThreads = 128;
constexpr int kMaxSplit = 2048;   // sources staged per CTA (<= 96 KB with torques)
constexpr int kMinSplit = 64;     // keep each split long enough to amortise staging
constexpr int kBlockSum = 64;     // sources per FP32 block sum before TwoSum
constexpr int kCtasPerSm = 8;     // launch bound: 8 x 128 threads x 64 registers = one SM's file
constexpr int kStageCost = 24;    // per-CTA staging/epilogue cost in units of one source

struct TileParams {
    const float4 *xt;
    const float4 *xs;
    const float4 *fs;
    const float4 *ts;
    float4 *partial;
    int nt, ns, split, ntp;
    float at, as, inv_mu;
    int *err;
    unsigned wait_limit;  // tries of the first wait for the staged sources
};

template <int VD>
__device__ __forceinline__ void two_sum_add(float *hi, float *lo, const float *a) {
#pragma unroll
    for (int c = 0; c < VD; ++c) {
        const float t = hi[c] + a[c];
        const float bp = t - hi[c];
        lo[c] += (hi[c] - (t - bp)) + (a[c] - bp);
        hi[c] = t;
    }
}

template <bool WALL, int VD, int FD, int TI, bool MASK>
__device__ __forceinline__ void tile_sum(const float4 *__restrict__ xs_s, const float4 *__restrict__ fs_s,
                                         const float4 *__restrict__ ts_s, int nsrc, int j0, const int *gi,
                                         const float (*xi)[3], float at, float as, float inv_mu,
                                         float (*hi)[VD], float (*lo)[VD]) {
    for (int jb = 0; jb < nsrc; jb += kBlockSum) {
        const int je = min(nsrc, jb + kBlockSum);
        float acc[TI][VD];
#pragma unroll
        for (int k = 0; k < TI; ++k)
#pragma unroll
            for (int c = 0; c < VD; ++c) acc[k][c] = 0.0f;
#pragma unroll 2
        for (int j = jb; j < je; ++j) {
            const float4 p = xs_s[j];
            const float4 f4 = fs_s[j];
            float f[6] = {f4.x, f4.y, f4.z, 0.f, 0.f, 0.f};
            if constexpr (FD > 3) {
                const float4 t4 = ts_s[j];
                f[3] = t4.x;
                f[4] = t4.y;
                f[5] = t4.z;
            }
#pragma unroll
            for (int k = 0; k < TI; ++k) {
                if constexpr (MASK) {
                    if (gi[k] == j0 + j) continue;  // the self block is added by the reduction
                }
                const float dx = xi[k][0] - p.x, dy = xi[k][1] - p.y, dz = xi[k][2] - p.z;
                if constexpr (WALL)
                    wall_pair_f32<VD, FD>(dx, dy, dz, xi[k][2], p.z, f, acc[k]);
                else
                    free_pair_f32<VD, FD>(dx, dy, dz, at, as, inv_mu, f, acc[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < TI; ++k) two_sum_add<VD>(hi[k], lo[k], acc[k]);
    }
}

// grid: (tiles, nsplit); block: 128.  SELF: targets and sources are the same
// particle set (wall mode skips j == i here; the reduction adds the self block).
template <bool WALL, int VD, int FD, int TI, bool SELF>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) rpy_tile_kernel(TileParams p) {
    chain_wait();  // launched as a programmatic dependent of the packing launch
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);
    float4 *xs_s = reinterpret_cast<float4 *>(smem_raw + 16);
    float4 *fs_s = xs_s + p.split;
    float4 *ts_s = fs_s + p.split;

    const int j0 = blockIdx.y * p.split;
    const int nsrc = max(0, min(p.ns, j0 + p.split) - j0);
    const int t0 = blockIdx.x * (kThreads * TI);

    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && nsrc > 0) {
        const uint32_t bytes = static_cast<uint32_t>(nsrc) * sizeof(float4);
        mbar_arrive_expect_tx(bar, bytes * (FD > 3 ? 3u : 2u));
        bulk_g2s(xs_s, p.xs + j0, bytes, bar);
        bulk_g2s(fs_s, p.fs + j0, bytes, bar);
        if constexpr (FD > 3) bulk_g2s(ts_s, p.ts + j0, bytes, bar);
    }

    // Targets of this thread (tail threads duplicate the last target and do not store).
    int gi[TI];
    float xi[TI][3];
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        const int i = t0 + k * kThreads + threadIdx.x;
        gi[k] = i;
        const float4 q = p.xt[min(i, p.nt - 1)];
        xi[k][0] = q.x;
        xi[k][1] = q.y;
        xi[k][2] = q.z;
    }
    float hi[TI][VD], lo[TI][VD];
#pragma unroll
    for (int k = 0; k < TI; ++k)
#pragma unroll
        for (int c = 0; c < VD; ++c) hi[k][c] = lo[k][c] = 0.0f;

    if (nsrc > 0) {
        if (!mbar_wait_bounded(bar, 0, p.wait_limit)) {
            // Gave up: flag it, skip the sum and the stores, and let every
            // thread drain the copies already issued (one more bounded wait
            // with the full limit) before it exits, so that no copy lands in
            // shared memory that another block has been given.  A copy still
            // in flight after that second limit is not handled.
            if (threadIdx.x == 0) atomicOr(p.err, kErrTmaTimeout);
            mbar_wait_bounded(bar, 0);
            return;
        }
        bool diag = false;
        if constexpr (WALL && SELF) diag = (j0 < t0 + kThreads * TI) && (t0 < j0 + nsrc);
        if (diag)
            tile_sum<WALL, VD, FD, TI, true>(xs_s, fs_s, ts_s, nsrc, j0, gi, xi, p.at, p.as, p.inv_mu, hi, lo);
        else
            tile_sum<WALL, VD, FD, TI, false>(xs_s, fs_s, ts_s, nsrc, j0, gi, xi, p.at, p.as, p.inv_mu, hi, lo);
    }

    constexpr int W = VD / 3;
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        const int i = gi[k];
        if (i >= p.nt) continue;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            float4 o;
            o.x = hi[k][3 * w + 0] + lo[k][3 * w + 0];
            o.y = hi[k][3 * w + 1] + lo[k][3 * w + 1];
            o.z = hi[k][3 * w + 2] + lo[k][3 * w + 2];
            o.w = 0.0f;
            p.partial[(static_cast<size_t>(i) * gridDim.y + blockIdx.y) * W + w] = o;
        }
    }
}

// ---------------------------------------------------------------------------
// Symmetric kernel for a set of particles acting on themselves: segments with or
// without torques and spins, blobs after them, above the wall or (equal spheres)
// unbounded.  The grand mobility is symmetric, so each unordered pair is evaluated
// once and applied in both directions (rpy_pairs.cuh, rpy_sym6.cuh).  Work unit:
// one warp and one pair of 32-particle tiles (I <= J) of the upper triangle.  The
// warp's lanes own the 32 targets of tile I; the 32 sources of tile J, with the
// accumulators of their own velocities, rotate around the warp by one lane per
// step, so after 32 steps every lane has met every source and every source
// accumulator is back in its home lane.  Diagonal tiles are evaluated one-sided
// (j != i; the other direction's results are dropped).  Each target receives exactly
// one partial per tile (RpyPlan says where) -- no atomics, deterministic; the
// reduction adds the self blocks.
//
// This kernel serves the sets with torques (the one below those without).  Bound by
// instruction issue: above the wall about 200 FP32 instructions and 21 shuffles a pair
// of particles with torques, where two one-sided evaluations take about 600.
// 5,120 particles with torques above the wall take 127 us a product, by tiles 214.
struct SymParams {
    const float4 *x;
    const float4 *f;
    const float4 *t;  // torques of particles [0, n6)
    float4 *partial;
    int n, n6, nb;
    long long items;
    FreeSym6 k;       // unbounded form
    float unit;       // with torques: positions and torques are multiplied by it (sym6_unit)
    const int *gate;  // may be null: nothing is done where *gate is zero
};

__device__ __forceinline__ void sym_item(long long t, int nb, int &I, int &J) {
    // t enumerates the upper triangle row by row: row I holds nb - I tiles.
    const double b = 2.0 * nb + 1.0;
    int r = static_cast<int>(floor(0.5 * (b - sqrt(fmax(0.0, b * b - 8.0 * static_cast<double>(t))))));
    r = max(0, min(r, nb - 1));
    auto start = [nb](long long row) { return row * nb - row * (row - 1) / 2; };
    while (r + 1 < nb && start(r + 1) <= t) ++r;
    while (r > 0 && start(r) > t) --r;
    I = r;
    J = r + static_cast<int>(t - start(r));
}

// Where lanes without a particle hold an inert one: far outside any system, since a pair at distance zero above the
// wall is NaN even without a force (at 1e5, as it was, a real particle could meet one).  Where the square of such a
// distance overflows, its reciprocal root is zero and the pair adds zero too.
constexpr float kFarAway = 1.0e18f;

__device__ __forceinline__ void sym_load(const SymParams &p, int idx, int lane, float4 &x, float4 &f) {
    if (idx < p.n) {
        x = p.x[idx];
        f = p.f[idx];
    } else {
        // inert padding: far from everything (and from each other), zero force
        x = make_float4(kFarAway * static_cast<float>(lane + 1), 0.0f, 1.0e4f, 0.0f);
        f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// First step of a tile against itself: its particles' neighbours along a filament come last.
constexpr int kOwnStart = 4;

// One pair of tiles.  SI, SJ: tile I, J holds particles with torques and spins (a tile that also holds others gives
// those zero torques, and their spins are dropped).
template <bool WALL, bool SCALED, bool SI, bool SJ>
__device__ __forceinline__ void sym_tiles(const SymParams &p, const FreeSym6 &k, int I, int J, int lane) {
    const unsigned full = 0xffffffffu;
    const int src_lane = (lane + 1) & 31;
    const int i = I * 32 + lane, j = J * 32 + lane;
    constexpr int NI = SI ? 6 : 3, NJ = SJ ? 6 : 3;
    float4 xi, fi4, xs, fs4;
    sym_load(p, i, lane, xi, fi4);
    sym_load(p, j, lane, xs, fs4);
    const float unit = SCALED ? p.unit : 1.0f;
    auto scale = [&](float4 &x, int q) {
        if (SCALED && q < p.n) x = make_float4(unit * x.x, unit * x.y, unit * x.z, 0.0f);
    };
    scale(xi, i);
    scale(xs, j);
    float fi[NI] = {fi4.x, fi4.y, fi4.z}, fs[NJ] = {fs4.x, fs4.y, fs4.z}, vi[NI] = {}, vs[NJ] = {};
    if constexpr (SI)
        if (i < p.n6) {
            const float4 t = p.t[i];
            fi[3] = unit * t.x;
            fi[4] = unit * t.y;
            fi[5] = unit * t.z;
        }
    if constexpr (SJ)
        if (j < p.n6) {
            const float4 t = p.t[j];
            fs[3] = unit * t.x;
            fs[4] = unit * t.y;
            fs[5] = unit * t.z;
        }
    auto rotate = [&](float &v) { v = __shfl_sync(full, v, src_lane); };
    auto rotate_source = [&] {
        rotate(xs.x);
        rotate(xs.y);
        rotate(xs.z);
#pragma unroll
        for (int c = 0; c < NJ; ++c) rotate(fs[c]);
    };
    auto pair = [&](float *vj) {
        const float dx = xi.x - xs.x, dy = xi.y - xs.y, dz = xi.z - xs.z;
        if constexpr (!SI && !SJ) {
            if constexpr (WALL) wall_pair_sym<float>(dx, dy, dz, xi.z, xs.z, wall_source(xs.z), fs, fi, vi, vj);
            else free_pair_sym<float>(dx, dy, dz, k.t, fs, fi, vi, vj);
        } else {
            if constexpr (WALL) wall_pair_sym6_f32<SI, SJ>(dx, dy, dz, xi.z, xs.z, fs, fi, vi, vj);
            else free_pair_sym6_f32<SI, SJ>(dx, dy, dz, k, fs, fi, vi, vj);
        }
    };
    auto place = [&](int q, int tile) {
        return p.partial + (q < p.n6 ? 2 * (static_cast<size_t>(q) * p.nb + tile)
                                     : static_cast<size_t>(p.n6 + q) * p.nb + tile);
    };
    auto store = [&](int q, int tile, const float *v, bool spins) {
        if (q >= p.n) return;
        float4 *o = place(q, tile);
        constexpr float scale = !SI && !SJ && WALL ? static_cast<float>(kPairScale) : 1.0f;
        const float c = !SI && !SJ && !WALL ? k.c8 : scale;  // the force-only pairs come without their factor
        o[0] = make_float4(c * v[0], c * v[1], c * v[2], 0.0f);
        if (spins && q < p.n6) o[1] = make_float4(v[3], v[4], v[5], 0.0f);
    };
    // Tiles with force-only particles form sums of 16 terms: the first half's are set aside.  (Relative L2 error against
    // FP64 in sets with 1,500 to 6,000 blobs 1.3 to 1.4e-7, the tile kernel's 1.3 to 2.1, sums of 32 1.5 to 1.8.  Between
    // particles with torques sums of 32 are nearer than the tile kernel's, 1.1 to 1.4e-7 against 1.6 to 2.2, and the
    // registers for shorter ones cost 8%.)
    constexpr bool kSplit = !(SI && SJ);
    float vi0[NI] = {}, vs0[NJ] = {};
    auto set_aside = [&] {
#pragma unroll
        for (int c = 0; c < NI; ++c) {
            vi0[c] = vi[c];
            vi[c] = 0.0f;
        }
#pragma unroll
        for (int c = 0; c < NJ; ++c) {
            vs0[c] = vs[c];
            vs[c] = 0.0f;
        }
    };
    if (I == J) {  // a filament's neighbours, the largest terms, come last: steps 4 .. 31, 1 .. 3
#pragma unroll
        for (int r = 0; r < kOwnStart; ++r) rotate_source();
#pragma unroll 1
        for (int step = kOwnStart; step < kOwnStart + 32; ++step) {
            if (kSplit && step == kOwnStart + 16) set_aside();
            float drop[NJ] = {};
            if (step != 32) pair(drop);
            rotate_source();
        }
#pragma unroll
        for (int c = 0; c < NI; ++c) vi[c] += vi0[c];
        store(i, I, vi, SI);
    } else {
#pragma unroll(SI || SJ ? 1 : 2)
        for (int step = 0; step < 32; ++step) {
            if (kSplit && step == 16) set_aside();
            pair(vs);
            rotate_source();
#pragma unroll
            for (int c = 0; c < NJ; ++c) rotate(vs[c]);
        }
#pragma unroll
        for (int c = 0; c < NI; ++c) vi[c] += vi0[c];
#pragma unroll
        for (int c = 0; c < NJ; ++c)
            if (kSplit) vs[c] += __shfl_sync(full, vs0[c], lane ^ 16);  // set aside 16 lanes from home
        store(i, J, vi, SI);
        store(j, I, vs, SJ);
    }
}

// The pair formulas with torques hold fifth powers of distances and sixth powers of the radius, which leave FP32 for
// spheres of 10 nm in metres.  Where the radius is not near 1 the kernel works in lengths of a power of two near it, and
// the reduction scales back: positions and torques times unit, then velocities times unit and spins times its square, all
// exact.  (With the powers taken apart inside the pair a product took 3 to 4% longer, with every radius scaled 1 to 2%.)
double sym6_unit(int wall, double a) {
    if (wall || (a >= 1.0e-3 && a <= 1.0e3)) return 1.0;
    return std::ldexp(1.0, -std::max(-100, std::min(100, std::ilogb(a))));
}

// The first p.n6 > 0 particles have torques and spins (5 blocks per SM for their registers).
constexpr int kSym6CtasPerSm = 5;
template <bool WALL, bool SCALED = false>
__global__ void __launch_bounds__(kThreads, kSym6CtasPerSm) rpy_sym6_kernel(SymParams p) {
    chain_wait();  // launched as a programmatic dependent of the packing launch
    if (p.gate && *p.gate == 0) return;
    const FreeSym6 &k = p.k;
    const int lane = threadIdx.x & 31;
    const long long nwarps = static_cast<long long>(gridDim.x) * (kThreads / 32);
    for (long long t = static_cast<long long>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5); t < p.items;
         t += nwarps) {
        int I, J;
        sym_item(t, p.nb, I, J);
        // uniform over the warp; J >= I, so J has torques only if I has
        if (J * 32 < p.n6) sym_tiles<WALL, SCALED, true, true>(p, k, I, J, lane);
        else if (I * 32 < p.n6) sym_tiles<WALL, SCALED, true, false>(p, k, I, J, lane);
        else sym_tiles<WALL, SCALED, false, false>(p, k, I, J, lane);
    }
}

// ---------------------------------------------------------------------------
// The same without torques, two sources a lane in packed arithmetic.  Work unit: one warp, the 32 targets of tile I
// and the 64 sources of tiles 2K and 2K + 1, K >= I / 2.  The sources lie in shared memory as packed pairs (source l of
// one tile with source l of the other), so a lane reads the pair of step s at l + s, and only the accumulators of the
// sources rotate.  In the units K = I / 2 the tile meets itself: those pairs are evaluated one-sided and a particle
// never meets itself; an odd I leaves the other half empty there.
//
// Every particle receives one partial per tile, as above, of two FP32 sums of 16 terms.  That is what the error against
// FP64 depends on: 1.0e-7 (relative L2, cilia above the wall, 600 to 7,500 segments; 1.0e-7 without a wall, 1.0 to 1.3e-7
// with blobs); 1.3, 1.3 and 1.7e-7 with one sum of 32 and the neighbours first.  Refining the reciprocal square roots did
// not change it.
//
// Bound by the FP32 pipe, at 81% of it (81 packed instructions above the wall for both directions of two pairs): a
// product of 20,480 segments takes 664 us (393 without a wall); 880 us with one source a lane and its position and force
// rotating by shuffles.  Five blocks an SM and eight steps unrolled: 678 with four blocks, 751 with sixteen steps (the
// warps are at different steps, and the loop outgrows the instruction cache), 705 with two.
constexpr int kSym3CtasPerSm = 5;
template <bool WALL>
using Sym3Smem = ulonglong2[WALL ? 4 : 3][64];

__device__ __forceinline__ void sym3_unit(long long t, int nb, int &I, int &K) {
    const int nk = (nb + 1) / 2;
    int T;
    sym_item(t >> 1, nk, T, K);
    I = 2 * T + static_cast<int>(t & 1);
}

// store(particle, tile, velocity)
template <bool WALL, class Store>
__device__ __forceinline__ void sym3_tiles(const float4 *__restrict__ x, const float4 *__restrict__ f, int n, int nb,
                                           const FreeSym &k, int I, int K, int lane, Sym3Smem<WALL> &sm, Store store) {
    if (I >= nb) return;
    const unsigned full = 0xffffffffu;
    const int src_lane = (lane + 2) & 31;
    const bool own = K == I >> 1, odd_own = own && (I & 1);
    const int i = I * 32 + lane, ja = odd_own ? i : K * 64 + lane, jb = odd_own ? n : K * 64 + 32 + lane;
    auto load = [&](int idx, float apart, float4 &xv, float4 &fv) {
        if (idx < n) {
            xv = x[idx];
            fv = f[idx];
        } else {  // inert: far from everything and from each other, no force
            xv = make_float4(kFarAway * static_cast<float>(lane + 1), apart, 1.0e4f, 0.0f);
            fv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    float4 xi, fi4, xa, fa, xb, fb;
    load(i, 0.0f, xi, fi4);
    load(ja, kFarAway, xa, fa);
    load(jb, 2.0f * kFarAway, xb, fb);
    const ulonglong2 q0 = make_ulonglong2(pack2(xa.x, xb.x).v, pack2(xa.y, xb.y).v),
                     q1 = make_ulonglong2(pack2(xa.z, xb.z).v, pack2(fa.x, fb.x).v),
                     q2 = make_ulonglong2(pack2(fa.y, fb.y).v, pack2(fa.z, fb.z).v);
    __syncwarp();  // the last unit's reads
    sm[0][lane] = sm[0][lane + 32] = q0;
    sm[1][lane] = sm[1][lane + 32] = q1;
    sm[2][lane] = sm[2][lane + 32] = q2;
    if constexpr (WALL) {
        const WallSource<F2> z = wall_source(pack2(xa.z, xb.z));
        sm[3][lane] = sm[3][lane + 32] = make_ulonglong2(z.p.v, z.q.v);
    }
    __syncwarp();
    const F2 tx = splat<F2>(xi.x), ty = splat<F2>(xi.y), tz = splat<F2>(xi.z);
    const F2 fi[3] = {splat<F2>(fi4.x), splat<F2>(fi4.y), splat<F2>(fi4.z)};
    // even and odd steps have their own sums, of 16 terms each; the sources' rotate by two lanes after each of theirs
    F2 vi_[2][3] = {}, vj_[2][3] = {};
    // step `at - lane`; the particle itself, where it comes up, is replaced by an inert one
    auto pair = [&](int at, bool self, F2 *vi, F2 *vj) {
        const ulonglong2 a = sm[0][at], b = sm[1][at], c = sm[2][at];
        F2 sx{a.x}, fj[3] = {F2{b.y}, F2{c.x}, F2{c.y}};
        const F2 sy{a.y}, sz{b.x};
        if (self) {
            sx = pack2(-kFarAway, unpack2(sx).y);
#pragma unroll
            for (int q = 0; q < 3; ++q) fj[q] = pack2(0.0f, unpack2(fj[q]).y);
        }
        const F2 dx = vsub(tx, sx), dy = vsub(ty, sy), dz = vsub(tz, sz);
        if constexpr (WALL) {
            const ulonglong2 d = sm[3][at];
            wall_pair_sym<F2>(dx, dy, dz, tz, sz, WallSource<F2>{F2{d.x}, F2{d.y}}, fj, fi, vi, vj);
        } else {
            free_pair_sym<F2>(dx, dy, dz, k, fj, fi, vi, vj);
        }
#pragma unroll
        for (int c3 = 0; c3 < 3; ++c3) vj[c3].v = __shfl_sync(full, vj[c3].v, src_lane);
    };
    if (!own) {
#pragma unroll 4
        for (int s = 0; s < 32; s += 2) {
            pair(lane + s, false, vi_[0], vj_[0]);
            pair(lane + s + 1, false, vi_[1], vj_[1]);
        }
    } else {  // a filament's neighbours, the largest terms, come last (28 .. 31, 0 .. 3); at step 0 the own tile's half
              // is the particle itself
#pragma unroll 1
        for (int t = kOwnStart; t < kOwnStart + 32; t += 2) {
            const int s = t & 31;
            pair(lane + s, s == 0, vi_[0], vj_[0]);
            pair(lane + s + 1, false, vi_[1], vj_[1]);
        }
    }
    F2 vi[3], vj[3];
    const int home = own ? kOwnStart : 0;  // the sources' sums end this far from home, the odd steps' one lane further
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vi[c] = vadd(vi_[0][c], vi_[1][c]);
        vj[c] = vadd(F2{__shfl_sync(full, vj_[0][c].v, (lane - home) & 31)},
                     F2{__shfl_sync(full, vj_[1][c].v, (lane - home - 1) & 31)});
    }
    auto lo = [](F2 a) { return unpack2(a).x; };
    auto hi = [](F2 a) { return unpack2(a).y; };
    if (i < n) {  // two partials: their sum is left to FP64
        store(i, odd_own ? I : 2 * K, make_float4(lo(vi[0]), lo(vi[1]), lo(vi[2]), 0.0f));
        if (!odd_own && 2 * K + 1 < nb) store(i, 2 * K + 1, make_float4(hi(vi[0]), hi(vi[1]), hi(vi[2]), 0.0f));
    }
    if (ja < n && !own) store(ja, I, make_float4(lo(vj[0]), lo(vj[1]), lo(vj[2]), 0.0f));
    if (jb < n) store(jb, I, make_float4(hi(vj[0]), hi(vj[1]), hi(vj[2]), 0.0f));
}

// The same sums from one source a lane: a warp takes the tiles I <= J alone, the sources and their accumulators rotate by
// shuffles.  Every operation and every order of summation is that of sym3_tiles, so the partials are the same bit for bit
// (an array's step does not depend on what else is in its batch); for launches too small to fill the SMs, where the
// latency of a unit's chain is what counts.
template <bool WALL, class Store>
__device__ __forceinline__ void sym1_tiles(const float4 *__restrict__ x, const float4 *__restrict__ f, int n,
                                           const FreeSym &k, int I, int J, int lane, Store store) {
    const unsigned full = 0xffffffffu;
    const int i = I * 32 + lane, j = J * 32 + lane;
    auto load = [&](int idx, float apart, float4 &xv, float4 &fv) {
        if (idx < n) {
            xv = x[idx];
            fv = f[idx];
        } else {
            xv = make_float4(kFarAway * static_cast<float>(lane + 1), apart, 1.0e4f, 0.0f);
            fv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    float4 xi, fi4, xs, fs;
    load(i, 0.0f, xi, fi4);
    load(j, kFarAway, xs, fs);
    const bool near = I >> 1 == J >> 1;  // the units K = I / 2: they start at kOwnStart
    const int start = near ? kOwnStart : 0;
    const F1 tx{xi.x}, ty{xi.y}, tz{xi.z}, fi[3] = {{fi4.x}, {fi4.y}, {fi4.z}};
    auto from = [&](float &v, int by) { v = __shfl_sync(full, v, (lane + by) & 31); };
    auto rotate = [&](int by) {
        from(xs.x, by);
        from(xs.y, by);
        from(xs.z, by);
        from(fs.x, by);
        from(fs.y, by);
        from(fs.z, by);
    };
    F1 vi_[2][3] = {}, vj_[2][3] = {};
    auto pair = [&](F1 *vi, F1 *vj) {
        const F1 sx{xs.x}, sy{xs.y}, sz{xs.z}, fj[3] = {{fs.x}, {fs.y}, {fs.z}};
        const F1 dx = vsub(tx, sx), dy = vsub(ty, sy), dz = vsub(tz, sz);
        if constexpr (WALL) wall_pair_sym<F1>(dx, dy, dz, tz, sz, wall_source(sz), fj, fi, vi, vj);
        else free_pair_sym<F1>(dx, dy, dz, k, fj, fi, vi, vj);
        rotate(1);
    };
    auto both = [&](F1 *vi, F1 *vj) {
        pair(vi, vj);
#pragma unroll
        for (int c = 0; c < 3; ++c) from(vj[c].v, 2);
    };
    if (near) rotate(kOwnStart);
    if (I != J) {
#pragma unroll 2
        for (int t = 0; t < 32; t += 2) {
            both(vi_[0], vj_[0]);
            both(vi_[1], vj_[1]);
        }
    } else {
#pragma unroll 1
        for (int t = kOwnStart; t < kOwnStart + 32; t += 2) {
            F1 drop[3] = {};
            if (t != 32) pair(vi_[0], drop);  // not with itself
            else rotate(1);
            pair(vi_[1], drop);
        }
    }
    F1 vi[3], vj[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        vi[c] = vadd(vi_[0][c], vi_[1][c]);
        vj[c] = vadd(F1{__shfl_sync(full, vj_[0][c].v, (lane - start) & 31)},
                     F1{__shfl_sync(full, vj_[1][c].v, (lane - start - 1) & 31)});
    }
    if (i < n) store(i, J, make_float4(vi[0].v, vi[1].v, vi[2].v, 0.0f));
    if (j < n && I != J) store(j, I, make_float4(vj[0].v, vj[1].v, vj[2].v, 0.0f));
}

template <bool WALL, bool PACKED>
__global__ void __launch_bounds__(kThreads, kSym3CtasPerSm) rpy_sym3_kernel(SymParams p) {
    __shared__ Sym3Smem<WALL> sm[PACKED ? kThreads / 32 : 1];
    chain_wait();  // launched as a programmatic dependent of the packing launch
    if (p.gate && *p.gate == 0) return;
    const FreeSym &k = p.k.t;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long nwarps = static_cast<long long>(gridDim.x) * (kThreads / 32);
    auto store = [&](int q, int slot, float4 v) { p.partial[static_cast<size_t>(q) * p.nb + slot] = v; };
    for (long long t = static_cast<long long>(blockIdx.x) * (kThreads / 32) + w; t < p.items; t += nwarps) {
        int I, K;
        if constexpr (PACKED) {
            sym3_unit(t, p.nb, I, K);
            sym3_tiles<WALL>(p.x, p.f, p.n, p.nb, k, I, K, lane, sm[w], store);
        } else {
            sym_item(t, p.nb, I, K);
            sym1_tiles<WALL>(p.x, p.f, p.n, k, I, K, lane, store);
        }
    }
}

// ---------------------------------------------------------------------------
// Batched form of the symmetric wall kernel: many independent particle sets
// (arrays) in one launch.  Work items of all arrays are concatenated; a warp
// finds its array by binary search over the arrays' first items.  Arrays whose
// `active` flag is 0 are skipped (converged GMRES systems).  Partials are
// stored slot-major per array, partial[poff + slot * n + i] (slot = the other
// tile of the pair), so that both these writes and the per-segment reduction
// that reads them are coalesced.
template <bool PACKED>
__global__ void __launch_bounds__(kThreads, kSym3CtasPerSm) rpy_wall_sym_batch_kernel(SymBatchParams p) {
    __shared__ Sym3Smem<true> sm[PACKED ? kThreads / 32 : 1];
    chain_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long nwarps = static_cast<long long>(gridDim.x) * (kThreads / 32);
    for (long long t = static_cast<long long>(blockIdx.x) * (kThreads / 32) + w; t < p.items; t += nwarps) {
        int lo = 0, hi = p.B - 1;  // last array whose first item <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (p.item0[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const int b = lo;
        if (p.active && !p.active[b]) continue;
        const int n = p.n[b], nb = p.nb[b];
        const float4 *x = p.x + p.seg0[b], *f = p.f + p.seg0[b];
        float4 *partial = p.partial + p.poff[b];
        auto store = [&](int q, int slot, float4 v) { partial[static_cast<size_t>(slot) * n + q] = v; };
        int I, K;
        if constexpr (PACKED) {
            sym3_unit(t - p.item0[b], nb, I, K);
            sym3_tiles<true>(x, f, n, nb, FreeSym{}, I, K, lane, sm[w], store);
        } else {
            sym_item(t - p.item0[b], nb, I, K);
            sym1_tiles<true>(x, f, n, FreeSym{}, I, K, lane, store);
        }
    }
}

struct ReduceParams {
    const float4 *partial;
    const float4 *xt, *ft, *tt;  // self block inputs (wall, self set)
    float *out;
    const int *err;  // may be null; when the word is non-zero every output is a quiet NaN
    int nsplit, nt, ntp, stride, mode;
};

// One warp per target: the lanes stride over the target's partials, FP64
// shuffle reduction (fixed order, deterministic), lane 0 adds the wall self
// block and writes or accumulates the result.
template <bool WALL_SELF, int VD, int FD>
__global__ void rpy_reduce_kernel(ReduceParams p) {
    chain_wait();  // launched as a programmatic dependent of the tile launch
    const int lane = threadIdx.x & 31;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= p.nt) return;
    constexpr int W = VD / 3;
    double v[VD];
#pragma unroll
    for (int c = 0; c < VD; ++c) v[c] = 0.0;
    const float4 *pt = p.partial + static_cast<size_t>(i) * p.nsplit * W;
    for (int s = lane; s < p.nsplit; s += 32) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const float4 q = pt[s * W + w];
            v[3 * w + 0] += q.x;
            v[3 * w + 1] += q.y;
            v[3 * w + 2] += q.z;
        }
    }
#pragma unroll
    for (int c = 0; c < VD; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
    if (lane != 0) return;
    if constexpr (WALL_SELF) {
        const float4 f4 = p.ft[i];
        float f[6] = {f4.x, f4.y, f4.z, 0.f, 0.f, 0.f};
        if constexpr (FD > 3) {
            const float4 t4 = p.tt[i];
            f[3] = t4.x;
            f[4] = t4.y;
            f[5] = t4.z;
        }
        float vs[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        wall_self_f32<VD, FD>(p.xt[i].z, f, vs);
#pragma unroll
        for (int c = 0; c < VD; ++c) v[c] += vs[c];
    }
    float *o = p.out + static_cast<size_t>(i) * p.stride;
    if (p.err && *p.err) {
        // A tile block gave up waiting and left its partials unwritten: poison
        // the result instead of summing stale partials.
        for (int c = 0; c < p.stride; ++c) o[c] = __int_as_float(0x7fc00000);
        return;
    }
    if (p.mode == kOutAdd) {
#pragma unroll
        for (int c = 0; c < VD; ++c) o[c] = static_cast<float>(static_cast<double>(o[c]) + v[c]);
    } else {
#pragma unroll
        for (int c = 0; c < VD; ++c) o[c] = static_cast<float>(v[c]);
        for (int c = VD; c < p.stride; ++c) o[c] = 0.0f;
    }
}

// The same for a whole set after the symmetric kernel: segments [0, n_seg) into out (stride 6), blobs into out_b
// (stride 3); the self blocks, which that kernel leaves out, are added here.
struct SetReduceParams {
    const float4 *partial, *x, *f, *t;
    float *out, *out_b;
    int n, n_seg, n6, nb;
    float self_t, self_r;  // unbounded: 1 / (6 pi mu a), 1 / (8 pi mu a^3)
    double scale, spin_scale;  // of the partials' velocities and spins
};
template <bool WALL>
__global__ void __launch_bounds__(256) rpy_set_reduce_kernel(SetReduceParams p) {
    chain_wait();
    const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= p.n) return;
    const bool six = i < p.n6;
    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (six) {
        const float4 *pt = p.partial + 2 * static_cast<size_t>(i) * p.nb;
        for (int s = lane; s < p.nb; s += 32) {
            const float4 a = __ldcs(pt + 2 * s), b = __ldcs(pt + 2 * s + 1);
            v[0] += a.x;
            v[1] += a.y;
            v[2] += a.z;
            v[3] += b.x;
            v[4] += b.y;
            v[5] += b.z;
        }
    } else {
        const float4 *pt = p.partial + static_cast<size_t>(p.n6 + i) * p.nb;
        for (int s = lane; s < p.nb; s += 32) {
            const float4 a = __ldcs(pt + s);
            v[0] += a.x;
            v[1] += a.y;
            v[2] += a.z;
        }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        if (c >= 3 && !six) continue;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
    }
    if (lane != 0) return;
    for (int c = 0; c < 6; ++c) v[c] *= c < 3 ? p.scale : p.spin_scale;
    const float4 f4 = p.f[i];
    float f[6] = {f4.x, f4.y, f4.z, 0.f, 0.f, 0.f}, vs[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (six) {
        const float4 t4 = p.t[i];
        f[3] = t4.x;
        f[4] = t4.y;
        f[5] = t4.z;
    }
    if constexpr (WALL) {
        if (six) wall_self_f32<6, 6>(p.x[i].z, f, vs);
        else wall_self_f32<3, 3>(p.x[i].z, f, vs);
    } else {
        for (int c = 0; c < 3; ++c) {
            vs[c] = p.self_t * f[c];
            vs[3 + c] = p.self_r * f[3 + c];
        }
    }
    if (i < p.n_seg) {
        float *o = p.out + 6 * static_cast<size_t>(i);
#pragma unroll
        for (int c = 0; c < 6; ++c) o[c] = (c < 3 || six) ? static_cast<float>(v[c] + vs[c]) : 0.0f;
    } else {
        float *o = p.out_b + 3 * static_cast<size_t>(i - p.n_seg);
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c] = static_cast<float>(v[c] + vs[c]);
    }
}

// Small sets of force-only particles, one launch: four warps per target, their lanes over the sources (FP32 sums of at
// most kRpyDirectMax / 128 terms a lane, then FP64), reading and writing the callers' layouts.  What it saves is the
// packing, the partials and two launches; what it costs is evaluating each pair twice, so it stops paying where the
// pairs outweigh the launches: above the wall 320 particles take 2.9 us, 7.9 by the symmetric kernel; 1,020 6.6 and
// 8.5; 1,520 12.0 and 11.0 (without a wall 2.7 and 7.9, 4.9 and 7.9, 8.0 and 9.6, and at 2,040 13.3 and 10.9).  Bound
// by the latency of a lane's chain of pairs: with one warp per target it was 6.0 us at 320, 10.4 at 640.
constexpr int kDirectWarps = 4;  // the last sum below is written for four
struct DirectParams {
    const float *xs, *fs, *xb, *fb;
    float *vs, *vb;
    float4 *x4, *f4;  // the particles' records, written for the evaluations that follow on the handle
    int ns, n;
    FreeSym k;
    float self_t;
    double scale;
};
template <bool WALL>
__global__ void __launch_bounds__(256) rpy_direct_kernel(DirectParams p) {
    constexpr int kLanes = 32 * kDirectWarps;
    __shared__ double part[256 / 32][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, rank = threadIdx.x % kLanes;
    const int target = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes, i = min(target, p.n - 1);
    auto position = [&](int q) { return q < p.ns ? p.xs + 3 * q : p.xb + 3 * (q - p.ns); };
    auto force = [&](int q) { return q < p.ns ? p.fs + 6 * q : p.fb + 3 * (q - p.ns); };
    const float *xi = position(i);
    const float x = xi[0], y = xi[1], z = xi[2];
    float v[3] = {0.0f, 0.0f, 0.0f};
    const float none[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 2
    for (int j = rank; j < p.n; j += kLanes) {
        const float *xj = position(j), *fj = force(j);
        const float f[3] = {fj[0], fj[1], fj[2]};
        const float px = xj[0], py = xj[1], pz = xj[2];
        if (j == i) continue;
        float drop[3] = {0.0f, 0.0f, 0.0f};
        if constexpr (WALL) wall_pair_sym<float>(x - px, y - py, z - pz, z, pz, wall_source(pz), f, none, v, drop);
        else free_pair_sym<float>(x - px, y - py, z - pz, p.k, f, none, v, drop);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double s = v[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) part[w][c] = s;
    }
    __syncthreads();
    if (rank != 0 || target >= p.n) return;
    const float *fi = force(i);
    const float f[3] = {fi[0], fi[1], fi[2]};
    p.x4[i] = make_float4(x, y, z, 0.0f);
    p.f4[i] = make_float4(f[0], f[1], f[2], 0.0f);
    float self[3] = {0.0f, 0.0f, 0.0f};
    if constexpr (WALL) wall_self_f32<3, 3>(z, f, self);
    else
        for (int c = 0; c < 3; ++c) self[c] = p.self_t * f[c];
    float *o = i < p.ns ? p.vs + 6 * static_cast<size_t>(i) : p.vb + 3 * static_cast<size_t>(i - p.ns);
    for (int c = 0; c < 3; ++c)
        o[c] = static_cast<float>(((part[w][c] + part[w + 1][c]) + (part[w + 2][c] + part[w + 3][c])) * p.scale + self[c]);
    if (i < p.ns)
        for (int c = 3; c < 6; ++c) o[c] = 0.0f;
}

__global__ void pack_xyz_kernel(const float *__restrict__ a, float4 *__restrict__ o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) o[i] = make_float4(a[3 * i], a[3 * i + 1], a[3 * i + 2], 0.0f);
}

__global__ void pack_ft6_kernel(const float *__restrict__ a, float4 *__restrict__ f, float4 *__restrict__ t,
                                int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        f[i] = make_float4(a[6 * i], a[6 * i + 1], a[6 * i + 2], 0.0f);
        if (t) t[i] = make_float4(a[6 * i + 3], a[6 * i + 4], a[6 * i + 5], 0.0f);
    }
}

// Positions and forces (+ torques) of one particle set in one launch.
__global__ void pack_set_kernel(const float *__restrict__ x, const float *__restrict__ ft, float4 *__restrict__ xo,
                                float4 *__restrict__ fo, float4 *__restrict__ to, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        xo[i] = make_float4(x[3 * i], x[3 * i + 1], x[3 * i + 2], 0.0f);
        fo[i] = make_float4(ft[6 * i], ft[6 * i + 1], ft[6 * i + 2], 0.0f);
        if (to) to[i] = make_float4(ft[6 * i + 3], ft[6 * i + 4], ft[6 * i + 5], 0.0f);
    }
}

// Segments, then blobs, of a mobility handle in one launch.
__global__ void pack_sets_kernel(const float *__restrict__ xs, const float *__restrict__ fs, const float *__restrict__ xb,
                                 const float *__restrict__ fb, int n_seg, int n, float4 *__restrict__ xo,
                                 float4 *__restrict__ fo, float4 *__restrict__ to) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *x, *f;
    if (i < n_seg) {
        x = xs + 3 * static_cast<size_t>(i);
        f = fs + 6 * static_cast<size_t>(i);
        to[i] = make_float4(f[3], f[4], f[5], 0.0f);
    } else {
        x = xb + 3 * static_cast<size_t>(i - n_seg);
        f = fb + 3 * static_cast<size_t>(i - n_seg);
    }
    xo[i] = make_float4(x[0], x[1], x[2], 0.0f);
    fo[i] = make_float4(f[0], f[1], f[2], 0.0f);
}

// Raises the dynamic shared-memory cap of one instantiation once per device.
// Called before any launch (and therefore before any stream capture).
template <bool WALL, int VD, int FD, int TI, bool SELF>
int configure_tiles_t() {
    auto kern = rpy_tile_kernel<WALL, VD, FD, TI, SELF>;
    static bool configured[64] = {};
    int dev = 0;
    CF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        CF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 + 3 * kMaxSplit * 16));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return CF_OK;
}

template <bool WALL, int VD, int FD, int TI, bool SELF>
int launch_tiles_t(const RpyBlockDesc &d, const RpyPlan &plan, float4 *scratch, int *dev_err,
                   cudaStream_t st) {
    auto kern = rpy_tile_kernel<WALL, VD, FD, TI, SELF>;
    CF_TRY((configure_tiles_t<WALL, VD, FD, TI, SELF>()));
    TileParams p;
    p.xt = d.xt;
    p.xs = d.xs;
    p.fs = d.fs;
    p.ts = d.ts;
    p.partial = scratch;
    p.nt = d.nt;
    p.ns = d.ns;
    p.split = plan.split;
    p.ntp = d.nt;
    p.at = d.at;
    p.as = d.as;
    p.inv_mu = 1.0f / d.mu;
    p.err = dev_err;
    p.wait_limit = rpy_wait_limit();
    dim3 grid(plan.tiles, plan.nsplit);
    CF_CUDA(launch_chained(kern, grid, dim3(kThreads), plan.smem, st, p));
    CF_CHECK_LAUNCH("rpy_tile_kernel");
    return CF_OK;
}

template <bool WALL, int VD, int FD, bool SELF>
int dispatch_ti(const RpyBlockDesc &d, const RpyPlan &plan, float4 *scratch, int *dev_err, cudaStream_t st) {
    if (plan.ti == 2) return launch_tiles_t<WALL, VD, FD, 2, SELF>(d, plan, scratch, dev_err, st);
    return launch_tiles_t<WALL, VD, FD, 1, SELF>(d, plan, scratch, dev_err, st);
}

template <bool WALL, bool SELF>
int dispatch_dof(const RpyBlockDesc &d, const RpyPlan &plan, float4 *scratch, int *dev_err, cudaStream_t st) {
    if (d.vd == 3 && d.fd == 3) return dispatch_ti<WALL, 3, 3, SELF>(d, plan, scratch, dev_err, st);
    if (d.vd == 6 && d.fd == 6) return dispatch_ti<WALL, 6, 6, SELF>(d, plan, scratch, dev_err, st);
    if (d.vd == 6 && d.fd == 3) return dispatch_ti<WALL, 6, 3, SELF>(d, plan, scratch, dev_err, st);
    if (d.vd == 3 && d.fd == 6) return dispatch_ti<WALL, 3, 6, SELF>(d, plan, scratch, dev_err, st);
    return set_error(CF_EINVAL, "rpy: unsupported dof pair %d/%d", d.vd, d.fd);
}

template <bool WS, int VD, int FD>
int launch_reduce_t(const ReduceParams &p, cudaStream_t st) {
    const int threads = 256;  // 8 targets per block
    const int blocks = (p.nt + 7) / 8;
    CF_CUDA(launch_chained(rpy_reduce_kernel<WS, VD, FD>, dim3(blocks), dim3(threads), 0, st, p));
    CF_CHECK_LAUNCH("rpy_reduce_kernel");
    return CF_OK;
}

}  // namespace

RpyPlan rpy_plan_sym(int n, int n6, int num_sms) {
    RpyPlan pl{};
    pl.sym = 1;
    pl.n6 = n6;
    pl.ti = 1;
    const int nb = std::max(1, (n + 31) / 32);
    pl.nb = nb;
    pl.packed = n6 == 0 && rpy_sym_packed(rpy_sym_items(nb, false), num_sms);
    pl.items = rpy_sym_items(nb, pl.packed);
    const int per_sm = n6 > 0 ? kSym6CtasPerSm : kSym3CtasPerSm;
    const long long max_warps = static_cast<long long>(std::max(1, num_sms)) * per_sm * (kThreads / 32);
    const long long per_warp = (pl.items + max_warps - 1) / max_warps;  // balanced: every warp does per_warp items
    const long long warps = (pl.items + per_warp - 1) / per_warp;
    pl.grid = static_cast<int>((warps + (kThreads / 32) - 1) / (kThreads / 32));
    pl.tiles = pl.grid;
    pl.nsplit = nb;  // partials per target
    pl.split = 32;
    pl.smem = 0;
    pl.scratch_float4 = static_cast<size_t>(nb) * std::max(n + n6, 1);
    return pl;
}

// Without torques the symmetric kernel serves every set.  With them it was faster at every size measured (320
// particles above the wall 11.3 us, by tiles 18.5; 1,000: 11.9 and 20.2; 5,120: 127 and 214; without a wall 9.7 and
// 20.9, 9.7 and 22.4, 71 and 102); sets below kSym6MinParticles stay with the tile kernel, whose bounded wait for its
// bulk copies is what their callers see as CF_TIMEOUT.
// One partial per particle and tile is n^2 / 2 bytes (twice that with torques): sets whose partials would pass 4 GB stay
// with the tile kernel, except the 3x3 product of one set.
constexpr int kSym6MinParticles = 512;
constexpr size_t kSetMaxPartials = static_cast<size_t>(1) << 28;
bool rpy_set_symmetric(int n, int n6) {
    return (n6 == 0 || n >= kSym6MinParticles) && static_cast<size_t>((n + 31) / 32) * (n + n6) <= kSetMaxPartials;
}

RpyPlan rpy_plan(int nt, int ns, int vd, int fd, int num_sms) {
    return rpy_plan_capped(nt, ns, vd, fd, num_sms, 1 << 30);
}

RpyPlan rpy_plan_capped(int nt, int ns, int vd, int fd, int num_sms, int max_nsplit) {
    // Every CTA does the same work (128*TI targets x `split` sources), so the
    // kernel time is (waves) x (time of one CTA).  Choose the split count that
    // minimises waves * (split + staging overhead), with the resident CTA count
    // per SM bounded by the launch bounds (8) and by shared memory.
    RpyPlan pl{};
    pl.ti = (vd == 3) ? 2 : 1;
    const int per_cta = kThreads * pl.ti;
    pl.tiles = std::max(1, (nt + per_cta - 1) / per_cta);
    const int sms = std::max(1, num_sms);
    const size_t src_bytes = sizeof(float4) * (fd > 3 ? 3 : 2);
    const int nmin = std::max(1, (ns + kMaxSplit - 1) / kMaxSplit);
    const int nmax = std::max(nmin, std::min(std::min(ns / kMinSplit, 8 * sms), max_nsplit));
    int best_nsplit = nmin;
    double best_cost = 1e300;
    for (int cand = nmin; cand <= nmax; ++cand) {
        const int split = std::max(1, (ns + cand - 1) / cand);
        const int nsplit = std::max(1, (ns + split - 1) / split);
        const size_t smem = 16 + static_cast<size_t>(split) * src_bytes;
        const int cap = std::min<int>(kCtasPerSm, static_cast<int>((227u * 1024u) / (smem + 1024u)));
        if (cap < 1) continue;
        const long long slots = static_cast<long long>(sms) * cap;
        const long long ctas = static_cast<long long>(pl.tiles) * nsplit;
        const long long waves = (ctas + slots - 1) / slots;
        // fewer than 4 resident CTAs (16 warps) per SM issues poorly: penalise
        const double occ = cap >= 4 ? 1.0 : 4.0 / cap;
        const double cost = static_cast<double>(waves) * (split + kStageCost) * occ;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best_nsplit = nsplit;
        }
    }
    pl.split = std::max(1, (ns + best_nsplit - 1) / best_nsplit);
    pl.nsplit = std::max(1, (ns + pl.split - 1) / pl.split);
    pl.smem = 16 + static_cast<size_t>(pl.split) * src_bytes;
    pl.scratch_float4 = static_cast<size_t>(pl.nsplit) * (vd / 3) * std::max(nt, 1);
    return pl;
}

size_t rpy_scratch_float4(int nt_max, int ns_max, int vd, int num_sms) {
    // The partial count is nsplit*nt; nsplit*tiles is bounded by the CTA target
    // or by the split caps, so take the maximum over both regimes.
    size_t best = 0;
    for (int fd : {3, 6}) {
        RpyPlan pl = rpy_plan(nt_max, ns_max, vd, fd, num_sms);
        best = std::max(best, pl.scratch_float4);
    }
    return best;
}

int rpy_launch_tiles(const RpyBlockDesc &d, const RpyPlan &plan, float4 *scratch, int *dev_err,
                     cudaStream_t st) {
    if (d.nt <= 0) return CF_OK;
    if (plan.sym) {
        SymParams p;
        p.x = d.xs;
        p.f = d.fs;
        p.partial = scratch;
        p.n = d.nt;
        p.nb = plan.nb;
        p.items = plan.items;
        const double unit = plan.n6 ? sym6_unit(d.wall, d.at) : 1.0;
        p.unit = static_cast<float>(unit);
        p.k = d.wall ? FreeSym6{} : free_sym6(d.at * unit, d.mu);
        p.gate = d.gate;
        p.t = d.ts;
        p.n6 = plan.n6;
        auto kern = d.wall ? (plan.n6 ? rpy_sym6_kernel<true>
                                      : plan.packed ? rpy_sym3_kernel<true, true> : rpy_sym3_kernel<true, false>)
                           : (plan.n6 ? rpy_sym6_kernel<false>
                                      : plan.packed ? rpy_sym3_kernel<false, true> : rpy_sym3_kernel<false, false>);
        if (unit != 1.0) kern = rpy_sym6_kernel<false, true>;
        CF_CUDA(launch_chained(kern, dim3(plan.grid), dim3(kThreads), 0, st, p));
        CF_CHECK_LAUNCH("rpy_sym kernel");
        return CF_OK;
    }
    const bool self = d.self_set != 0;
    if (d.wall) return self ? dispatch_dof<true, true>(d, plan, scratch, dev_err, st)
                            : dispatch_dof<true, false>(d, plan, scratch, dev_err, st);
    // Unbounded blocks need no mask: r = 0 is handled by the containment branch.
    return dispatch_dof<false, false>(d, plan, scratch, dev_err, st);
}

int rpy_prepare(const RpyBlockDesc &d, const RpyPlan &plan) {
    if (plan.sym) return CF_OK;  // no dynamic shared memory
    const bool self = d.self_set != 0;
    if (d.wall && self) {
        if (d.vd == 3 && d.fd == 3) return plan.ti == 2 ? configure_tiles_t<true, 3, 3, 2, true>() : configure_tiles_t<true, 3, 3, 1, true>();
        if (d.vd == 6 && d.fd == 6) return plan.ti == 2 ? configure_tiles_t<true, 6, 6, 2, true>() : configure_tiles_t<true, 6, 6, 1, true>();
    }
    return CF_OK;  // other instantiations configure themselves on first launch
}

int rpy_launch_reduce_f32(const RpyBlockDesc &d, const RpyPlan &plan, const float4 *scratch, float *out_f,
                          int stride, int mode, cudaStream_t st, const int *dev_err) {
    if (plan.sym) return set_error(CF_EINVAL, "rpy: a symmetric plan's partials are not a block's");
    if (d.nt <= 0) return CF_OK;
    ReduceParams p;
    p.partial = scratch;
    p.err = dev_err;
    p.xt = d.xt;
    p.ft = d.fs;
    p.tt = d.ts;
    p.out = out_f;
    p.nsplit = d.ns > 0 ? plan.nsplit : 0;
    p.nt = d.nt;
    p.ntp = d.nt;
    p.stride = stride;
    p.mode = mode;
    const bool ws = d.wall && d.self_set;
    if (d.vd == 3 && d.fd == 3) return ws ? launch_reduce_t<true, 3, 3>(p, st) : launch_reduce_t<false, 3, 3>(p, st);
    if (d.vd == 6 && d.fd == 6) return ws ? launch_reduce_t<true, 6, 6>(p, st) : launch_reduce_t<false, 6, 6>(p, st);
    if (d.vd == 6 && d.fd == 3) return ws ? launch_reduce_t<true, 6, 3>(p, st) : launch_reduce_t<false, 6, 3>(p, st);
    if (d.vd == 3 && d.fd == 6) return ws ? launch_reduce_t<true, 3, 6>(p, st) : launch_reduce_t<false, 3, 6>(p, st);
    return set_error(CF_EINVAL, "rpy: unsupported dof pair %d/%d", d.vd, d.fd);
}

int rpy_direct_product(int wall, const float *x_segs, const float *f_segs, const float *x_blobs, const float *f_blobs,
                       int n_seg, int n_blob, float a, float mu, float *v_segs, float *v_blobs, float4 *x, float4 *force,
                       cudaStream_t st) {
    DirectParams p{x_segs, f_segs, x_blobs, f_blobs, v_segs, v_blobs, x, force, n_seg, n_seg + n_blob};
    if (!wall) {
        p.k = free_sym(a);
        p.self_t = static_cast<float>(1.0 / (6.0 * 3.14159265358979323846 * mu * a));
    }
    p.scale = kPairScale / (wall ? 1.0 : mu);
    if (p.n <= 0) return CF_OK;
    const int per_block = 256 / (32 * kDirectWarps), blocks = (p.n + per_block - 1) / per_block;
    if (wall) rpy_direct_kernel<true><<<blocks, 256, 0, st>>>(p);
    else rpy_direct_kernel<false><<<blocks, 256, 0, st>>>(p);
    CF_CHECK_LAUNCH("rpy_direct_kernel");
    return CF_OK;
}

int pack_xyz_to_float4(const float *aos3, float4 *out, int n, cudaStream_t st) {
    if (n <= 0) return CF_OK;
    pack_xyz_kernel<<<(n + 255) / 256, 256, 0, st>>>(aos3, out, n);
    CF_CHECK_LAUNCH("pack_xyz_kernel");
    return CF_OK;
}

int pack_set_to_float4(const float *aos3, const float *aos6, float4 *x, float4 *force, float4 *torque, int n,
                       cudaStream_t st) {
    if (n <= 0) return CF_OK;
    pack_set_kernel<<<(n + 255) / 256, 256, 0, st>>>(aos3, aos6, x, force, torque, n);
    CF_CHECK_LAUNCH("pack_set_kernel");
    return CF_OK;
}

int pack_sets_to_float4(const float *x_segs, const float *f_segs, const float *x_blobs, const float *f_blobs, int n_seg,
                        int n_blob, float4 *x, float4 *force, float4 *torque, cudaStream_t st) {
    const int n = n_seg + n_blob;
    if (n <= 0) return CF_OK;
    pack_sets_kernel<<<(n + 127) / 128, 128, 0, st>>>(x_segs, f_segs, x_blobs, f_blobs, n_seg, n, x, force, torque);
    CF_CHECK_LAUNCH("pack_sets_kernel");
    return CF_OK;
}

int pack_ft6_to_float4(const float *aos6, float4 *force, float4 *torque, int n, cudaStream_t st) {
    if (n <= 0) return CF_OK;
    pack_ft6_kernel<<<(n + 255) / 256, 256, 0, st>>>(aos6, force, torque, n);
    CF_CHECK_LAUNCH("pack_ft6_kernel");
    return CF_OK;
}

RpyPlan rpy_plan_for(const RpyBlockDesc &d, int num_sms) {
    const bool itself = d.nt == d.ns && d.xt == d.xs && (d.wall ? d.self_set != 0 : d.at == d.as);  // equal spheres
    const int n6 = d.vd == 6 ? d.nt : 0;
    if (itself && d.vd == d.fd && (n6 == 0 || rpy_set_symmetric(d.nt, n6))) return rpy_plan_sym(d.nt, n6, num_sms);
    return rpy_plan(d.nt, d.ns, d.vd, d.fd, num_sms);
}

int rpy_set_product(const RpySetDesc &s, float4 *scratch, size_t scratch_cap, float *v_segs, float *v_blobs, int num_sms,
                    cudaStream_t st) {
    RpyBlockDesc d{};
    d.wall = s.wall;
    d.vd = d.fd = 3;
    d.self_set = 1;
    d.xt = d.xs = s.x;
    d.nt = d.ns = s.n;
    d.at = d.as = s.a;
    d.fs = s.f;
    d.ts = s.t;
    d.mu = s.mu;
    const int n6 = s.seg_dof == 6 ? s.n_seg : 0;
    const RpyPlan plan = rpy_plan_sym(s.n, n6, num_sms);
    if (plan.scratch_float4 > scratch_cap)
        return set_error(CF_EINVAL, "rpy: scratch too small (%zu < %zu float4)", scratch_cap, plan.scratch_float4);
    CF_TRY(rpy_launch_tiles(d, plan, scratch, nullptr, st));
    SetReduceParams p;
    p.partial = scratch;
    p.x = s.x;
    p.f = s.f;
    p.t = s.t;
    p.out = v_segs;
    p.out_b = v_blobs;
    p.n = s.n;
    p.n_seg = s.n_seg;
    p.n6 = n6;
    p.nb = plan.nb;
    const double pi = 3.14159265358979323846;
    p.self_t = static_cast<float>(1.0 / (6.0 * pi * s.mu * s.a));
    p.self_r = static_cast<float>(1.0 / (8.0 * pi * s.mu * s.a * s.a * s.a));
    const double unit = sym6_unit(s.wall, s.a);
    p.scale = n6 ? unit : kPairScale / (s.wall ? 1.0 : s.mu);
    p.spin_scale = unit * unit;
    auto kern = s.wall ? rpy_set_reduce_kernel<true> : rpy_set_reduce_kernel<false>;
    CF_CUDA(launch_chained(kern, dim3((s.n + 7) / 8), dim3(256), 0, st, p));
    CF_CHECK_LAUNCH("rpy_set_reduce_kernel");
    return CF_OK;
}

int rpy_block_product(const RpyBlockDesc &d, float4 *scratch, size_t scratch_cap, int *dev_err, float *out_f,
                      int stride, int mode, int num_sms, cudaStream_t st) {
    if (d.nt <= 0) return CF_OK;
    RpyPlan plan = rpy_plan_for(d, num_sms);
    if (plan.sym && plan.scratch_float4 > scratch_cap) plan = rpy_plan(d.nt, d.ns, d.vd, d.fd, num_sms);
    if (plan.scratch_float4 > scratch_cap)
        return set_error(CF_EINVAL, "rpy: scratch too small (%zu < %zu float4)", scratch_cap, plan.scratch_float4);
    if (plan.sym && mode == kOutWrite && (stride == 6 || (stride == 3 && d.vd == 3))) {
        const bool segs = stride == 6;
        RpySetDesc s{d.wall, d.vd, segs ? d.nt : 0, d.nt, d.xs, d.fs, d.ts, d.as, d.mu};
        return rpy_set_product(s, scratch, scratch_cap, segs ? out_f : nullptr, segs ? nullptr : out_f, num_sms, st);
    }
    if (plan.sym) {  // accumulating self products do not occur; the general kernel serves them
        plan = rpy_plan(d.nt, d.ns, d.vd, d.fd, num_sms);
        if (plan.scratch_float4 > scratch_cap)
            return set_error(CF_EINVAL, "rpy: scratch too small (%zu < %zu float4)", scratch_cap, plan.scratch_float4);
    }
    if (d.ns > 0) CF_TRY(rpy_launch_tiles(d, plan, scratch, dev_err, st));
    return rpy_launch_reduce_f32(d, plan, scratch, out_f, stride, mode, st, dev_err);
}

}  // namespace cufil

namespace {
std::atomic<unsigned> g_wait_limit{cufil::kMbarSpinLimit};
}

namespace cufil {

unsigned rpy_wait_limit() { return g_wait_limit.load(std::memory_order_relaxed); }

}  // namespace cufil

// Test hook: sets the tries of the first bounded wait of later tile launches
// (0: give up at once); a value above the default is clamped to it.
extern "C" int cf_set_wait_limit(unsigned limit) {
    cufil::clear_error();
    g_wait_limit.store(limit < cufil::kMbarSpinLimit ? limit : cufil::kMbarSpinLimit, std::memory_order_relaxed);
    return CF_OK;
}

namespace cufil {

int rpy_launch_sym_batch(const SymBatchParams &p, int grid, cudaStream_t st) {
    if (p.items <= 0) return CF_OK;
    auto kern = p.packed ? rpy_wall_sym_batch_kernel<true> : rpy_wall_sym_batch_kernel<false>;
    CF_CUDA(launch_chained(kern, dim3(grid), dim3(kThreads), 0, st, p));
    return CF_OK;
}

}  // namespace cufil
