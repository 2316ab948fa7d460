// patch_kernels.cuh -- line-patch block-Jacobi preconditioner of the implicit step.
//
// Filaments are grouped into patches of up to P neighbours along a lattice
// line in the beat direction (the beat plane of the wall frame is y-z, so a
// patch is a run of filaments with equal x, consecutive in y).  Each patch's
// saddle-point block
//     [ M_pp   -K_p ]      M_pp : wall RPY mobility of all segments of the patch
//     [ -K_p^T   0  ]      K_p  : velocity directions (K_phase, K_angle) per filament
// -- the same operator as system_matrix_mult_new (mobility_solver.cpp:1887-2105)
// restricted to the patch -- is assembled in FP32 and inverted in place by a
// blocked Gauss-Jordan elimination without pivoting, in per-filament order
// ([3*nseg lambda | phase rate | angle rate] per filament): every 62-unknown
// filament block is eliminated lambda-first, so the rate pivots are Schur
// complements -k^T M^-1 k and stay away from zero.  The elimination is the
// symmetric sweep (every intermediate matrix stays symmetric), so only the upper
// block triangle is updated and the result is -A_pp^-1.  The preconditioner is
// P^-1 r = blockdiag(A_pp^-1) r; it replaces apply_preconditioner_new
// (mobility_solver.cpp:1102-1243), whose block-diagonal form (6 pi a on the
// forces, a 2x2 Schur solve for the rates) remains the fallback of any patch
// whose inverse is not finite.  The GMRES residual is always formed with the
// exact operator, so the patch inverses change only the iteration count.
//
// Cost: one refresh is sum_p n_p^3 FP32 FMAs (n_p = 62 * filaments), done as
// ceil(n/64) rounds of (a) inverting the 64x64 pivot block (one block per
// patch), (b) scaling the pivot rows and saving the pivot columns (one thread
// per column) and (c) a rank-64 update of the matrix in 64x64 tiles.  One application is a dense n_p x n_p product per
// patch, reading the FP32 inverses once.
#pragma once

#include "rpy_pairs.cuh"
#include "sim_kernels.cuh"
#include "tc_tf32.cuh"

namespace cufil {

constexpr int kGjBlock = 64;  // pivot block of the Gauss-Jordan rounds
constexpr int kGjTile = 64;   // tile of the rank-64 updates

struct PatchDev {
    int np;                  // patches
    int nbf;                 // unknowns per filament (3*nseg + rate rows)
    int max_n;               // largest patch system
    int T;                   // 64-wide tiles per side of the largest patch
    const int *fil0;         // first entry of each patch in `fils` [np]
    const int *nf;           // filaments per patch [np]
    const int *fils;         // filament ids (batch numbering), patch by patch
    const long long *moff;   // first float of each patch matrix [np]
    const long long *roff;   // first entry of each patch in `rows` [np]
    const long long *rows;   // batch-vector row of each local unknown
    float *A;                // patch matrices, then their inverses (row-major n x n, row stride patch_ld(n))
    // Round operands of the tile update, per patch and 64-column tile, split for the tensor cores
    // (tc_tf32.cuh: a TF32 high part and an FP32 remainder, 4096 floats each, canonical K-major
    // layout with k the pivot row s and m or n the tile column c):
    float *csplit;           // the pivot-row copies U[s][c], [np][T][2][4096]
    float *rsplit;           // the scaled pivot rows (D^-1 U)[s][c] (-D^-1 in the pivot columns), same shape
    float *dinv;             // inverted pivot blocks, [np][kGjBlock][kGjBlock]
    int *ok;                 // [np] 1 when the inverse is finite
    int *counter;            // per-round tile counters of the update [rounds]
};

// Row stride of a patch system of n unknowns: rows start on 16 bytes, so tiles
// move in 16-byte copies.  The padding columns [n, ld) are never part of a result.
__host__ __device__ __forceinline__ int patch_ld(int n) { return (n + 3) & ~3; }

// Mobility entries: one thread per (target segment, source segment) pair of a
// patch; writes the 3x3 block into the lambda rows / columns.
__global__ void patch_mobility_kernel(SimDev d, PatchDev P) {
    const int p = blockIdx.y;
    const int nfp = P.nf[p];
    const int ns = nfp * d.nseg;
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= static_cast<long long>(ns) * ns) return;
    const int si = static_cast<int>(t / ns), sj = static_cast<int>(t - static_cast<long long>(si) * ns);
    const int ai = si / d.nseg, ki = si - ai * d.nseg;
    const int aj = sj / d.nseg, kj = sj - aj * d.nseg;
    const int gi = P.fils[P.fil0[p] + ai] * d.nseg + ki;
    const int gj = P.fils[P.fil0[p] + aj] * d.nseg + kj;
    const int ld = patch_ld(nfp * P.nbf);
    float *A = P.A + P.moff[p];
    const long long r0 = static_cast<long long>(ai) * P.nbf + 3 * ki;
    const long long c0 = static_cast<long long>(aj) * P.nbf + 3 * kj;
    if (r0 / kGjTile > (c0 + 2) / kGjTile) return;  // wholly in the lower block triangle, which the sweep never reads
    const float zi = static_cast<float>(d.xd[3 * gi + 2]);
    for (int c = 0; c < 3; ++c) {
        float f[3] = {0.0f, 0.0f, 0.0f}, v[3] = {0.0f, 0.0f, 0.0f};
        f[c] = 1.0f;
        if (gi == gj) {
            wall_self_f32<3, 3>(zi, f, v);
        } else {
            const float dx = static_cast<float>(d.xd[3 * gi] - d.xd[3 * gj]);
            const float dy = static_cast<float>(d.xd[3 * gi + 1] - d.xd[3 * gj + 1]);
            const float dz = static_cast<float>(d.xd[3 * gi + 2] - d.xd[3 * gj + 2]);
            wall_pair_f32<3, 3>(dx, dy, dz, zi, static_cast<float>(d.xd[3 * gj + 2]), f, v);
        }
        for (int q = 0; q < 3; ++q)  // the sweep reads the upper block triangle only
            if ((r0 + q) / kGjTile <= (c0 + c) / kGjTile) A[(r0 + q) * ld + c0 + c] = v[q];
    }
}

// Rate rows and columns of a patch: -K / -K^T of each filament, zero between
// filaments and between rates.  grid = (entry chunks, patches).
__global__ void patch_rates_kernel(SimDev d, PatchDev P) {
    const int p = blockIdx.y;
    const int nfp = P.nf[p];
    const int n = nfp * P.nbf, ld = patch_ld(n);
    const int nl = 3 * d.nseg, nr = P.nbf - nl;  // lambda rows and rate rows per filament
    float *A = P.A + P.moff[p];
    // every (row, rate column) entry and its transpose: -k of the row's own filament, zero elsewhere (the
    // matrix is not cleared between rebuilds: the lambda block is assembled in full, and this covers the rest)
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * nfp * nr; e += gridDim.x * blockDim.x) {
        const int rc = e / n, r = e - rc * n;
        const int a = rc / nr, q = rc - a * nr;  // rate column: filament a, rate q (phase first)
        const int c = a * P.nbf + nl + q;
        const int ar = r / P.nbf, li = r - ar * P.nbf;
        float v = 0.0f;
        if (ar == a && li < nl) {
            const int g3 = 3 * P.fils[P.fil0[p] + a] * d.nseg + li;  // entry of kp / ka
            v = -static_cast<float>((d.dyn_phase && q == 0) ? d.kp[g3] : d.ka[g3]);
        }
        A[static_cast<size_t>(r) * ld + c] = v;
        A[static_cast<size_t>(c) * ld + r] = v;
    }
}

// acc = L R for 64x64 blocks in shared memory (leading dimension kInvLd, 16-byte
// rows); each of the 256 threads owns rows 4*(tid/16) + u and columns
// 4*(tid%16) + v, the R operand read as one float4 per step.
constexpr int kInvLd = kGjBlock + 4;
__device__ __forceinline__ void block_gemm64(const float *L, const float *R, float (&acc)[4][4]) {
    const int r0 = 4 * (threadIdx.x >> 4), c0 = 4 * (threadIdx.x & 15);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = 0.0f;
#pragma unroll 8
    for (int k = 0; k < kGjBlock; ++k) {
        float l[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) l[u] = L[(r0 + u) * kInvLd + k];
        const float4 r4 = *reinterpret_cast<const float4 *>(&R[k * kInvLd + c0]);
        const float r[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(l[u], r[v], acc[u][v]);
    }
}

// Part (a) of a round: inverts pivot block K of patch p (rows and columns
// [64K, 64K + b)) into its dinv block, zero-padded to 64 x 64; called by all
// 256 threads of a block.  The 64x64 block D (padded with the identity beyond
// b) is inverted in place by block Gauss-Jordan elimination without pivoting,
// in registers: thread (ty, tx) holds rows 4ty .. + 3 and columns 4tx .. + 3.
// The pivots are taken in eight panels of eight: the panel's rows and columns
// are published, warp 0 inverts the panel's 8 x 8 block by shuffles (a chain of
// eight reciprocals), every row forms its eight coefficients (-a_r D^-1, or row
// r of D^-1 inside the panel), and the block takes the rank-8 update
//   x <- [x outside the panel's rows and columns] + coefficients panel.
// Forming the inverse explicitly loses accuracy when D is ill conditioned, so
// the result X is refined by one Newton step, X <- X + X (I - D X), which
// squares its residual.  A zero or non-finite pivot clears the patch's ok flag.
// The inverse is the critical path of the refresh (the next round waits for
// it): 26.6 -> 16.4 us alone (16 blocks, 1.965 GHz), of which the elimination
// 34 600 -> 15 900 cycles: sixteen columns of one row per thread read the panel
// with bank conflicts, four 128-bit loads per sixteen FMAs, where a 4 x 4 tile
// reads two without; and each warp eliminating its own panel moved sixteen
// values per pivot by shuffles.  The Newton products take 7 700.
// The reciprocals are the hardware's approximation: |D X - I| of random and of mobility blocks (condition 2 to 1e4) has
// the same mean over 148 blocks, 2.4e-8 to 1.2e-5, as with correctly rounded ones and as in the elimination before, within
// 1%; the inverses of whole patches likewise (80a apart, one step forth and back: 5.4e-5, 5.5e-5 and 5.2e-5 of 40 blocks of
// 62, 5.7, 5.5 and 5.7e-5 of 24 filaments in patches of 3), and so the solver's iterations on colliding cilia.
// A: the patch matrix (n x n), dv: its dinv block, ok: its flag, ws: shared
// memory of at least kInvWs floats.
constexpr int kInvWs = 2 * kGjBlock * kInvLd;
__device__ __noinline__ void pivot_invert(const float *A, int n, float *dv, int *ok, int K, float *ws) {
    static_assert(kGjBlock == 64, "sixteen 4 x 4 tiles a side");
    const int k0 = K * kGjBlock;
    const int b = min(kGjBlock, n - k0);
    float *X = ws, *W = ws + kGjBlock * kInvLd;  // X: the inverse; W: D, then I - D X
    constexpr int kCoefLd = kGjBlock + 4;  // the four coefficient pairs of a row land on different banks
    __shared__ __align__(16) float rows[2][8][kGjBlock];
    __shared__ __align__(16) float cols[2][kGjBlock][8];
    __shared__ __align__(16) float dinv[8][8];
    __shared__ __align__(16) float coef[8][kCoefLd];
    __shared__ int sbad;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, lane = threadIdx.x & 31;
    const size_t ld = patch_ld(n);
    float v[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = 4 * ty + u, c = 4 * tx;
        // rows start on 16 bytes and the padding columns are mapped, so whole chunks inside the row stride are read
        float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < b && k0 + c < static_cast<int>(ld)) q = *reinterpret_cast<const float4 *>(A + (k0 + r) * ld + k0 + c);
        const float e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int s = 0; s < 4; ++s) v[u][s] = (r < b && c + s < b) ? e[s] : (r == c + s ? 1.0f : 0.0f);
        *reinterpret_cast<float4 *>(W + r * kInvLd + c) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    }
    if (threadIdx.x == 0) sbad = 0;
#pragma unroll 1
    for (int m = 0; m < 8; ++m) {
        const int par = m & 1;
        const bool prow = (ty >> 1) == m, pcol = (tx >> 1) == m;
        if (prow)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                *reinterpret_cast<float4 *>(&rows[par][4 * (ty & 1) + u][4 * tx]) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
        if (pcol)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                *reinterpret_cast<float4 *>(&cols[par][4 * ty + u][4 * (tx & 1)]) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
        __syncthreads();
        if (threadIdx.x < 32) {  // warp 0: the panel's 8 x 8 block, lane (row lane / 4, columns 2 (lane % 4), + 1)
            float2 d = *reinterpret_cast<const float2 *>(&cols[par][8 * m + (lane >> 2)][2 * (lane & 3)]);
            bool bad = false;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float mine = (t & 1) ? d.y : d.x;
                const float piv = __shfl_sync(0xffffffffu, mine, 4 * t + (t >> 1));
                const float f = __shfl_sync(0xffffffffu, mine, (lane & ~3) | (t >> 1));
                const float px = __shfl_sync(0xffffffffu, d.x, 4 * t + (lane & 3)), py = __shfl_sync(0xffffffffu, d.y, 4 * t + (lane & 3));
                float ip;
                asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ip) : "f"(piv));
                bad |= !(fabsf(piv) > 0.0f) || !(fabsf(piv) < INFINITY);
                const bool own = (lane >> 2) == t, here = (lane & 3) == (t >> 1);
                const float a = own ? 0.0f : 1.0f, bq = own ? ip : -f * ip;
                const float nx = fmaf(bq, px, a * d.x), ny = fmaf(bq, py, a * d.y);
                d.x = (here && !(t & 1)) ? bq : nx;
                d.y = (here && (t & 1)) ? bq : ny;
            }
            *reinterpret_cast<float2 *>(&dinv[lane >> 2][2 * (lane & 3)]) = d;
            if (bad) sbad = 1;
        }
        __syncthreads();
        {  // two of the row's eight coefficients: -a_r D^-1 outside the panel, row r of D^-1 inside
            const int r = threadIdx.x >> 2, s = 2 * (threadIdx.x & 3);
            float cx = 0.0f, cy = 0.0f;
            if ((r >> 3) == m) {
                cx = dinv[r & 7][s];
                cy = dinv[r & 7][s + 1];
            } else {
                const float4 a0 = *reinterpret_cast<const float4 *>(&cols[par][r][0]), a1 = *reinterpret_cast<const float4 *>(&cols[par][r][4]);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const float2 e = *reinterpret_cast<const float2 *>(&dinv[t][s]);
                    cx = fmaf(-av[t], e.x, cx);
                    cy = fmaf(-av[t], e.y, cy);
                }
            }
            coef[s][r] = cx;
            coef[s + 1][r] = cy;
        }
        __syncthreads();
        if (prow)
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int s = 0; s < 4; ++s) v[u][s] = 0.0f;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const float4 p4 = *reinterpret_cast<const float4 *>(&rows[par][t][4 * tx]);
            const float4 c4 = *reinterpret_cast<const float4 *>(&coef[t][4 * ty]);
            const float p[4] = {p4.x, p4.y, p4.z, p4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int s = 0; s < 4; ++s) v[u][s] = fmaf(c[u], p[s], v[u][s]);
        }
        if (pcol)  // the panel's columns hold the coefficients themselves
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float4 c4 = *reinterpret_cast<const float4 *>(&coef[4 * (tx & 1) + s][4 * ty]);
                v[0][s] = c4.x;
                v[1][s] = c4.y;
                v[2][s] = c4.z;
                v[3][s] = c4.w;
            }
    }
    const int r0 = 4 * ty, c0 = 4 * tx;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        *reinterpret_cast<float4 *>(X + (r0 + u) * kInvLd + c0) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    __syncthreads();
    float acc[4][4];
    block_gemm64(W, X, acc);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) W[(r0 + u) * kInvLd + c0 + q] = (r0 + u == c0 + q ? 1.0f : 0.0f) - acc[u][q];
    __syncthreads();
    block_gemm64(X, W, acc);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int rr = r0 + u, c = c0 + q;
            dv[rr * kGjBlock + c] = (rr < b && c < b) ? v[u][q] + acc[u][q] : 0.0f;
        }
    if (threadIdx.x == 0) {
        if (sbad) *ok = 0;
        else if (K == 0) *ok = 1;
    }
}

__device__ __forceinline__ void pivot_invert_patch(const PatchDev &P, int p, int K, float *ws) {
    pivot_invert(P.A + P.moff[p], P.nf[p] * P.nbf, P.dinv + static_cast<size_t>(p) * kGjBlock * kGjBlock, P.ok + p, K,
                 ws);
}

// Round 0, part (a): the first pivot block of every patch (later pivot blocks
// are inverted by the previous round's update, see gj_update_kernel).
__global__ void __launch_bounds__(256) gj_pivot_kernel(PatchDev P, int K) {
    __shared__ __align__(16) float ws[kInvWs];
    const int p = blockIdx.x;
    const int n = P.nf[p] * P.nbf;
    if (K * kGjBlock >= n) return;
    pivot_invert_patch(P, p, K, ws);
}

// Round K, part (b), one 64-column tile [j0, j0 + 64) of a patch per block.
// The matrix is kept symmetric and only its upper block triangle is
// maintained, so the pivot rows' entries are
//   U[s][j] = A[k0 + s][j] for j >= k0,   A[j][k0 + s] for j < k0  (by symmetry);
// both are read as 64 contiguous floats per row of A and staged in shared
// memory as U[s][c].  The pass writes, for the tile's columns c (j = j0 + c),
//   rsplit: (D^-1 U)[s][c] outside the pivot columns, -D^-1[s][c] inside,
//   csplit: U[s][c]         outside the pivot columns (zero inside),
// each split into its TF32 high part and FP32 remainder in the canonical layout of
// the tensor-core operands (element (c, s) at tc::canon(c, s)), the form in which
// the update pass multiplies them.  Tiles and pivot blocks are both 64 wide, so a tile is either the pivot
// block's or disjoint from it.  Each thread owns 4 rows x 4 columns of
// D^-1 U (rows 4ty + u, columns 4tx + v); the loads and stores of the
// product's operands and results move 16 bytes each.  grid = (tiles, patches).
__global__ void __launch_bounds__(256) gj_prep_kernel(PatchDev P, int K) {
    static_assert(kGjTile == kGjBlock, "column tiles are pivot-block wide");
    constexpr int LD = kGjTile + 4;  // 16-byte rows
    __shared__ __align__(16) float DvT[kGjBlock][LD];  // DvT[s][r] = D^-1[r][s]
    __shared__ __align__(16) float Us[kGjBlock][LD];
    chain_wait();
    const int p = blockIdx.y;
    const int n = P.nf[p] * P.nbf;
    const int k0 = K * kGjBlock;
    const int j0 = blockIdx.x * kGjTile;
    if (k0 >= n || j0 >= n) return;
    const int b = min(kGjBlock, n - k0);
    const int w = min(kGjTile, n - j0);  // columns in this tile
    const size_t ld = patch_ld(n);
    const float *A = P.A + P.moff[p];
    float *rs = P.rsplit + (static_cast<size_t>(p) * P.T + blockIdx.x) * 2 * tc::kOperandFloats;
    float *cs = P.csplit + (static_cast<size_t>(p) * P.T + blockIdx.x) * 2 * tc::kOperandFloats;
    const float *dv = P.dinv + static_cast<size_t>(p) * kGjBlock * kGjBlock;
    if (j0 == k0) {  // the pivot columns: -D^-1, and no pivot-row copies
        for (int e = threadIdx.x; e < kGjBlock * kGjTile; e += blockDim.x) {
            const int r = e / kGjTile, c = e - r * kGjTile;
            float h, l;
            tc::split_tf32(c < w ? -dv[r * kGjBlock + c] : 0.0f, h, l);  // zero-padded rows
            rs[tc::canon(c, r)] = h;
            rs[tc::kOperandFloats + tc::canon(c, r)] = l;
            cs[tc::canon(c, r)] = 0.0f;
            cs[tc::kOperandFloats + tc::canon(c, r)] = 0.0f;
        }
        return;
    }
    // D^-1, 16-byte loads, stored transposed: a warp takes 32 rows, so that its stores do not share banks (with the
    // lanes along the rows eight of them did: 14.2 us a round, 12.9 so)
    for (int e4 = threadIdx.x; e4 < kGjBlock * kGjBlock / 4; e4 += blockDim.x) {
        const int r = e4 & 63, c4 = 4 * (e4 >> 6);
        const float4 v = *reinterpret_cast<const float4 *>(dv + r * kGjBlock + c4);
        DvT[c4][r] = v.x;
        DvT[c4 + 1][r] = v.y;
        DvT[c4 + 2][r] = v.z;
        DvT[c4 + 3][r] = v.w;
    }
    // U, 16-byte chunks of rows of A; chunks at or beyond the row stride are zeros, and so are the padding
    // columns [n, ld) inside it, so U[s][c] is zero for s >= b or c >= w as the product needs
    if (j0 > k0) {  // U[s][c] = A[k0 + s][j0 + c]
        for (int e4 = threadIdx.x; e4 < kGjBlock * kGjTile / 4; e4 += blockDim.x) {
            const int s_ = e4 >> 4, c4 = 4 * (e4 & 15);
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (s_ < b && j0 + c4 < static_cast<int>(ld)) v = *reinterpret_cast<const float4 *>(A + (k0 + s_) * ld + j0 + c4);
            *reinterpret_cast<float4 *>(&Us[s_][c4]) = v;
        }
    } else {  // j0 + 64 <= k0: U[s][c] = A[j0 + c][k0 + s], rows of A stored transposed
        for (int e4 = threadIdx.x; e4 < kGjTile * kGjBlock / 4; e4 += blockDim.x) {
            const int c = e4 & 63, s4 = 4 * (e4 >> 6);
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (k0 + s4 < static_cast<int>(ld)) v = *reinterpret_cast<const float4 *>(A + (j0 + c) * ld + k0 + s4);
            Us[s4][c] = v.x;
            Us[s4 + 1][c] = v.y;
            Us[s4 + 2][c] = v.z;
            Us[s4 + 3][c] = v.w;
        }
    }
    __syncthreads();
    // rows 4ty + u, columns 4tx + v of D^-1 U: one float4 of each operand per step
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4] = {};
#pragma unroll 8
    for (int s_ = 0; s_ < kGjBlock; ++s_) {
        const float4 d4 = *reinterpret_cast<const float4 *>(&DvT[s_][4 * ty]);
        const float4 u4 = *reinterpret_cast<const float4 *>(&Us[s_][4 * tx]);
        const float dr[4] = {d4.x, d4.y, d4.z, d4.w}, uc[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(dr[u], uc[v], acc[u][v]);
    }
    const int c0 = 4 * tx;
    __syncthreads();  // DvT is free: it holds the product tile while it is written out
    float(*Pt)[LD] = DvT;
#pragma unroll
    for (int u = 0; u < 4; ++u)  // rows >= b: zeros (D^-1 is zero-padded); columns >= w: zeros
        *reinterpret_cast<float4 *>(&Pt[4 * ty + u][c0]) =
            make_float4(c0 < w ? acc[u][0] : 0.0f, c0 + 1 < w ? acc[u][1] : 0.0f, c0 + 2 < w ? acc[u][2] : 0.0f,
                        c0 + 3 < w ? acc[u][3] : 0.0f);
    __syncthreads();
    // both operands written in the canonical order (consecutive threads, consecutive addresses): element q of
    // the layout is (c, s) = tc::canon_inverse(q); the pivot-row entries are U itself (zero beyond w, as U is)
    for (int q = threadIdx.x; q < tc::kOperandFloats; q += blockDim.x) {
        const int c = tc::canon_mn(q), s_ = tc::canon_k(q);
        float h, l;
        tc::split_tf32(Pt[s_][c], h, l);
        rs[q] = h;
        rs[tc::kOperandFloats + q] = l;
        tc::split_tf32(Us[s_][c], h, l);
        cs[q] = h;
        cs[tc::kOperandFloats + q] = l;
    }
}

// One tile of round K's update: which tile of which patch, and its kind.
struct GjTile {
    int p, n, row0, col0;
    bool valid, prow, pcol, diag;
};

// Work item -> tile.  Items run patch-fastest over a triangle enumeration of
// the upper block triangle (T = the largest patch's tiles per side) in which
// index 0 is the next round's diagonal tile (K + 1, K + 1), so the first np
// items are the patches' diagonal tiles and are taken first.
__device__ __forceinline__ GjTile gj_tile(const PatchDev &P, int K, int T, int item) {
    GjTile t{};
    t.p = item % P.np;
    int q = item / P.np;
    t.n = P.nf[t.p] * P.nbf;
    const int Tp = (t.n + kGjTile - 1) / kGjTile;
    const int d = K + 1;
    if (d < T) {
        const int qd = d * T - d * (d - 1) / 2;  // triangle index of (d, d)
        q = (q == 0) ? qd : (q <= qd ? q - 1 : q);
    }
    int ti = 0;
    while (ti < T && q >= T - ti) {
        q -= T - ti;
        ++ti;
    }
    const int tj = ti + q;
    t.valid = K * kGjBlock < t.n && ti < Tp && tj < Tp;
    t.row0 = ti * kGjTile;
    t.col0 = tj * kGjTile;
    t.prow = ti == K;
    t.pcol = tj == K;
    t.diag = ti == d && tj == d;
    return t;
}

// Stage of the update: the tile's split operands as the prep pass left them
// (A = the pivot-row copies of its row tile, B = the scaled pivot rows of its
// column tile, each a TF32 high part and an FP32 remainder in the canonical
// layout, 4 x 16 KB), and behind it the product tile on its way from tensor
// memory to the rows of A.  Two blocks per SM.
constexpr int kUpStage = 4 * tc::kOperandFloats;
constexpr int kUpLd = kGjTile + 4;  // 16-byte rows
constexpr size_t kUpdateSmem = (kUpStage + kGjTile * kUpLd) * sizeof(float);

// Starts the copies of a tile's operands into `stage` (one thread): each is one contiguous 32 KB block.  The pivot rows
// need B only.
__device__ __forceinline__ void gj_issue_tile(const PatchDev &P, const GjTile &t, float *stage, uint64_t *full) {
    constexpr uint32_t kBytes = 2 * tc::kOperandFloats * sizeof(float);
    const float *csrc = P.csplit + (static_cast<size_t>(t.p) * P.T + t.row0 / kGjTile) * 2 * tc::kOperandFloats;
    const float *rsrc = P.rsplit + (static_cast<size_t>(t.p) * P.T + t.col0 / kGjTile) * 2 * tc::kOperandFloats;
    mbar_arrive_expect_tx(full, t.prow ? kBytes : 2 * kBytes);
    bulk_g2s(stage + 2 * tc::kOperandFloats, rsrc, kBytes, full);
    if (!t.prow) bulk_g2s(stage, csrc, kBytes, full);
}

// Round K, part (c), the 64x64 tiles of the upper block triangle:
//   pivot rows       A[i, j] = rbuf[i - k0][j]      (-D^-1 in the pivot block)
//   other rows       A[i, j] -= C_i . rbuf[:, j]   (j outside the pivot columns)
//                    A[i, j]  = -C_i . rbuf[:, j]  (pivot columns: C_i D^-1)
// with C_i = cbuf[:][i] (the pivot-row copies) and rbuf the scaled pivot rows
// -- the symmetric sweep, which leaves -A^-1 after the last round.  Tiles and
// pivot blocks are both 64 wide, so a tile lies in the pivot rows (ti == K, a
// copy), in the pivot columns (tj == K) or in neither.  Persistent blocks (two
// per SM) take tiles from a per-round counter.  The tile product C^T rbuf runs
// on the tensor cores (tc_tf32.cuh: the operands as the prep pass split them,
// three TF32 products accumulated in FP32 in tensor memory, issued by one
// thread and committed to an mbarrier).  A tile is a chain of waits (operands,
// products, read-back), so the chain is overlapped: the next tile is drawn
// while the operands land and its copies start as soon as the products have
// read theirs, and the products go through shared memory so that the rows of A
// are read and written 256 contiguous bytes at a time: a round of 16 patches of
// 992 unknowns takes 31.6 us, 41 without (33.0 with 16-byte copies by every
// thread instead of two bulk copies a tile), of which the chain diagonal tile ->
// inversion is about 22 when it has its SM alone.
// The block that takes a patch's diagonal tile (K + 1, K + 1) inverts it for
// the next round right after its update, while the other blocks go on with the
// rest.  A wait for copies or products that gives up (bounded) marks the tile's patch
// unusable -- it falls back to the block-diagonal preconditioner -- and the
// block computes no further products.  Dynamic shared memory: kUpdateSmem.
__global__ void __launch_bounds__(256, 2) gj_update_kernel(PatchDev P, int K, int T, int *counter) {
    static_assert(kGjTile == 64 && kGjBlock == 64 && tc::kTileMN == 64 && tc::kTileK == 64, "64-wide tiles");
    static_assert(kUpStage >= kInvWs, "the inversion reuses the stage");
    extern __shared__ __align__(128) float usm[];
    __shared__ int next_item[2];  // drawn ahead; drawn after an inversion
    __shared__ __align__(8) uint64_t bar, full;
    __shared__ uint32_t tbase;
    __shared__ int tc_ok, dead;
    chain_wait();
    const int total = P.np * (T * (T + 1) / 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) next_item[0] = atomicAdd(counter, 1);
    __syncthreads();
    const int item = next_item[0];
    if (item >= total) return;
    if (warp == 0) tc::tmem_alloc(&tbase, tc::kTmemCols);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_init(&full, 1);
        fence_barrier_init();
        dead = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tbase;
    uint32_t products = 0;  // completed phases of `bar`
    const float *Ab = usm, *Bb = usm + 2 * tc::kOperandFloats;
    float *Ct = usm + kUpStage;
    // this thread's output: rows tr + 16 k, columns tc4 .. + 3
    const int tr = threadIdx.x >> 4, tc4 = 4 * (threadIdx.x & 15);
    GjTile cur = gj_tile(P, K, T, item);
    uint32_t copies = 0;  // tiles whose operands were waited for
    bool broken = false;  // such a wait gave up: nothing more is copied or multiplied
    if (cur.valid && threadIdx.x == 0) gj_issue_tile(P, cur, usm, &full);
    for (;;) {
        int drawn = 0;
        if (threadIdx.x == 0 && !cur.diag) drawn = atomicAdd(counter, 1);
        const int n = cur.n, ld = patch_ld(n);
        const int i0 = cur.row0 + tr, j = cur.col0 + tc4;
        float *Arow = P.A + P.moff[cur.p] + static_cast<size_t>(i0) * ld + j;
        float res[4][4] = {};
        // the old values, while the operands land (the pivot columns and rows are overwritten)
        if (cur.valid && !cur.prow && !cur.pcol && j < ld) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + 16 * k < n) {
                    const float4 o4 = *reinterpret_cast<const float4 *>(Arow + static_cast<size_t>(16 * k) * ld);
                    res[k][0] = o4.x;
                    res[k][1] = o4.y;
                    res[k][2] = o4.z;
                    res[k][3] = o4.w;
                }
        }
        if (threadIdx.x == 0) next_item[0] = drawn;
        bool landed = true;
        if (cur.valid && !broken) landed = mbar_wait_bounded(&full, copies++ & 1u);
        tc::fence_before_sync();
        if (!__syncthreads_and(landed)) broken = true;
        tc::fence_after_sync();
        int next = next_item[0];
        const bool stopped = dead != 0 || broken;
        if (cur.valid && !cur.prow && !stopped && threadIdx.x == 0) {
            tc::issue_tile_products(tmem, Ab, Ab + tc::kOperandFloats, Bb, Bb + tc::kOperandFloats);
            tc::commit(&bar);
        }
        GjTile nxt{};
        if (next < total && !cur.diag) nxt = gj_tile(P, K, T, next);
        if (cur.valid) {
            if (cur.prow) {  // the pivot rows: the scaled pivot rows themselves (row0 == k0), high + low parts
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int e = tc::canon(tc4 + q, tr + 16 * k);
                        res[k][q] = Bb[e] + Bb[tc::kOperandFloats + e];
                    }
            } else if (!stopped) {
                if (threadIdx.x == 0) {
                    bool ok = mbar_wait_bounded(&bar, products & 1u);
                    if (!ok) ok = mbar_wait_bounded(&bar, products & 1u);  // drain before going on
                    tc_ok = ok ? 1 : 0;
                }
                ++products;
            }
        }
        tc::fence_proxy_async();
        __syncthreads();  // the stage has been read
        tc::fence_after_sync();
        const bool product = cur.valid && !cur.prow, have = product ? !stopped && tc_ok != 0 : !broken;
        if (nxt.valid && !broken && threadIdx.x == 0) gj_issue_tile(P, nxt, usm, &full);
        if (product && have) {
            // row m of the product lies in lane m % 16 of warps m / 16 and m / 16 + 4 (32 columns each)
            float v[32];
            tc::tmem_ld32(tc::tmem_addr(tmem, warp, 32 * (warp >> 2)), v);
            if (lane < 16) {
                float4 *o = reinterpret_cast<float4 *>(Ct + (16 * (warp & 3) + lane) * kUpLd + 32 * (warp >> 2));
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
            tc::fence_before_sync();
        }
        __syncthreads();
        if (cur.valid && !have && threadIdx.x == 0) {
            P.ok[cur.p] = 0;
            dead = 1;
        }
        if (cur.valid && have) {
            if (product)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 v4 = *reinterpret_cast<const float4 *>(Ct + (tr + 16 * k) * kUpLd + tc4);
                    res[k][0] -= v4.x;
                    res[k][1] -= v4.y;
                    res[k][2] -= v4.z;
                    res[k][3] -= v4.w;
                }
            // the patch's last round writes its final values: a non-finite one marks the inverse unusable
            const bool last = (K + 1) * kGjBlock >= n, mirror = last && cur.row0 < cur.col0;
            bool bad = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (i0 + 16 * k >= n) continue;
                float *o = Arow + static_cast<size_t>(16 * k) * ld;
                if (j + 3 < n) {
                    *reinterpret_cast<float4 *>(o) = make_float4(res[k][0], res[k][1], res[k][2], res[k][3]);
                } else {  // the row's last, partial chunk: nothing beyond column n - 1
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (j + q < n) o[q] = res[k][q];
                }
                if (last)
#pragma unroll
                    for (int q = 0; q < 4; ++q) bad |= (j + q < n) && !isfinite(res[k][q]);
            }
            if (bad) P.ok[cur.p] = 0;
            if (mirror) {  // final values: also the transposed tile of the lower block triangle (A^-1 is symmetric)
                __syncthreads();
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    *reinterpret_cast<float4 *>(Ct + (tr + 16 * k) * kUpLd + tc4) =
                        make_float4(res[k][0], res[k][1], res[k][2], res[k][3]);
                __syncthreads();
                for (int e = threadIdx.x; e < kGjTile * kGjTile; e += blockDim.x) {
                    const int c = e >> 6, r = e & 63;
                    if (cur.row0 + r < n && cur.col0 + c < n)
                        P.A[P.moff[cur.p] + static_cast<size_t>(cur.col0 + c) * ld + cur.row0 + r] = Ct[r * kUpLd + c];
                }
            }
        }
        if (cur.diag) {  // the tile is final for round K + 1: invert it now (its writes are the block's own).  The
            __syncthreads();  // inversion works in the stage, so the next tile is drawn and copied after it
            if (cur.valid) pivot_invert_patch(P, cur.p, K + 1, usm);
            if (threadIdx.x == 0) next_item[1] = atomicAdd(counter, 1);
            tc::fence_proxy_async();
            __syncthreads();
            next = next_item[1];
            if (next < total) nxt = gj_tile(P, K, T, next);
            if (nxt.valid && !broken && threadIdx.x == 0) gj_issue_tile(P, nxt, usm, &full);
        }
        if (next >= total) break;
        cur = nxt;
    }
    if (broken && threadIdx.x == 0) mbar_wait_bounded(&full, (copies - 1) & 1u);  // copies still in flight land first
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, tc::kTmemCols);
}

// out = blockdiag(A_pp^-1) in over the patches (in and out must differ).
// grid = (row chunks of kApplyRows, patches), kApplyThreads threads; the block
// gathers the patch's rows of `in` into shared memory, each warp forms two
// output rows with the lanes striding the (coalesced, 16-byte) matrix rows,
// four loads per row in flight.  A patch without a finite inverse uses the
// block-diagonal preconditioner instead (first row chunk only).
// Dynamic shared memory: max(patch_ld(max_n), 3*nseg) doubles.
// With `masked`, patches of arrays whose GMRES stopped are skipped.
constexpr int kApplyRows = 32, kApplyThreads = 16 * 32;  // two rows per warp
__global__ void __launch_bounds__(kApplyThreads) patch_apply_kernel(SimDev d, PatchDev P, const double *in,
                                                                   double *out, int masked) {
    extern __shared__ __align__(16) double xs[];
    __shared__ double sm32[32];
    const int p = blockIdx.y;
    const int n = P.nf[p] * P.nbf;
    const int r0 = blockIdx.x * kApplyRows;
    if (r0 >= n) return;
    if (masked && !d.active[d.fil_arr[P.fils[P.fil0[p]]]]) return;
    if (!P.ok[p]) {
        if (blockIdx.x != 0) return;
        for (int a = 0; a < P.nf[p]; ++a) {
            const int m = P.fils[P.fil0[p] + a];
            precond_block(d, m, fil_rows(d, m), in, out, xs, sm32);
            __syncthreads();
        }
        return;
    }
    const long long *rows = P.rows + P.roff[p];
    const int ld = patch_ld(n), n4 = ld >> 2;
    for (int c = threadIdx.x; c < ld; c += blockDim.x) xs[c] = c < n ? in[rows[c]] : 0.0;  // padding: zeros
    __syncthreads();
    const float *A = P.A + P.moff[p];
    const double2 *x2 = reinterpret_cast<const double2 *>(xs);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const int r = r0 + 2 * warp;  // this warp's two rows
        if (r >= n) return;
        const bool two = r + 1 < n;
        const float4 *a0 = reinterpret_cast<const float4 *>(A + static_cast<size_t>(r) * ld);
        const float4 *a1 = a0 + n4;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
        for (int c4 = lane; c4 < n4; c4 += 32) {
            const float4 v0 = __ldg(a0 + c4);
            const float4 v1 = two ? __ldg(a1 + c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const double2 xa = x2[2 * c4], xb = x2[2 * c4 + 1];
            s0 = fma(static_cast<double>(v0.x), xa.x, s0);
            s0 = fma(static_cast<double>(v0.y), xa.y, s0);
            s0 = fma(static_cast<double>(v0.z), xb.x, s0);
            s0 = fma(static_cast<double>(v0.w), xb.y, s0);
            s1 = fma(static_cast<double>(v1.x), xa.x, s1);
            s1 = fma(static_cast<double>(v1.y), xa.y, s1);
            s1 = fma(static_cast<double>(v1.z), xb.x, s1);
            s1 = fma(static_cast<double>(v1.w), xb.y, s1);
        }
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
        if (lane == 0) {  // the refresh leaves -A_pp^-1
            out[rows[r]] = -s0;
            if (two) out[rows[r + 1]] = -s1;
        }
    }
}

// The preconditioning step of one GMRES iteration with the line patches in a
// single launch (in place of arnoldi_precond_kernel + patch_apply_kernel +
// pack_rows_kernel).  Block (a, p) serves filament a of patch p: it clears the
// loop condition (block (0, 0)), gathers the patch's rows of the new basis
// vector Q_k = src * inv_scale (src = r0 or A z in w, or rhs after a discarded
// guess), stores its own filament's rows of Q_k (and of the copy t that the
// network's features read), forms its filament's rows of z = P^-1 Q_k (the
// refresh leaves -A_pp^-1: each warp two rows, lanes striding the 16-byte
// matrix rows) and packs their forces for the pair kernel.  The filament rows
// of A z are written by the saddle epilogue (epi_fil_rows): other blocks of
// the patch still read w here.  A patch without a finite inverse falls back to
// the block-diagonal preconditioner for the filament.
// Dynamic shared memory: patch_ld(max_n) + max(nbf, 3*nseg) doubles.
constexpr int kArnThreads = 256;
constexpr int kArnParts = 2;  // blocks per filament: the rows of segments [0, ceil(nseg/2)) and the rest
__global__ void __launch_bounds__(kArnThreads, 4) patch_arnoldi_kernel(SimDev d, PatchDev P,
                                                                       cudaGraphConditionalHandle h) {
    extern __shared__ __align__(16) double xs[];
    __shared__ double sm32[32];
    chain_wait();
    const int p = blockIdx.y, a = blockIdx.x / kArnParts, part = blockIdx.x % kArnParts;
    if (p == 0 && blockIdx.x == 0 && threadIdx.x == 0) set_loop(h, d.lc, 0);
    if (a >= P.nf[p]) return;
    const int m = P.fils[P.fil0[p] + a];
    const FilRows fr = fil_rows(d, m);
    if (!d.active[fr.b]) return;  // uniform over the block
    const int k = d.lc->k;
    if (k >= d.arr[fr.b].max_iter) return;  // defensive: the cap was reached
    const GmresCtl &c = d.ctl[fr.b];
    const double sc = c.inv_scale;
    const double *src = (k == 0 && c.zero_guess) ? d.rhs : d.w;
    double *q = d.Q + static_cast<size_t>(k) * d.ldq;
    const int n = P.nf[p] * P.nbf, nbf = P.nbf, r_lo = a * nbf;
    // this block's rows of the filament: whole segments (3 rows each), the rate rows with the second part
    const int split = 3 * ((d.nseg + 1) / 2);
    const int r_beg = part == 0 ? 0 : split, r_end = part == 0 ? split : nbf;
    const long long *rows = P.rows + P.roff[p];
    const int ld = patch_ld(n), n4 = ld >> 2;
    double *zs = xs + ld;
    for (int cc = threadIdx.x; cc < ld; cc += blockDim.x) xs[cc] = cc < n ? src[rows[cc]] * sc : 0.0;
    __syncthreads();
    if (!P.ok[p]) {  // the first part alone: the whole filament through the block-diagonal preconditioner
        if (part != 0) return;
        for (int r = threadIdx.x; r < nbf; r += blockDim.x) q[rows[r_lo + r]] = xs[r_lo + r];
        if (d.learned)
            for (int r = threadIdx.x; r < nbf; r += blockDim.x) d.t[rows[r_lo + r]] = xs[r_lo + r];
        __syncthreads();  // this block's rows of Q_k are in global memory
        precond_block(d, m, fr, q, d.z, zs, sm32);
        __syncthreads();
        for (int kk = threadIdx.x; kk < d.nseg; kk += blockDim.x) {
            const long long r = fr.lam + 3 * kk;
            d.f4[m * d.nseg + kk] = make_float4(static_cast<float>(d.z[r]), static_cast<float>(d.z[r + 1]),
                                                static_cast<float>(d.z[r + 2]), 0.0f);
        }
        return;
    }
    for (int r = r_beg + threadIdx.x; r < r_end; r += blockDim.x) q[rows[r_lo + r]] = xs[r_lo + r];
    if (d.learned)
        for (int r = r_beg + threadIdx.x; r < r_end; r += blockDim.x) d.t[rows[r_lo + r]] = xs[r_lo + r];
    const float *A = P.A + P.moff[p];
    const double2 *x2 = reinterpret_cast<const double2 *>(xs);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = r_beg + 2 * warp; r < r_end; r += 2 * (kArnThreads / 32)) {
        const bool two = r + 1 < r_end;
        const float4 *a0 = reinterpret_cast<const float4 *>(A + static_cast<size_t>(r_lo + r) * ld);
        const float4 *a1 = a0 + n4;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
        for (int c4 = lane; c4 < n4; c4 += 32) {
            const float4 v0 = __ldg(a0 + c4);
            const float4 v1 = two ? __ldg(a1 + c4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const double2 xa = x2[2 * c4], xb = x2[2 * c4 + 1];
            s0 = fma(static_cast<double>(v0.x), xa.x, s0);
            s0 = fma(static_cast<double>(v0.y), xa.y, s0);
            s0 = fma(static_cast<double>(v0.z), xb.x, s0);
            s0 = fma(static_cast<double>(v0.w), xb.y, s0);
            s1 = fma(static_cast<double>(v1.x), xa.x, s1);
            s1 = fma(static_cast<double>(v1.y), xa.y, s1);
            s1 = fma(static_cast<double>(v1.z), xb.x, s1);
            s1 = fma(static_cast<double>(v1.w), xb.y, s1);
        }
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
        if (lane == 0) {
            d.z[rows[r_lo + r]] = -s0;
            zs[r] = -s0;
            if (two) {
                d.z[rows[r_lo + r + 1]] = -s1;
                zs[r + 1] = -s1;
            }
        }
    }
    __syncthreads();
    const int kk_end = min(d.nseg, r_end / 3);
    for (int kk = r_beg / 3 + threadIdx.x; kk < kk_end; kk += blockDim.x)
        d.f4[m * d.nseg + kk] = make_float4(static_cast<float>(zs[3 * kk]), static_cast<float>(zs[3 * kk + 1]),
                                            static_cast<float>(zs[3 * kk + 2]), 0.0f);
}

// After a patch application: packs the force rows of z for the pair kernel
// and writes the filament rows of A z (one block per filament), the work that
// arnoldi_precond_kernel does itself with the block-diagonal preconditioner.
__global__ void pack_rows_kernel(SimDev d, const double *z, double *w) {
    __shared__ double sm32[32];
    const int m = blockIdx.x;
    const FilRows fr = fil_rows(d, m);
    if (!d.active[fr.b]) return;
    for (int kk = threadIdx.x; kk < d.nseg; kk += blockDim.x) {
        const long long r = fr.lam + 3 * kk;
        d.f4[m * d.nseg + kk] = make_float4(static_cast<float>(z[r]), static_cast<float>(z[r + 1]),
                                            static_cast<float>(z[r + 2]), 0.0f);
    }
    filament_rows(d, fr, z, w, sm32);
}

}  // namespace cufil
