// mlp_fused.cuh -- the network of the learned preconditioner in three kernels:
//   mlp_rows_kernel   a block takes 128 rows through all three layers (and, in
//                     training, back through them): activations never leave the
//                     chip except as the operands of the weight gradients
//   mlp_wgrad_kernel  the weight gradients, operand^T x operand over the rows,
//                     split over row ranges into partial sums
//   mlp_finish_kernel partial sums -> gradients, in a fixed order, and the Adam
//                     step with the new operand images of the weights
// for widths in, hidden <= 256 and out <= 128 (mlp.cu has the general GEMM for
// the others).  All products are BF16 x BF16 with FP32 accumulation on the
// 5th-generation tensor cores, 128 rows per tcgen05.mma.
//
// Operand images.  Every operand lies in memory as the tensor core reads it:
// BF16, K-major without swizzling, 8 rows x 16 bytes per core matrix, the core
// matrices of one group of 8 rows next to each other along K, so element
// (row, k) of an image with K padded to KP is at img(row, k, KP) and any run of
// whole 8-row groups is one contiguous block: one cp.async.bulk fetches 128
// rows of a weight image.  The weights' images are made when the weights are
// set and by the Adam step; the FP32 weights stay the master copy.
//
// What bounds it.  A pass over 1024 rows is 0.27 GFLOP and 0.9 MB: the time is
// the chain of dependent steps (stage, multiply, read back, three times), so
// each step moves its data once, 16 bytes at a time, and the next weights
// arrive while the current product runs.  With 182 x 256 x 256 x 62: forward of 1024 rows 7.9 us a call (37 with three
// GEMM launches and their activations in memory); loss and gradients of 2048 rows 115 us a call (947 with six GEMMs,
// those over K = 2048 rows unsplit, and serial column sums), of which the transfer of the gradients to the host is about
// half.  Sixteen warps for the epilogues: eight took 8.2 and 119 us.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "tc_tf32.cuh"

namespace cufil {
namespace mlpk {

constexpr int kRows = 128;      // rows of a block: the M of one tcgen05.mma
constexpr int kMaxW = 256;      // widest input and hidden layer
constexpr int kMaxOut = 128;    // widest output layer
constexpr int kChunk = 128;     // image rows (output columns) of one weight chunk
constexpr int kThreads = 256;
constexpr int kRowThreads = 512, kGroups = kRowThreads / 128;  // groups of four warps: each every kGroups-th 32 columns
constexpr uint32_t kCols = 256; // accumulator columns
constexpr size_t kABytes = static_cast<size_t>(kRows) * kMaxW * 2;
constexpr size_t kWBytes = static_cast<size_t>(kChunk) * kMaxW * 2;
constexpr size_t kRowsSmem = kABytes + 2 * kWBytes;
constexpr size_t kGradSmem = 4 * static_cast<size_t>(kChunk) * kRows * 2;

__host__ __device__ constexpr int pad32(int x) { return (x + 31) & ~31; }
__host__ __device__ constexpr int pad128(int x) { return (x + 127) & ~127; }
// Element (row, k) of an operand image whose K is padded to kp (a multiple of 16).
__host__ __device__ constexpr int img(int row, int k, int kp) {
    return (row >> 3) * (kp * 8) + (k >> 3) * 64 + (row & 7) * 8 + (k & 7);
}

struct RowArgs {
    const float *x, *t;   // [n][in], targets [n][out] (training)
    float *y;             // [n][out] (forward)
    int n, in, hid, out;
    const __nv_bfloat16 *f1, *f2, *f3;  // images of W1^T [hid x in], W2^T [hid x hid], W3^T [out x hid]
    const __nv_bfloat16 *g3, *g2;       // images of W3 [hid x out], W2 [hid x hid] (backward)
    const float *b1, *b2, *b3;
    // training: transposed operands [tile][features][128 rows], column sums and loss of each tile
    __nv_bfloat16 *xt, *a1t, *a2t, *dyt, *dz2t, *dz1t;
    float *db;            // [tile][2 pad32(hid) + pad32(out)]: db1, db2, db3
    double *loss;         // [tile]
    float scale;          // 1 / (n out)
};

__device__ __forceinline__ uint64_t image_desc(const void *p, int kp) {
    const uint64_t addr = (static_cast<uint64_t>(smem_u32(p)) >> 4) & 0x3FFFull;
    return addr | (static_cast<uint64_t>(128 >> 4) << 16) | (static_cast<uint64_t>(kp) << 32) | (1ull << 46);
}

// D[128 x cols] (+)= A B^T over K = kp (a multiple of 16): kp / 16 instructions, issued by one thread.
__device__ __forceinline__ void issue_product(uint32_t tmem_d, const void *a, const void *b, int kp, int cols,
                                              bool accumulate) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(cols >> 3) << 17) |
                           (static_cast<uint32_t>(kRows >> 4) << 24);
    const uint64_t da = image_desc(a, kp), db = image_desc(b, kp);
    for (int s = 0; s < kp / 16; ++s)
        tc::mma_bf16_idesc(tmem_d, da + s * (256 >> 4), db + s * (256 >> 4), idesc, (accumulate || s > 0) ? 1u : 0u);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// 32 consecutive values of one row into an image, 16 bytes per 8 columns.
__device__ __forceinline__ void store_image(__nv_bfloat16 *im, int row, int col0, int kp, const float *v) {
#pragma unroll
    for (int q = 0; q < 32; q += 8) {
        const uint4 w = make_uint4(pack_bf16(v[q], v[q + 1]), pack_bf16(v[q + 2], v[q + 3]),
                                   pack_bf16(v[q + 4], v[q + 5]), pack_bf16(v[q + 6], v[q + 7]));
        *reinterpret_cast<uint4 *>(im + img(row, col0 + q, kp)) = w;
    }
}

// The transpose of the image [128 rows x kp] in shared memory into global memory, [features][128 rows]: each
// 8 x 8 core matrix is transposed by ldmatrix and written as one 128-byte run.
__device__ __forceinline__ void write_transposed(const __nv_bfloat16 *im, int kp, __nv_bfloat16 *out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nk = kp >> 3, total = (kRows / 8) * nk;  // core matrices, four at a time
    for (int c0 = 4 * warp; c0 < total; c0 += 4 * (kRowThreads / 32)) {
        // core matrix c: feature group c / 16, row group c % 16, so four consecutive ones are 512 contiguous bytes
        const int c = c0 + (lane >> 3);
        const int fg = c >> 4, rg = c & 15;
        const uint32_t addr = smem_u32(im + (rg * nk + fg) * 64 + (lane & 7) * 8);
        uint32_t r[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr)
                     : "memory");
        uint32_t *o = reinterpret_cast<uint32_t *>(out) + c0 * 32 + lane;
#pragma unroll
        for (int q = 0; q < 4; ++q) o[32 * q] = r[q];
    }
}

// Column sums over the 32 rows of a warp: lane c returns the sum of column c (v is overwritten).
__device__ __forceinline__ float column_sums(float *v, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool up = (lane & o) != 0;
            const float keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    return v[0];
}

// One block per 128 rows.  Thread 0 fetches the weight chunks (two buffers, the next chunk's copy issued as soon
// as the product that read its buffer is done) and issues the products; all threads stage the input and run the
// epilogues: warp w reads the accumulator rows 32 (w % 4) .. + 31, its group w / 4 every kGroups-th block of 32 columns,
// the same assignment in every layer, so the ReLU masks of the backward pass stay in registers.  A bounded wait
// that gives up ends the products: the outputs (or the gradients) are NaN then.
template <bool TRAIN>
__global__ void __launch_bounds__(kRowThreads, 1) mlp_rows_kernel(RowArgs g) {
    extern __shared__ __align__(128) unsigned char dyn[];
    __nv_bfloat16 *As = reinterpret_cast<__nv_bfloat16 *>(dyn);
    __nv_bfloat16 *Ws[2] = {reinterpret_cast<__nv_bfloat16 *>(dyn + kABytes),
                            reinterpret_cast<__nv_bfloat16 *>(dyn + kABytes + kWBytes)};
    __shared__ __align__(8) uint64_t full[2], done[2];
    __shared__ uint32_t tbase;
    __shared__ int alive;
    __shared__ float bias[2 * kMaxW + kMaxOut];
    __shared__ float csum[TRAIN ? 4 : 1][TRAIN ? kMaxW : 1];
    __shared__ double lsum[kRowThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp >> 2;
    const int tile = blockIdx.x, m0 = tile * kRows;
    const int row = 32 * (warp & 3) + lane;
    const bool live_row = m0 + row < g.n;
    const int inP = pad32(g.in), hidP = pad32(g.hid), outP = pad32(g.out);
    const int ch = (hidP + kChunk - 1) / kChunk;  // chunks of a product with hid columns; one with out columns
    const int total = TRAIN ? 4 * ch + 1 : 2 * ch + 1;
    if (warp == 0) tc::tmem_alloc(&tbase, kCols);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&done[b], 1);
        }
        fence_barrier_init();
        alive = 1;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tbase;
    chain_wait();

    // chunk q of the pass: its source, first column, columns and K
    auto chunk_of = [&](int q, const __nv_bfloat16 *&src, int &col0, int &cols, int &kp) {
        int width = hidP;
        if (q < ch) { src = g.f1; kp = inP; }
        else if ((q -= ch) < ch) { src = g.f2; kp = hidP; }
        else if ((q -= ch) < 1) { src = g.f3; kp = hidP; width = outP; }
        else if ((q -= 1) < ch) { src = g.g3; kp = outP; }
        else { q -= ch; src = g.g2; kp = hidP; }
        col0 = q * kChunk;
        cols = min(kChunk, width - col0);
        src += static_cast<size_t>(col0) * kp;
    };
    int loaded = 0;  // thread 0: chunks fetched
    auto fetch = [&](int q) {
        if (q >= total) return;
        const __nv_bfloat16 *src;
        int col0, cols, kp;
        chunk_of(q, src, col0, cols, kp);
        const uint32_t bytes = static_cast<uint32_t>(cols) * kp * 2;
        mbar_arrive_expect_tx(&full[q & 1], bytes);
        bulk_g2s(Ws[q & 1], src, bytes, &full[q & 1]);
        loaded = q + 1;
    };
    if (threadIdx.x == 0) {
        fetch(0);
        fetch(1);
    }
    for (int j = threadIdx.x; j < 2 * kMaxW + kMaxOut; j += kRowThreads) {
        const int l = j < kMaxW ? 0 : (j < 2 * kMaxW ? 1 : 2), c = j - l * kMaxW;
        const float *b = l == 0 ? g.b1 : (l == 1 ? g.b2 : g.b3);
        bias[j] = c < (l == 2 ? g.out : g.hid) ? b[c] : 0.0f;
    }
    // the input rows as an image: a warp takes 8 rows x 4 groups of 8 columns at a time (128-byte runs of each
    // row, conflict-free 16-byte stores); columns beyond `in` and rows beyond n are zero
    {
        const int r8 = lane & 7, kg = lane >> 3;
        const int kblocks = inP / 32;  // 32 columns each
        const bool pairs = (g.in & 1) == 0 && (reinterpret_cast<uintptr_t>(g.x) & 7) == 0;
        for (int it = warp; it < (kRows / 8) * kblocks; it += kRowThreads / 32) {
            const int r = 8 * (it / kblocks) + r8, k = 32 * (it % kblocks) + 8 * kg;
            const float *src = g.x + static_cast<size_t>(m0 + r) * g.in + k;
            float v[8];
            const bool ok = m0 + r < g.n;
            if (pairs) {
#pragma unroll
                for (int q = 0; q < 8; q += 2) {
                    float2 p = make_float2(0.0f, 0.0f);
                    if (ok && k + q < g.in) p = __ldg(reinterpret_cast<const float2 *>(src + q));
                    v[q] = p.x;
                    v[q + 1] = p.y;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = (ok && k + q < g.in) ? __ldg(src + q) : 0.0f;
            }
            const uint4 w = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                                       pack_bf16(v[6], v[7]));
            *reinterpret_cast<uint4 *>(As + img(r, k, inP)) = w;
        }
    }

    // Starts the products of chunks [q0, q0 + nq) on the image in As (everyone's stores visible to the tensor core
    // first) ...
    auto start = [&](int q0, int nq) {
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (threadIdx.x == 0 && alive)
            for (int q = q0; q < q0 + nq; ++q) {
                const __nv_bfloat16 *src;
                int col0, cols, kp;
                chunk_of(q, src, col0, cols, kp);
                if (!mbar_wait_bounded(&full[q & 1], (q >> 1) & 1)) {
                    alive = 0;
                    break;
                }
                issue_product(tmem + col0, As, Ws[q & 1], kp, cols, false);
                tc::commit(&done[q & 1]);
            }
    };
    // ... and waits for them, fetching the next chunks into the freed buffers.
    auto finish = [&](int q0, int nq) {
        if (threadIdx.x == 0 && alive)
            for (int q = q0; q < q0 + nq; ++q) {
                if (!mbar_wait_bounded(&done[q & 1], (q >> 1) & 1)) {
                    mbar_wait_bounded(&done[q & 1], (q >> 1) & 1);  // drain before the buffers go
                    alive = 0;
                    break;
                }
                fetch(q + 2);
            }
        __syncthreads();
        tc::fence_after_sync();
    };

    const float nan = __int_as_float(0x7fc00000);
    uint32_t mask[2][kMaxW / (32 * kGroups)];
    // hidden layers: bias, ReLU, the next image
    auto hidden = [&](int l) {
#pragma unroll
        for (int u = 0; u < kMaxW / (32 * kGroups); ++u) {
            const int c0 = 32 * (kGroups * u + group);
            if (c0 >= hidP) continue;
            float v[32];
            tc::tmem_ld32(tc::tmem_addr(tmem, warp, c0), v);
            uint32_t bits = 0;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float a = fmaxf(v[j] + bias[l * kMaxW + c0 + j], 0.0f);
                v[j] = live_row ? a : 0.0f;
                bits |= (v[j] > 0.0f ? 1u : 0u) << j;
            }
            mask[l][u] = bits;
            store_image(As, row, c0, hidP, v);
        }
        tc::fence_before_sync();
    };
    // backward: ReLU mask, column sums, the next image
    auto hidden_back = [&](int l, int db0) {
#pragma unroll
        for (int u = 0; u < kMaxW / (32 * kGroups); ++u) {
            const int c0 = 32 * (kGroups * u + group);
            if (c0 >= hidP) continue;
            float v[32];
            tc::tmem_ld32(tc::tmem_addr(tmem, warp, c0), v);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = (mask[l][u] >> j & 1u) ? v[j] : 0.0f;
            store_image(As, row, c0, hidP, v);
            csum[TRAIN ? warp & 3 : 0][TRAIN ? c0 + lane : 0] = column_sums(v, lane);
        }
        tc::fence_before_sync();
        __syncthreads();
        for (int c = threadIdx.x; c < hidP; c += kRowThreads)
            g.db[static_cast<size_t>(tile) * (2 * hidP + outP) + db0 + c] =
                (csum[0][c] + csum[TRAIN ? 1 : 0][c]) + (csum[TRAIN ? 2 : 0][c] + csum[TRAIN ? 3 : 0][c]);
    };
    const size_t tileI = static_cast<size_t>(tile) * kRows;

    start(0, ch);
    if (TRAIN) write_transposed(As, inP, g.xt + tileI * pad128(g.in));
    finish(0, ch);
    hidden(0);
    start(ch, ch);
    if (TRAIN) write_transposed(As, hidP, g.a1t + tileI * pad128(g.hid));
    finish(ch, ch);
    hidden(1);
    start(2 * ch, 1);
    if (TRAIN) write_transposed(As, hidP, g.a2t + tileI * pad128(g.hid));
    finish(2 * ch, 1);
    if constexpr (!TRAIN) {
        // the rows of y are contiguous: gathered in shared memory (the image is no longer needed), then copied
        float *ys = reinterpret_cast<float *>(dyn);
        const bool ok = alive != 0;
        for (int c0 = 32 * group; c0 < outP; c0 += 32 * kGroups) {
            float v[32];
            tc::tmem_ld32(tc::tmem_addr(tmem, warp, c0), v);
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (c0 + j < g.out) ys[row * g.out + c0 + j] = ok ? v[j] + bias[2 * kMaxW + c0 + j] : nan;
        }
        tc::fence_before_sync();
        __syncthreads();
        const int cnt = min(kRows, g.n - m0) * g.out;
        float *dst = g.y + static_cast<size_t>(m0) * g.out;
        for (int e = threadIdx.x; e < cnt; e += kRowThreads) dst[e] = ys[e];
    } else {
        double ss = 0.0;
        for (int c0 = 32 * group; c0 < outP; c0 += 32 * kGroups) {
            float v[32];
            tc::tmem_ld32(tc::tmem_addr(tmem, warp, c0), v);
            const float *t = g.t + static_cast<size_t>(m0 + row) * g.out + c0;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float dy = 0.0f;
                if (live_row && c0 + j < g.out) {
                    const float d = v[j] + bias[2 * kMaxW + c0 + j] - __ldg(t + j);
                    dy = 2.0f * d * g.scale;
                    ss += static_cast<double>(d) * d;
                }
                v[j] = dy;
            }
            store_image(As, row, c0, outP, v);
            csum[warp & 3][c0 + lane] = column_sums(v, lane);
        }
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
        if (lane == 0) lsum[warp] = ss;
        tc::fence_before_sync();
        __syncthreads();
        for (int c = threadIdx.x; c < outP; c += kRowThreads)
            g.db[static_cast<size_t>(tile) * (2 * hidP + outP) + 2 * hidP + c] =
                (csum[0][c] + csum[1][c]) + (csum[2][c] + csum[3][c]);
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < kRowThreads / 32; ++w) s += lsum[w];
            g.loss[tile] = alive ? s : static_cast<double>(nan);
        }
        start(2 * ch + 1, ch);
        write_transposed(As, outP, g.dyt + tileI * outP);
        finish(2 * ch + 1, ch);
        hidden_back(1, hidP);
        start(3 * ch + 1, ch);
        write_transposed(As, hidP, g.dz2t + tileI * pad128(g.hid));
        finish(3 * ch + 1, ch);
        hidden_back(0, 0);
        tc::fence_before_sync();
        __syncthreads();
        write_transposed(As, hidP, g.dz1t + tileI * pad128(g.hid));
        if (!alive) {  // a product is missing: no gradient may look valid
            __syncthreads();
            for (int c = threadIdx.x; c < 2 * hidP + outP; c += kRowThreads)
                g.db[static_cast<size_t>(tile) * (2 * hidP + outP) + c] = nan;
            const __nv_bfloat16 bn = __float2bfloat16_rn(nan);
            for (int e = threadIdx.x; e < kRows * hidP; e += kRowThreads) {
                g.dz1t[tileI * pad128(g.hid) + e] = bn;
                g.dz2t[tileI * pad128(g.hid) + e] = bn;
                if (e < kRows * outP) g.dyt[tileI * outP + e] = bn;
            }
        }
    }
    if (threadIdx.x == 0 && !alive)  // copies still in flight land before the block's shared memory is released
        for (int q = max(0, loaded - 2); q < loaded; ++q) mbar_wait_bounded(&full[q & 1], (q >> 1) & 1);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kCols);
}

// One output tile of a weight gradient over a range of row tiles: rows m0 .. + 127 of A^T B, columns n0 .. + cols.
struct GradArgs {
    const __nv_bfloat16 *xt, *a1t, *a2t, *dyt, *dz2t, *dz1t;
    float *partial;     // [splits][nparam], in the layout of the parameters
    long long nparam;
    int in, hid, out, tiles, splits;
};

// grid (output tiles, splits).  Split s takes row tiles [s tiles / splits, (s + 1) tiles / splits); both operands
// of a row tile are contiguous 128-feature blocks, two row tiles in flight.
__global__ void __launch_bounds__(kThreads) mlp_wgrad_kernel(GradArgs g) {
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ __align__(8) uint64_t full[2], done[2];
    __shared__ uint32_t tbase;
    __shared__ int alive;
    constexpr size_t kOp = static_cast<size_t>(kChunk) * kRows * 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hidP = pad32(g.hid), outP = pad32(g.out);
    const int mi = (g.in + kChunk - 1) / kChunk, mh = (g.hid + kChunk - 1) / kChunk;
    int q = blockIdx.x;
    const __nv_bfloat16 *A, *B;
    int fa, fb, mw, nw, m0, n0;       // features per tile of A and B, true widths, first feature and column
    long long off;                    // first parameter
    if (q < mi * mh) {                // dW1 = X^T dZ1
        A = g.xt; B = g.dz1t; fa = pad128(g.in); fb = pad128(g.hid); mw = g.in; nw = g.hid; off = 0;
        m0 = (q / mh) * kChunk; n0 = (q % mh) * kChunk;
    } else if ((q -= mi * mh) < mh * mh) {  // dW2 = A1^T dZ2
        A = g.a1t; B = g.dz2t; fa = pad128(g.hid); fb = pad128(g.hid); mw = g.hid; nw = g.hid;
        off = static_cast<long long>(g.in) * g.hid + g.hid;
        m0 = (q / mh) * kChunk; n0 = (q % mh) * kChunk;
    } else {                          // dW3 = A2^T dY
        q -= mh * mh;
        A = g.a2t; B = g.dyt; fa = pad128(g.hid); fb = outP; mw = g.hid; nw = g.out;
        off = static_cast<long long>(g.in) * g.hid + 2LL * g.hid + static_cast<long long>(g.hid) * g.hid;
        m0 = q * kChunk; n0 = 0;
    }
    const int cols = min(kChunk, (nw == g.out && B == g.dyt ? outP : hidP) - n0);
    const int t0 = static_cast<int>(static_cast<long long>(blockIdx.y) * g.tiles / g.splits);
    const int t1 = static_cast<int>(static_cast<long long>(blockIdx.y + 1) * g.tiles / g.splits);
    if (warp == 0) tc::tmem_alloc(&tbase, kChunk);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&done[b], 1);
        }
        fence_barrier_init();
        alive = 1;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tbase;
    chain_wait();
    if (threadIdx.x == 0) {
        const uint32_t abytes = kOp, bbytes = static_cast<uint32_t>(cols) * kRows * 2;
        auto fetch = [&](int i) {
            unsigned char *s = dyn + (i & 1) * 2 * kOp;
            const size_t tr = static_cast<size_t>(t0 + i) * kRows;
            mbar_arrive_expect_tx(&full[i & 1], abytes + bbytes);
            bulk_g2s(s, A + tr * fa + static_cast<size_t>(m0) * kRows, abytes, &full[i & 1]);
            bulk_g2s(s + kOp, B + tr * fb + static_cast<size_t>(n0) * kRows, bbytes, &full[i & 1]);
        };
        const int nt = t1 - t0;
        int loaded = 0;
        while (loaded < min(2, nt)) fetch(loaded++);
        for (int i = 0; i < nt && alive; ++i) {
            unsigned char *s = dyn + (i & 1) * 2 * kOp;
            if (!mbar_wait_bounded(&full[i & 1], (i >> 1) & 1)) {
                alive = 0;
                break;
            }
            issue_product(tmem, s, s + kOp, kRows, cols, i > 0);
            tc::commit(&done[i & 1]);
            if (!mbar_wait_bounded(&done[i & 1], (i >> 1) & 1)) {
                mbar_wait_bounded(&done[i & 1], (i >> 1) & 1);
                alive = 0;
                break;
            }
            if (loaded < nt) fetch(loaded++);
        }
        if (!alive)
            for (int i = max(0, loaded - 2); i < loaded; ++i) mbar_wait_bounded(&full[i & 1], (i >> 1) & 1);
    }
    __syncthreads();
    tc::fence_after_sync();
    const int m = m0 + 32 * (warp & 3) + lane;
    float *P = g.partial + static_cast<size_t>(blockIdx.y) * g.nparam + off + static_cast<long long>(m) * nw;
    const bool ok = alive != 0;
    for (int c0 = 32 * (warp >> 2); c0 < cols; c0 += 64) {
        float v[32];
        tc::tmem_ld32(tc::tmem_addr(tmem, warp, c0), v);
        if (m >= mw) continue;
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (n0 + c0 + j < nw) P[n0 + c0 + j] = ok ? v[j] : __int_as_float(0x7fc00000);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kChunk);
}

// Positions of a parameter in the weights' images.
struct Images {
    __nv_bfloat16 *f1, *f2, *f3, *g3, *g2;
    int in, hid, out;
};
__device__ __forceinline__ void write_images(const Images &w, long long i, float p) {
    const int hidP = pad32(w.hid);
    const __nv_bfloat16 b = __float2bfloat16_rn(p);
    long long o = i;
    if (o < static_cast<long long>(w.in) * w.hid) {
        const int a = static_cast<int>(o / w.hid), c = static_cast<int>(o % w.hid);
        w.f1[img(c, a, pad32(w.in))] = b;
        return;
    }
    o -= static_cast<long long>(w.in) * w.hid + w.hid;
    if (o >= 0 && o < static_cast<long long>(w.hid) * w.hid) {
        const int a = static_cast<int>(o / w.hid), c = static_cast<int>(o % w.hid);
        w.f2[img(c, a, hidP)] = b;
        w.g2[img(a, c, hidP)] = b;
        return;
    }
    o -= static_cast<long long>(w.hid) * w.hid + w.hid;
    if (o >= 0 && o < static_cast<long long>(w.hid) * w.out) {
        const int a = static_cast<int>(o / w.out), c = static_cast<int>(o % w.out);
        w.f3[img(c, a, hidP)] = b;
        w.g3[img(a, c, pad32(w.out))] = b;
    }
}

__global__ void mlp_images_kernel(Images w, const float *p, long long count) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i < count) write_images(w, i, p[i]);
}

struct FinishArgs {
    const float *partial, *db;
    float *grads, *p, *m, *v;
    long long nparam;
    int tiles, splits, adam;
    float lr, b1, b2, c1, c2, eps;
};

// Gradient of each parameter: its partial sums over the splits (weights) or the row tiles (biases) in order; with
// `adam`, the optimiser step and the weight's new images.
__global__ void mlp_finish_kernel(FinishArgs g, Images w) {
    chain_wait();
    const int hidP = pad32(w.hid), outP = pad32(w.out), ldb = 2 * hidP + outP;
    const long long o1 = static_cast<long long>(w.in) * w.hid, o2 = o1 + w.hid + static_cast<long long>(w.hid) * w.hid,
                    o3 = o2 + w.hid + static_cast<long long>(w.hid) * w.out;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < g.nparam;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int col = (i >= o1 && i < o1 + w.hid)   ? static_cast<int>(i - o1)
                        : (i >= o2 && i < o2 + w.hid) ? hidP + static_cast<int>(i - o2)
                        : i >= o3                     ? 2 * hidP + static_cast<int>(i - o3)
                                                      : -1;
        const float *src = col >= 0 ? g.db + col : g.partial + i;
        const long long ld = col >= 0 ? ldb : g.nparam;
        const int cnt = col >= 0 ? g.tiles : g.splits;
        float s = 0.0f;
        int k = 0;
        for (; k + 4 <= cnt; k += 4) {
            const float a = src[k * ld], b = src[(k + 1) * ld], c = src[(k + 2) * ld], d = src[(k + 3) * ld];
            s += (a + b) + (c + d);
        }
        for (; k < cnt; ++k) s += src[k * ld];
        g.grads[i] = s;
        if (g.adam) {
            const float mi = g.b1 * g.m[i] + (1.0f - g.b1) * s;
            const float vi = g.b2 * g.v[i] + (1.0f - g.b2) * s * s;
            g.m[i] = mi;
            g.v[i] = vi;
            const float p = g.p[i] - g.lr * (mi / g.c1) / (sqrtf(vi / g.c2) + g.eps);
            g.p[i] = p;
            write_images(w, i, p);
        }
    }
}

}  // namespace mlpk
}  // namespace cufil
