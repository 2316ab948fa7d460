// fcm_fft.cuh -- the Stokes solve of the force-coupling method on a grid of
// which only the rows near particles are used: forward transform, spectral
// projector and inverse transform in five passes.
//
//   x     real rows -> half spectra          rows that a particle's support touches
//   y     complex, along y                   planes that hold such a row
//   z     complex, along z; the projector; back along z, in one pass
//   y, x  back                               planes and rows as above
//
// A row that no particle's support touches holds zeros, so its transform is
// zero and is neither formed nor read; and the velocities are read only where
// the forces were spread, so nothing else is formed on the way back.  With
// particles everywhere this is the full transform.
//
// What bounds it.  Every pass moves each value once, 64 bytes or more at a
// time (z: read, three transforms forward, projector, three back, write).  The
// x and y passes run near the memory's rate, z at the latency of its chain of
// stages (z_kernel); a library transform of the whole grid takes six passes and
// the projector a seventh, on every point.  At 512^3 with 28% of the planes used (10,000 blobs and 20,000
// segments on a sphere, and their neighbourhood) the five passes take 88 + 207 +
// 851 + 172 + 82 us, the library's two transforms, the projector and the clearing
// of whole grids 5.8 ms.
//
// One transform: lengths 2^a 3^b 5^c in stages of radix 8, 5, 4, 3 and 2, in
// place in shared memory.  Forward stages run from the whole length down
// (decimation in frequency) and leave the frequencies in digit-reversed
// places; inverse stages run back up from there, so nothing is ever reordered:
// the projector looks up the frequency of a place, and y keeps its places in
// memory.  The first and last stages read and write global memory directly.
#pragma once

#include <cmath>
#include <vector>

#include "fcm_plan.cuh"
#include "packed.cuh"

namespace cufil {
namespace fftk {

constexpr int kCols = 8;       // kx columns of a block: 64 bytes of each row

// One axis: length, radices (forward order), twiddles exp(-2 pi i k / n), frequency of each place.
struct Axis {
    int n, ns;
    int radix[kMaxStages];
    const float2 *tw;  // [n]
    const int *freq;   // [n] frequency 0 .. n-1 of place p
    const int *place;  // [n] place of frequency k
};

struct Grid {
    int nx, ny, nz, mx, ldx;  // mx = nx / 2 complex points of a real row; ldx: row stride of the spectra
    Axis x, y, z;             // x: the complex transform of mx points
    const float2 *wx;         // [mx + 1] exp(-2 pi i k / nx)
    float *real;              // [3][nz][ny][nx]
    float2 *spec;             // [3][nz][ny][ldx]
    const unsigned *row_bits;         // [nz][words] one bit per row y: a particle's support touches it
    int words;
    const unsigned char *plane_used;  // [nz]
    const int *rows, *planes;         // used rows (z ny + y) and planes
    const int *counts;                // [0] used rows, [1] used planes
    float Lx, Ly, Lz;
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// The transforms are written for a real type T: float (one row along x) or F2, the same value of two adjacent columns.
template <class T>
struct Cx {
    T x, y;
};
template <class T>
__device__ __forceinline__ Cx<T> operator+(Cx<T> a, Cx<T> b) {
    return {vadd(a.x, b.x), vadd(a.y, b.y)};
}
template <class T>
__device__ __forceinline__ Cx<T> operator-(Cx<T> a, Cx<T> b) {
    return {vsub(a.x, b.x), vsub(a.y, b.y)};
}
// s + r b and s - r b with r = -i (forward) or i (inverse): no negation is formed.
template <bool INV, class T>
__device__ __forceinline__ void add_sub_rot(Cx<T> s, Cx<T> b, Cx<T> &sum, Cx<T> &diff) {
    const Cx<T> up = {vadd(s.x, b.y), vsub(s.y, b.x)}, down = {vsub(s.x, b.y), vadd(s.y, b.x)};
    sum = INV ? down : up;
    diff = INV ? up : down;
}

template <bool INV, class T>
__device__ __forceinline__ void dft3(Cx<T> *a) {
    const T s = splat<T>(0.86602540378443864676f), h = splat<T>(-0.5f);
    const Cx<T> t = a[1] + a[2], d = a[1] - a[2];
    const Cx<T> m = {vfma(h, t.x, a[0].x), vfma(h, t.y, a[0].y)};
    a[0] = a[0] + t;
    add_sub_rot<INV>(m, Cx<T>{vmul(s, d.x), vmul(s, d.y)}, a[1], a[2]);
}
template <bool INV, class T>
__device__ __forceinline__ void dft4(Cx<T> &a0, Cx<T> &a1, Cx<T> &a2, Cx<T> &a3) {
    const Cx<T> s = a0 + a2, d = a0 - a2, t = a1 + a3, e = a1 - a3;
    a0 = s + t;
    a2 = s - t;
    add_sub_rot<INV>(d, e, a1, a3);
}
template <bool INV, class T>
__device__ __forceinline__ void dft5(Cx<T> *a) {
    const T c1 = splat<T>(0.30901699437494742410f), c2 = splat<T>(-0.80901699437494742410f);
    const T s1 = splat<T>(0.95105651629515357212f), s2 = splat<T>(0.58778525229247312917f);
    const T s3 = splat<T>(-0.95105651629515357212f);
    const Cx<T> t1 = a[1] + a[4], t2 = a[2] + a[3], d1 = a[1] - a[4], d2 = a[2] - a[3];
    const Cx<T> m1 = {vfma(c1, t1.x, vfma(c2, t2.x, a[0].x)), vfma(c1, t1.y, vfma(c2, t2.y, a[0].y))};
    const Cx<T> m2 = {vfma(c2, t1.x, vfma(c1, t2.x, a[0].x)), vfma(c2, t1.y, vfma(c1, t2.y, a[0].y))};
    const Cx<T> e1 = {vfma(s1, d1.x, vmul(s2, d2.x)), vfma(s1, d1.y, vmul(s2, d2.y))};
    const Cx<T> e2 = {vfma(s2, d1.x, vmul(s3, d2.x)), vfma(s2, d1.y, vmul(s3, d2.y))};
    a[0] = a[0] + (t1 + t2);
    add_sub_rot<INV>(m1, e1, a[1], a[4]);
    add_sub_rot<INV>(m2, e2, a[2], a[3]);
}
template <bool INV, class T>
__device__ __forceinline__ void dft8(Cx<T> *a) {
    const T h = splat<T>(0.70710678118654752440f);
    Cx<T> e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6], o0 = a[1], o1 = a[3], o2 = a[5], o3 = a[7];
    dft4<INV>(e0, e1, e2, e3);
    dft4<INV>(o0, o1, o2, o3);
    // o_k times r^(k / 2), r = -i or i:  r^(1/2) = h (1 + r),  r^(3/2) = r h (1 + r)
    const T p1 = vmul(h, vadd(o1.x, o1.y)), m1 = vmul(h, vsub(o1.x, o1.y));
    const T p3 = vmul(h, vadd(o3.x, o3.y)), m3 = vmul(h, vsub(o3.x, o3.y));
    a[0] = e0 + o0;
    a[4] = e0 - o0;
    add_sub_rot<INV>(e2, o2, a[2], a[6]);
    if (INV) {  // (m1, p1) and (-p3, m3)
        a[1] = {vadd(e1.x, m1), vadd(e1.y, p1)};
        a[5] = {vsub(e1.x, m1), vsub(e1.y, p1)};
        a[3] = {vsub(e3.x, p3), vadd(e3.y, m3)};
        a[7] = {vadd(e3.x, p3), vsub(e3.y, m3)};
    } else {  // (p1, -m1) and (-m3, -p3)
        a[1] = {vadd(e1.x, p1), vsub(e1.y, m1)};
        a[5] = {vsub(e1.x, p1), vadd(e1.y, m1)};
        a[3] = {vsub(e3.x, m3), vsub(e3.y, p3)};
        a[7] = {vadd(e3.x, m3), vadd(e3.y, p3)};
    }
}
template <int R, bool INV, class T>
__device__ __forceinline__ void dft(Cx<T> *a) {
    if constexpr (R == 8) {
        dft8<INV>(a);
    } else if constexpr (R == 5) {
        dft5<INV>(a);
    } else if constexpr (R == 4) {
        dft4<INV>(a[0], a[1], a[2], a[3]);
    } else if constexpr (R == 3) {
        dft3<INV>(a);
    } else {
        const Cx<T> t = a[1];
        a[1] = a[0] - t;
        a[0] = a[0] + t;
    }
}

// Elements in memory: complex numbers along x and in the grids; in the shared arrays of y and z a pair of columns is
// kept as (re, re, im, im), ready for the packed instructions.
__device__ __forceinline__ Cx<float> load_complex(const float2 *p) {
    const float2 q = *p;
    return {q.x, q.y};
}
__device__ __forceinline__ void store_complex(float2 *p, Cx<float> v) { *p = make_float2(v.x, v.y); }
__device__ __forceinline__ Cx<F2> load_columns(const float4 *p) {
    const float4 q = *p;
    return {pack2(q.x, q.z), pack2(q.y, q.w)};
}
__device__ __forceinline__ void store_columns(float4 *p, Cx<F2> v) {
    const float2 re = unpack2(v.x), im = unpack2(v.y);
    *p = make_float4(re.x, im.x, re.y, im.y);
}
__device__ __forceinline__ Cx<F2> load_pair(const ulonglong2 *p) {
    const ulonglong2 q = *p;
    return {F2{q.x}, F2{q.y}};
}
__device__ __forceinline__ void store_pair(ulonglong2 *p, Cx<F2> v) { *p = make_ulonglong2(v.x.v, v.y.v); }

// Place of element p of a line in shared memory: one element of padding per eight keeps the strided accesses of the
// short stages off the same banks.
__host__ __device__ constexpr int padded(int p) { return p + (p >> 3); }

// The stages of a length known at compile time (N > 0): the same radices as radices() below, so that strides,
// places and twiddle steps are constants.  N = 0 takes them from the Axis.
__host__ __device__ constexpr int radix_of(int n) { return n % 8 == 0 ? 8 : n % 5 == 0 ? 5 : n % 4 == 0 ? 4 : n % 3 == 0 ? 3 : 2; }
__host__ __device__ constexpr int len_at(int n, int s) {
    while (s-- > 0) n /= radix_of(n);
    return n;
}
__host__ __device__ constexpr int stages_of(int n) {
    int c = 0;
    while (n > 1) {
        n /= radix_of(n);
        ++c;
    }
    return c;
}

// The threads that share one set of lines: a block, or (rows along x) a warp.
struct BlockTeam {
    __device__ static int rank() { return threadIdx.x; }
    __device__ static int size() { return blockDim.x; }
    __device__ static void sync() { __syncthreads(); }
};
struct WarpTeam {
    __device__ static int rank() { return threadIdx.x & 31; }
    __device__ static int size() { return 32; }
    __device__ static void sync() { __syncwarp(); }
};

// One stage of SETS x 2^LINES transforms with block length ls and radix R (m = ls / R): work items (butterfly, line),
// lines fastest; an item takes element j of block b of every set, over load(set, line, place, padded place) and
// store(set, line, place, padded place, value), with one set of twiddles.  Forward: transform, then output p by
// w^(j p); inverse: input p by conj w^(j p), then transform; w = exp(-2 pi i / ls) = tw[n / ls].  N > 0: the length,
// and LS the block length, at compile time.
template <class Team, int R, bool INV, class T, int N, int LS, int LINES, int SETS, class Load, class Store>
__device__ __forceinline__ void stage_items(const Axis &ax, int ls_, Load load, Store store) {
    const int n = N ? N : ax.n, ls = N ? LS : ls_;
    const int m = ls / R, tstep = n / ls, total = (n / R) << LINES;
    constexpr int kM = N ? LS / R : 0;
    for (int it = Team::rank(); it < total; it += Team::size()) {
        const int line = it & ((1 << LINES) - 1), bf = it >> LINES;
        const int b = bf / m, j = bf - b * m;
        const int base = b * ls + j, pbase = padded(base);
        auto off = [&](int q) {
            if constexpr (kM > 0 && kM % 8 == 0) return pbase + q * (kM + kM / 8);
            else if constexpr (kM == 1 && R == 8) return pbase + q;
            else return padded(base + q * m);
        };
        T wx[R], wy[R], wn[R];  // w and -Im w; the inverse takes the conjugate
        if constexpr (kM != 1) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                const float2 w = __ldg(ax.tw + j * q * tstep);
                wx[q] = splat<T>(w.x);
                wy[q] = splat<T>(INV ? -w.y : w.y);
                wn[q] = splat<T>(INV ? w.y : -w.y);
            }
        }
        auto twiddle = [&](Cx<T> *a) {
            if constexpr (kM != 1)
#pragma unroll
            for (int q = 1; q < R; ++q)
                a[q] = {vfma(a[q].x, wx[q], vmul(a[q].y, wn[q])), vfma(a[q].x, wy[q], vmul(a[q].y, wx[q]))};
        };
        // the next set's elements are read before this one is stored, so that their latency is hidden
        Cx<T> a[SETS > 1 ? 2 : 1][R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[0][q] = load(0, line, base + q * m, off(q));
#pragma unroll
        for (int set = 0; set < SETS; ++set) {
            Cx<T> *c = a[SETS > 1 ? set & 1 : 0];
            if (set + 1 < SETS)
#pragma unroll
                for (int q = 0; q < R; ++q) a[SETS > 1 ? (set + 1) & 1 : 0][q] = load(set + 1, line, base + q * m, off(q));
            if constexpr (!INV) dft<R, false>(c);
            twiddle(c);
            if constexpr (INV) dft<R, true>(c);
#pragma unroll
            for (int q = 0; q < R; ++q) store(set, line, base + q * m, off(q), c[q]);
        }
    }
}

// Stage S of a fixed length, or stage s of an Axis with block length ls.
template <class Team, int N, int S, bool INV, class T, int LINES, int SETS, class Load, class Store>
__device__ __forceinline__ void stage(const Axis &ax, int s, int ls, Load load, Store store) {
    if constexpr (N > 0) {
        constexpr int kLs = len_at(N, S);
        stage_items<Team, radix_of(kLs), INV, T, N, kLs, LINES, SETS>(ax, ls, load, store);
    } else {
        switch (ax.radix[s]) {
            case 8: stage_items<Team, 8, INV, T, 0, 0, LINES, SETS>(ax, ls, load, store); break;
            case 5: stage_items<Team, 5, INV, T, 0, 0, LINES, SETS>(ax, ls, load, store); break;
            case 4: stage_items<Team, 4, INV, T, 0, 0, LINES, SETS>(ax, ls, load, store); break;
            case 3: stage_items<Team, 3, INV, T, 0, 0, LINES, SETS>(ax, ls, load, store); break;
            default: stage_items<Team, 2, INV, T, 0, 0, LINES, SETS>(ax, ls, load, store); break;
        }
    }
}

// The stages between the first and the last, in place in shared memory, each followed by a barrier; forward they
// run down from stage S, inverse up from stage S.
template <class Team, int N, int S, class T, int LINES, int SETS, class Load, class Store>
__device__ __forceinline__ void middle_forward(const Axis &ax, Load load, Store store) {
    if constexpr (N > 0) {
        if constexpr (S + 1 < stages_of(N)) {
            stage<Team, N, S, false, T, LINES, SETS>(ax, S, 0, load, store);
            Team::sync();
            middle_forward<Team, N, S + 1, T, LINES, SETS>(ax, load, store);
        }
    } else {
        int ls = ax.n / ax.radix[0];
        for (int s = 1; s < ax.ns - 1; ++s) {
            stage<Team, 0, 0, false, T, LINES, SETS>(ax, s, ls, load, store);
            ls /= ax.radix[s];
            Team::sync();
        }
    }
}
template <class Team, int N, int S, class T, int LINES, int SETS, class Load, class Store>
__device__ __forceinline__ void middle_inverse(const Axis &ax, Load load, Store store) {
    if constexpr (N > 0) {
        if constexpr (S > 0) {
            stage<Team, N, S, true, T, LINES, SETS>(ax, S, 0, load, store);
            Team::sync();
            middle_inverse<Team, N, S - 1, T, LINES, SETS>(ax, load, store);
        }
    } else {
        int ls = ax.radix[ax.ns - 1];
        for (int s = ax.ns - 2; s > 0; --s) {
            ls *= ax.radix[s];
            stage<Team, 0, 0, true, T, LINES, SETS>(ax, s, ls, load, store);
            Team::sync();
        }
    }
}
template <int N>
constexpr int last_stage() {
    return N > 0 ? stages_of(N) - 1 : 0;
}

// ---------------------------------------------------------------- which rows are used
// One block per plane: its used rows appended to `rows`, the plane to `planes`.
__global__ void __launch_bounds__(256) list_rows_kernel(const unsigned *__restrict__ row_bits, int words, int ny,
                                                        unsigned char *plane_used, int *rows, int *planes,
                                                        int *counts) {
    __shared__ int base, warp_off[9];
    const int z = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int found = 0;
    for (int y0 = 0; y0 < ny; y0 += blockDim.x) {
        const int y = y0 + threadIdx.x;
        const bool used = y < ny && (row_bits[static_cast<size_t>(z) * words + (y >> 5)] >> (y & 31) & 1u);
        const unsigned bits = __ballot_sync(0xffffffffu, used);
        if (lane == 0) warp_off[w] = __popc(bits);
        __syncthreads();
        if (threadIdx.x == 0) {
            int s = 0;
            for (int q = 0; q < 8; ++q) {
                const int c = warp_off[q];
                warp_off[q] = s;
                s += c;
            }
            warp_off[8] = s;
            base = s ? atomicAdd(counts, s) : 0;
        }
        __syncthreads();
        if (used) rows[base + warp_off[w] + __popc(bits & ((1u << lane) - 1u))] = z * ny + y;
        found |= warp_off[8];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        plane_used[z] = found ? 1 : 0;
        if (found) planes[atomicAdd(counts + 1, 1)] = z;
    }
}

// Zeroes the used rows of the three real grids, a warp per row (16 bytes a lane where the rows allow it).
__global__ void __launch_bounds__(256) clear_rows_kernel(Grid g) {
    const int n = g.counts[0], lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    const size_t gs = static_cast<size_t>(g.nx) * g.ny * g.nz;
    for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
        float *p = g.real + static_cast<size_t>(g.rows[i]) * g.nx;
        for (int c = 0; c < 3; ++c, p += gs) {
            if ((g.nx & 3) == 0)
                for (int x = lane; x < g.nx / 4; x += 32)
                    reinterpret_cast<float4 *>(p)[x] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            else
                for (int x = lane; x < g.nx / 2; x += 32) reinterpret_cast<float2 *>(p)[x] = make_float2(0.0f, 0.0f);
        }
    }
}

// ---------------------------------------------------------------- x: real rows <-> half spectra
// A warp takes one used row of one component at a time, in its own part of the shared memory: no block barriers.
// The row's nx reals are mx = nx / 2 complex numbers z; their transform Z gives the row's half spectrum as
// X(k) = E + w^k O, E = (Z(k) + Z*(mx - k)) / 2, O = -i (Z(k) - Z*(mx - k)) / 2, w = exp(-2 pi i / nx), and back as
// Z(k) = (X(k) + X*(mx - k)) + i w^-k (X(k) - X*(mx - k)) (unnormalised, so twice the sums above; the imaginary parts
// of X(0) and X(mx) count as zero, as in any complex-to-real transform).
// Short rows go two or four to a warp, so that a stage has a butterfly for every lane (x_lines).
constexpr int kRowWarps = 8;
__host__ __device__ constexpr int x_lines(int n) { return n == 64 ? 2 : (n == 0 || n == 128) ? 1 : 0; }  // log2; n = 0: any
template <int N>  // N: mx, or 0
__global__ void __launch_bounds__(32 * kRowWarps) x_forward_kernel(Grid g) {
    extern __shared__ __align__(16) float2 xs[];
    constexpr int kL = x_lines(N), kLines = 1 << kL;
    const int mx = N ? N : g.mx, nrows = g.counts[0], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int stride = padded(mx) + 1;
    const size_t gs = static_cast<size_t>(g.nx) * g.ny * g.nz, ss = static_cast<size_t>(g.ldx) * g.ny * g.nz;
    float2 *row = xs + w * kLines * stride;
    auto from_smem = [&](int, int line, int, int pp) { return load_complex(row + line * stride + pp); };
    auto to_smem = [&](int, int line, int, int pp, Cx<float> v) { store_complex(row + line * stride + pp, v); };
    const float2 *real = reinterpret_cast<const float2 *>(g.real + blockIdx.y * gs);
    float2 *spec = g.spec + blockIdx.y * ss;
    for (int i = (blockIdx.x * kRowWarps + w) * kLines; i < nrows; i += gridDim.x * kRowWarps * kLines) {
        size_t r[kLines];  // a last warp with too few rows repeats its last one
#pragma unroll
        for (int l = 0; l < kLines; ++l) r[l] = g.rows[min(i + l, nrows - 1)];
        auto pick = [&](int line) {
            size_t v = r[0];
#pragma unroll
            for (int l = 1; l < kLines; ++l) v = line == l ? r[l] : v;
            return v;
        };
        auto from_row = [&](int, int line, int p, int) { return load_complex(real + pick(line) * mx + p); };
        stage<WarpTeam, N, 0, false, float, kL, 1>(g.x, 0, mx, from_row, to_smem);
        __syncwarp();
        middle_forward<WarpTeam, N, 1, float, kL, 1>(g.x, from_smem, to_smem);
        stage<WarpTeam, N, last_stage<N>(), false, float, kL, 1>(g.x, g.x.ns - 1, g.x.radix[g.x.ns - 1], from_smem, to_smem);
        __syncwarp();
        for (int k = lane; k <= mx; k += 32) {
            const int pa = padded(__ldg(g.x.place + (k == mx ? 0 : k))), pb = padded(__ldg(g.x.place + (k == 0 ? 0 : mx - k)));
            const float2 wk = __ldg(g.wx + k);
#pragma unroll
            for (int l = 0; l < kLines; ++l) {
                const float2 a = row[l * stride + pa], b = row[l * stride + pb];
                const float2 e = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
                const float2 o = make_float2(0.5f * (a.y + b.y), -0.5f * (a.x - b.x));
                spec[r[l] * g.ldx + k] = cadd(e, cmul(o, wk));
            }
        }
        __syncwarp();  // the next rows reuse the shared memory
    }
}

template <int N>
__global__ void __launch_bounds__(32 * kRowWarps) x_inverse_kernel(Grid g) {
    extern __shared__ __align__(16) float2 xs[];
    constexpr int kL = x_lines(N), kLines = 1 << kL;
    const int mx = N ? N : g.mx, nrows = g.counts[0], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int stride = padded(mx) + 1;
    const size_t gs = static_cast<size_t>(g.nx) * g.ny * g.nz, ss = static_cast<size_t>(g.ldx) * g.ny * g.nz;
    float2 *row = xs + w * kLines * stride;
    auto from_smem = [&](int, int line, int, int pp) { return load_complex(row + line * stride + pp); };
    auto to_smem = [&](int, int line, int, int pp, Cx<float> v) { store_complex(row + line * stride + pp, v); };
    float2 *real = reinterpret_cast<float2 *>(g.real + blockIdx.y * gs);
    const float2 *spec = g.spec + blockIdx.y * ss;
    for (int i = (blockIdx.x * kRowWarps + w) * kLines; i < nrows; i += gridDim.x * kRowWarps * kLines) {
        size_t r[kLines];
#pragma unroll
        for (int l = 0; l < kLines; ++l) r[l] = g.rows[min(i + l, nrows - 1)];
        auto pick = [&](int line) {
            size_t v = r[0];
#pragma unroll
            for (int l = 1; l < kLines; ++l) v = line == l ? r[l] : v;
            return v;
        };
        for (int k = lane; k < mx; k += 32) {
            float2 wk = __ldg(g.wx + k);
            wk.y = -wk.y;
            const int place = padded(__ldg(g.x.place + k));
#pragma unroll
            for (int l = 0; l < kLines; ++l) {
                const float2 *sp = spec + r[l] * g.ldx;
                float2 a = sp[k], b = sp[mx - k];
                if (k == 0) a.y = b.y = 0.0f;
                const float2 e = make_float2(a.x + b.x, a.y - b.y), d = make_float2(a.x - b.x, a.y + b.y);
                const float2 o = cmul(d, wk);
                row[l * stride + place] = make_float2(e.x - o.y, e.y + o.x);
            }
        }
        __syncwarp();
        stage<WarpTeam, N, last_stage<N>(), true, float, kL, 1>(g.x, g.x.ns - 1, g.x.radix[g.x.ns - 1], from_smem, to_smem);
        __syncwarp();
        middle_inverse<WarpTeam, N, last_stage<N>() - 1, float, kL, 1>(g.x, from_smem, to_smem);
        auto to_row = [&](int, int line, int p, int, Cx<float> v) { store_complex(real + pick(line) * mx + p, v); };
        stage<WarpTeam, N, 0, true, float, kL, 1>(g.x, 0, mx, from_smem, to_row);
        __syncwarp();
    }
}

// ---------------------------------------------------------------- y: complex, columns of 8 kx
// grid (kx blocks, planes in turn, components).  Unused rows read as zero on the way in and are not written on the
// way back; the spectra keep the digit-reversed places along y.
template <bool INV, int N>
__global__ void __launch_bounds__(256) y_kernel(Grid g) {
    extern __shared__ __align__(16) ulonglong2 ys[];
    constexpr int kL = 2, kLanes = 1 << kL;  // 4 lanes of two columns
    const int n = N ? N : g.ny, last = g.y.ns - 1, nplanes = g.counts[1];
    unsigned char *used = reinterpret_cast<unsigned char *>(ys + padded(n) * kLanes);  // [n] rows of the plane in use
    const size_t ss = static_cast<size_t>(g.ldx) * g.ny * g.nz;
    float2 *spec = g.spec + blockIdx.z * ss + static_cast<size_t>(blockIdx.x) * kCols;
    auto from_smem = [&](int, int line, int, int pp) { return load_pair(ys + pp * kLanes + line); };
    auto to_smem = [&](int, int line, int, int pp, Cx<F2> v) { store_pair(ys + pp * kLanes + line, v); };
    for (int i = blockIdx.y; i < nplanes; i += gridDim.y) {
        const int z = g.planes[i];
        float2 *plane = spec + static_cast<size_t>(z) * g.ny * g.ldx;
        for (int p = threadIdx.x; p < n; p += blockDim.x)
            used[p] = g.row_bits[static_cast<size_t>(z) * g.words + (p >> 5)] >> (p & 31) & 1u;
        __syncthreads();
        auto at = [&](int line, int p) { return reinterpret_cast<float4 *>(plane + static_cast<size_t>(p) * g.ldx) + line; };
        if constexpr (!INV) {
            auto from_used = [&](int, int line, int p, int) {
                return used[p] ? load_columns(at(line, p)) : Cx<F2>{};
            };
            auto to_all = [&](int, int line, int p, int, Cx<F2> v) { store_columns(at(line, p), v); };
            stage<BlockTeam, N, 0, false, F2, kL, 1>(g.y, 0, n, from_used, to_smem);
            __syncthreads();
            middle_forward<BlockTeam, N, 1, F2, kL, 1>(g.y, from_smem, to_smem);
            stage<BlockTeam, N, last_stage<N>(), false, F2, kL, 1>(g.y, last, g.y.radix[last], from_smem, to_all);
        } else {
            auto from_all = [&](int, int line, int p, int) { return load_columns(at(line, p)); };
            auto to_used = [&](int, int line, int p, int, Cx<F2> v) {
                if (used[p]) store_columns(at(line, p), v);
            };
            stage<BlockTeam, N, last_stage<N>(), true, F2, kL, 1>(g.y, last, g.y.radix[last], from_all, to_smem);
            __syncthreads();
            middle_inverse<BlockTeam, N, last_stage<N>() - 1, F2, kL, 1>(g.y, from_smem, to_smem);
            stage<BlockTeam, N, 0, true, F2, kL, 1>(g.y, 0, n, from_smem, to_used);
        }
        __syncthreads();  // the next plane reuses the shared array
    }
}

// ---------------------------------------------------------------- z, the projector, and z back
// u = (f - q (q.f) / q^2) / (q^2 n) per place, q = 0 removed (the spectral Stokes solve of stokes_kernel, fcm.cu).
__device__ __forceinline__ float reciprocal(float q) {  // the hardware approximation and one Newton step
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(q));
    return fmaf(r, fmaf(-q, r, 1.0f), r);
}
__device__ __forceinline__ void project(Cx<F2> &a, Cx<F2> &b, Cx<F2> &c, F2 q1, F2 q2, F2 q3, F2 inv_n) {
    const F2 qq = vfma(q1, q1, vfma(q2, q2, vmul(q3, q3)));
    const float2 q = unpack2(qq);
    const F2 qi = pack2(reciprocal(q.x), reciprocal(q.y));
    const F2 norm = vmul(qi, inv_n), w = vmul(vmul(splat<F2>(-1.0f), qi), norm);  // u = norm f - q (w (q.f)), w < 0
    const F2 kr = vmul(w, vfma(q1, a.x, vfma(q2, b.x, vmul(q3, c.x))));
    const F2 ki = vmul(w, vfma(q1, a.y, vfma(q2, b.y, vmul(q3, c.y))));
    a = {vfma(norm, a.x, vmul(q1, kr)), vfma(norm, a.y, vmul(q1, ki))};
    b = {vfma(norm, b.x, vmul(q2, kr)), vfma(norm, b.y, vmul(q2, ki))};
    c = {vfma(norm, c.x, vmul(q3, kr)), vfma(norm, c.y, vmul(q3, ki))};
    if (q.x == 0.0f) {  // q = 0, the first column only
        auto clear = [](F2 &v) { v = pack2(0.0f, unpack2(v).y); };
        clear(a.x);
        clear(a.y);
        clear(b.x);
        clear(b.y);
        clear(c.x);
        clear(c.y);
    }
}

// The last forward stage, the projector and the first inverse stage on the R places of one butterfly (block length
// R: no twiddles), for the three components of two columns at a time.
constexpr int kZPairs = 4;  // pairs of columns of a block
template <int R>
__device__ __forceinline__ void z_middle(const Grid &g, ulonglong2 *zs, int comp_stride, int b, int line, F2 q1, F2 q2,
                                         F2 inv_n) {
    Cx<F2> a[3][R];
    const int base = b * R;
    auto off = [&](int q) { return (R == 8 ? padded(base) + q : padded(base + q)) * kZPairs + line; };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int q = 0; q < R; ++q) a[c][q] = load_pair(zs + c * comp_stride + off(q));
        dft<R, false>(a[c]);
    }
    const float step = 6.28318530717959f / g.Lz;
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int k = __ldg(g.z.freq + base + q);
        project(a[0][q], a[1][q], a[2][q], q1, q2, splat<F2>((k <= g.nz / 2 ? k : k - g.nz) * step), inv_n);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        dft<R, true>(a[c]);
#pragma unroll
        for (int q = 0; q < R; ++q) store_pair(zs + c * comp_stride + off(q), a[c][q]);
    }
}

// grid (kx blocks, y places): the three components of 8 columns in shared memory, from and to the used planes.
// Bound by latency, not by a pipe or the memory (at 512^3: 42% of issue slots, 35% of the FP32 pipe, 50% of the shared
// memory's cycles): the shared memory holds two blocks, eight warps each, and every stage ends at a barrier.  What
// helped, 512^3 with 28% of the planes: lengths known at compile time 1300 -> 1033 us, packed columns and the next
// component's elements read ahead -> 851 (one scalar column a thread and twice the warps: 910).  Four columns a block,
// four blocks an SM: 1.3 times slower, for its 32-byte rows.
template <int N>
__global__ void __launch_bounds__(64 * kZPairs, 8 / kZPairs) z_kernel(Grid g) {
    extern __shared__ __align__(16) ulonglong2 zs[];
    constexpr int kL = kZPairs == 4 ? 2 : 1;
    const int n = N ? N : g.nz, last = g.z.ns - 1;
    const int cstride = padded(n) * kZPairs;  // per component
    unsigned char *used = reinterpret_cast<unsigned char *>(zs + 3 * cstride);
    for (int p = threadIdx.x; p < n; p += blockDim.x) used[p] = g.plane_used[p];
    __syncthreads();
    const size_t ss = static_cast<size_t>(g.ldx) * g.ny * g.nz, plane = static_cast<size_t>(g.ldx) * g.ny;
    float2 *col0 = g.spec + static_cast<size_t>(blockIdx.y) * g.ldx + static_cast<size_t>(blockIdx.x) * (2 * kZPairs);
    auto at = [&](int c, int line, int p) { return reinterpret_cast<float4 *>(col0 + c * ss + p * plane) + line; };
    auto from_used = [&](int c, int line, int p, int) { return used[p] ? load_columns(at(c, line, p)) : Cx<F2>{}; };
    auto to_used = [&](int c, int line, int p, int, Cx<F2> v) {
        if (used[p]) store_columns(at(c, line, p), v);
    };
    auto from_smem = [&](int c, int line, int, int pp) { return load_pair(zs + c * cstride + pp * kZPairs + line); };
    auto to_smem = [&](int c, int line, int, int pp, Cx<F2> v) { store_pair(zs + c * cstride + pp * kZPairs + line, v); };
    stage<BlockTeam, N, 0, false, F2, kL, 3>(g.z, 0, n, from_used, to_smem);
    __syncthreads();
    middle_forward<BlockTeam, N, 1, F2, kL, 3>(g.z, from_smem, to_smem);
    {
        const int ky = __ldg(g.y.freq + blockIdx.y);
        const F2 q2 = splat<F2>((ky <= g.ny / 2 ? ky : ky - g.ny) * (6.28318530717959f / g.Ly));
        const F2 inv_n = splat<F2>(1.0f / (static_cast<float>(g.nx) * g.ny * g.nz));
        const int R = N ? radix_of(len_at(N, last_stage<N>())) : g.z.radix[last];
        for (int it = threadIdx.x; it < (n / R) * kZPairs; it += blockDim.x) {
            const int line = it & (kZPairs - 1), b = it / kZPairs;
            const int kx = blockIdx.x * 2 * kZPairs + 2 * line;
            const F2 q1 = pack2(kx * (6.28318530717959f / g.Lx), (kx + 1) * (6.28318530717959f / g.Lx));
            if constexpr (N > 0) {
                z_middle<radix_of(len_at(N, last_stage<N>()))>(g, zs, cstride, b, line, q1, q2, inv_n);
            } else {
                switch (R) {
                    case 8: z_middle<8>(g, zs, cstride, b, line, q1, q2, inv_n); break;
                    case 5: z_middle<5>(g, zs, cstride, b, line, q1, q2, inv_n); break;
                    case 4: z_middle<4>(g, zs, cstride, b, line, q1, q2, inv_n); break;
                    case 3: z_middle<3>(g, zs, cstride, b, line, q1, q2, inv_n); break;
                    default: z_middle<2>(g, zs, cstride, b, line, q1, q2, inv_n); break;
                }
            }
        }
    }
    __syncthreads();
    middle_inverse<BlockTeam, N, last_stage<N>() - 1, F2, kL, 3>(g.z, from_smem, to_smem);
    stage<BlockTeam, N, 0, true, F2, kL, 3>(g.z, 0, n, from_smem, to_used);
}

// ---------------------------------------------------------------- host side
// Kernels of one axis: lengths that are powers of two from 128 to 1024 (64 to 512 along x, half the row) have their
// own instantiation, the others share the runtime one.
using Kernel = void (*)(Grid);
inline Kernel pick_x(int n, bool inv) {
    switch (n) {
        case 64: return inv ? x_inverse_kernel<64> : x_forward_kernel<64>;
        case 128: return inv ? x_inverse_kernel<128> : x_forward_kernel<128>;
        case 256: return inv ? x_inverse_kernel<256> : x_forward_kernel<256>;
        case 512: return inv ? x_inverse_kernel<512> : x_forward_kernel<512>;
        default: return inv ? x_inverse_kernel<0> : x_forward_kernel<0>;
    }
}
inline Kernel pick_y(int n, bool inv) {
    switch (n) {
        case 128: return inv ? y_kernel<true, 128> : y_kernel<false, 128>;
        case 256: return inv ? y_kernel<true, 256> : y_kernel<false, 256>;
        case 512: return inv ? y_kernel<true, 512> : y_kernel<false, 512>;
        case 1024: return inv ? y_kernel<true, 1024> : y_kernel<false, 1024>;
        default: return inv ? y_kernel<true, 0> : y_kernel<false, 0>;
    }
}
inline Kernel pick_z(int n) {
    switch (n) {
        case 128: return z_kernel<128>;
        case 256: return z_kernel<256>;
        case 512: return z_kernel<512>;
        case 1024: return z_kernel<1024>;
        default: return z_kernel<0>;
    }
}

// Frequency of each place after the forward stages.
inline std::vector<int> place_freq(int n, const std::vector<int> &r) {
    std::vector<int> f(n);
    for (int p = 0; p < n; ++p) {
        int k = 0, mul = 1, len = n, q = p;
        for (int radix : r) {
            len /= radix;
            k += mul * (q / len);
            q %= len;
            mul *= radix;
        }
        f[p] = k;
    }
    return f;
}

inline std::vector<float2> twiddles(int n, int count) {
    std::vector<float2> w(count);
    for (int k = 0; k < count; ++k) {
        const double a = -2.0 * 3.14159265358979323846 * k / n;
        w[k] = make_float2(static_cast<float>(std::cos(a)), static_cast<float>(std::sin(a)));
    }
    return w;
}

inline int x_fixed(int mx) { return mx == 64 || mx == 128 || mx == 256 || mx == 512 ? mx : 0; }  // as pick_x
inline size_t x_smem(const Grid &g) { return sizeof(float2) * (padded(g.mx) + 1) * (kRowWarps << x_lines(x_fixed(g.mx))); }
inline size_t y_smem(const Grid &g) { return sizeof(float2) * kCols * padded(g.ny) + (g.ny + 15) / 16 * 16; }
inline size_t z_smem(const Grid &g) { return sizeof(ulonglong2) * kZPairs * 3 * padded(g.nz) + (g.nz + 15) / 16 * 16; }

}  // namespace fftk
}  // namespace cufil
