// flow.cu -- cf_flow: flow velocities at field points from saved segment and
// blob forces, the reference's flow-field post-processor
// (src/flow_field/flow_field_evaluator.cu:13-217, flow_velocities; host side
// :222-557).  Per flow point i:
//   v_i = 1/(8 pi mu) * ( sum over segments j of  S(x_i - x_j) f_j
//                           [+ Blake image terms of a wall at z = 0 when the data has no blobs]
//                           + rotlet of the segment torque
//                           [- S(x_i - X_body(j)) f_j with remove_net_force]
//                       + sum over blobs k of  S(x_i - x_k) f_k  [- S(x_i - X_body(k)) f_k] )
// with S(r) f = f/|r| + r (r.f)/|r|^3, the kernel's expressions term by term.
//
// The reference runs one thread per flow point over 64-wide shared-memory
// tiles.  Here: float4 source records packed once per call, 64-source tiles
// in shared memory, one or two flow points per thread, the source range
// split over gridDim.y so that a small set of flow points still fills every
// SM, FP32 sums of one tile under a TwoSum accumulation, and an FP64 reduction
// of the split partials in a fixed order (deterministic, no atomics).
#include "common.cuh"
#include "host_stage.cuh"

#include <algorithm>
#include <new>

struct cf_flow {
    cf_flow_config cfg{};
    int num_sms = CF_B200_SMS;
    cudaStream_t stream = nullptr;
    float4 *sx = nullptr, *sf = nullptr, *st = nullptr, *sb = nullptr;  // sources: centre, force, torque, body
    float4 *partial = nullptr;
    size_t partial_cap = 0;
    cufil::HostStage stage;  // host entry point: the call's arrays back to back, velocities last
    int max_bodies = 0;
};

namespace cufil {
namespace {

constexpr int kFlowThreads = 128;
constexpr int kFlowTile = 64;     // sources per shared-memory tile and per FP32 sum
constexpr int kFlowMaxTI = 2;     // flow points per thread: 1 or 2
constexpr int kFlowCtasPerSm = 8;

struct FlowParams {
    const float *xf;                  // [3 Nf]
    const float4 *sx, *sf, *st, *sb;  // sources
    float4 *partial;                  // [Nf][nsplit]
    int nf, ns, split, nsplit;
};

// 1/sqrt(x) by the hardware approximation (relative error up to 2^-22.9).  The sums are FP32 over 64 sources at a time,
// so their error stays below that of divisions and square roots under sums of 256: 4.9e-7 against 6.5e-7 (relative L2,
// 16,000 points above 5,120 segments, FP64 the measure).  Refining each root by a Newton step changed it by 5% and took
// 201 us for 176.
__device__ __forceinline__ float inv_sqrt(float x) {
    return rsqrtf(fminf(x, 3.0e38f));  // an overflowed distance contributes nothing, as 1 / infinity does
}

// One source at one flow point.  With d = x - x_s, p = dx fx + dy fy and R = (dx, dy, z + z_s), the terms are
// gathered by vector so that the pair takes about 55 multiply-adds and two reciprocal square roots:
//   direct   (f + ((d.f) d + t x d) / r^2) / r
//   image    -f / R - (R.f) R / R^3
//            + 2 z_s / R^5 (z (3 a R - R^2 f*) + R^2 (p e_z + f_z (dx, dy, 0))),   f* = (fx, fy, -fz), a = R.f*
// xs.w holds 2 z_s.  The direct terms form no cube of 1 / r: it leaves FP32 below r = 1.4e-13 (a flow point on a blob up
// to the rounding of cos(pi / 2)) and above 4e12, where the velocity itself does not.
template <bool SEG, bool WALL, bool NET>
__device__ __forceinline__ void flow_pair(float xi, float yi, float zi, float z3, const float4 &xs, const float4 &f,
                                          const float4 &t, const float4 &xb, float &vx, float &vy, float &vz) {
    const float dx = xi - xs.x, dy = yi - xs.y, dz = zi - xs.z;
    const float q2 = fmaf(dx, dx, dy * dy);
    const float p = fmaf(dx, f.x, dy * f.y);
    const float rm1 = inv_sqrt(fmaf(dz, dz, q2));
    const float rm2 = rm1 * rm1;
    const float df = fmaf(dz, f.z, p);
    if constexpr (SEG) {  // with the rotlet of the segment torque
        const float cx = fmaf(t.y, dz, fmaf(-t.z, dy, df * dx));
        const float cy = fmaf(t.z, dx, fmaf(-t.x, dz, df * dy));
        const float cz = fmaf(t.x, dy, fmaf(-t.y, dx, df * dz));
        vx = fmaf(rm1, fmaf(rm2, cx, f.x), vx);
        vy = fmaf(rm1, fmaf(rm2, cy, f.y), vy);
        vz = fmaf(rm1, fmaf(rm2, cz, f.z), vz);
    } else {
        const float g = rm2 * df;
        vx = fmaf(rm1, fmaf(g, dx, f.x), vx);
        vy = fmaf(rm1, fmaf(g, dy, f.y), vy);
        vz = fmaf(rm1, fmaf(g, dz, f.z), vz);
    }
    if constexpr (SEG && WALL) {  // Blake's image system (no blobs: half-space data)
        const float Rz = zi + xs.z;
        const float Rm1 = inv_sqrt(fmaf(Rz, Rz, q2));
        const float Rm2 = Rm1 * Rm1;
        const float Rm3 = Rm2 * Rm1;
        const float E = xs.w * Rm3;        // 2 z_s / R^3
        const float D = E * (z3 * Rm2);    // 6 z z_s / R^5
        const float zf = Rz * f.z;
        const float g = fmaf(D, p - zf, -Rm3 * (p + zf));
        const float h = fmaf(E, f.z, g);
        const float cp = fmaf(-E, zi, -Rm1), cm = fmaf(E, zi, -Rm1);
        vx = fmaf(h, dx, fmaf(cp, f.x, vx));
        vy = fmaf(h, dy, fmaf(cp, f.y, vy));
        vz = fmaf(E, p, fmaf(g, Rz, fmaf(cm, f.z, vz)));
    }
    if constexpr (NET) {  // minus a Stokeslet of the same force at the source's body
        const float ex = xi - xb.x, ey = yi - xb.y, ez = zi - xb.z;
        const float qm1 = inv_sqrt(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
        const float g = (qm1 * qm1) * fmaf(ex, f.x, fmaf(ey, f.y, ez * f.z));
        vx = fmaf(-qm1, fmaf(g, ex, f.x), vx);
        vy = fmaf(-qm1, fmaf(g, ey, f.y), vy);
        vz = fmaf(-qm1, fmaf(g, ez, f.z), vz);
    }
}

__device__ __forceinline__ void two_sum3(float *hi, float *lo, float ax, float ay, float az) {
    const float a[3] = {ax, ay, az};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float s = hi[c] + a[c];
        const float bp = s - hi[c];
        lo[c] += (hi[c] - (s - bp)) + (a[c] - bp);
        hi[c] = s;
    }
}

// grid (ceil(nf / (128 TI)), nsplit): block (x, y) sums sources [y*split, (y+1)*split)
// of its 128 TI flow points.  Sources [0, nseg_src) are segments, the rest blobs.
// Bound by the FP32 pipe: 16,000 points and 5,120 segments (8.2e7 pairs above the wall) take 168 us, about 53 TFLOP/s;
// term by term with divisions and square roots, in tiles of 256 at four blocks an SM, it was 425 us.  Four points a
// thread leave too few warps (201 us).
template <bool WALL, bool NET, int TI>
__global__ void __launch_bounds__(kFlowThreads, kFlowCtasPerSm) flow_tile_kernel(FlowParams p, int nseg_src) {
    constexpr int kTargets = kFlowThreads * TI;
    __shared__ float4 s_x[kFlowTile], s_f[kFlowTile], s_t[kFlowTile], s_b[kFlowTile];
    const int j0 = blockIdx.y * p.split;
    const int j1 = min(p.ns, j0 + p.split);
    float xi[TI], yi[TI], zi[TI], z3[TI];
    float hi[TI][3], lo[TI][3];
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        const int i = min(static_cast<int>(blockIdx.x * kTargets + k * kFlowThreads + threadIdx.x), p.nf - 1);
        xi[k] = p.xf[3 * i];
        yi[k] = p.xf[3 * i + 1];
        zi[k] = p.xf[3 * i + 2];
        z3[k] = 3.0f * zi[k];
#pragma unroll
        for (int c = 0; c < 3; ++c) hi[k][c] = lo[k][c] = 0.0f;
    }
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t0 = j0; t0 < j1; t0 += kFlowTile) {
        const int nt = min(kFlowTile, j1 - t0);
        __syncthreads();
        if (threadIdx.x < kFlowTile) {
            const int q = threadIdx.x;
            if (q < nt) {
                float4 x = p.sx[t0 + q];
                x.w = 2.0f * x.z;
                s_x[q] = x;
                s_f[q] = p.sf[t0 + q];
            }
        } else {
            const int q = threadIdx.x - kFlowTile;
            if (q < nt) {
                s_t[q] = (t0 + q < nseg_src) ? p.st[t0 + q] : zero4;
                if (NET) s_b[q] = p.sb[t0 + q];
            }
        }
        __syncthreads();
        // Segments and blobs of this tile: two branch-free loops.
        const int nsg = max(0, min(nt, nseg_src - t0));
        float vx[TI], vy[TI], vz[TI];
#pragma unroll
        for (int k = 0; k < TI; ++k) vx[k] = vy[k] = vz[k] = 0.0f;
#pragma unroll 2
        for (int q = 0; q < nsg; ++q) {
            const float4 xs = s_x[q], f = s_f[q], tq = s_t[q], xb = NET ? s_b[q] : zero4;
#pragma unroll
            for (int k = 0; k < TI; ++k)
                flow_pair<true, WALL, NET>(xi[k], yi[k], zi[k], z3[k], xs, f, tq, xb, vx[k], vy[k], vz[k]);
        }
#pragma unroll 2
        for (int q = nsg; q < nt; ++q) {
            const float4 xs = s_x[q], f = s_f[q], xb = NET ? s_b[q] : zero4;
#pragma unroll
            for (int k = 0; k < TI; ++k)
                flow_pair<false, false, NET>(xi[k], yi[k], zi[k], z3[k], xs, f, zero4, xb, vx[k], vy[k], vz[k]);
        }
#pragma unroll
        for (int k = 0; k < TI; ++k) two_sum3(hi[k], lo[k], vx[k], vy[k], vz[k]);
    }
#pragma unroll
    for (int k = 0; k < TI; ++k) {
        const int i = static_cast<int>(blockIdx.x * kTargets + k * kFlowThreads + threadIdx.x);
        if (i < p.nf)
            p.partial[static_cast<size_t>(i) * p.nsplit + blockIdx.y] =
                make_float4(hi[k][0] + lo[k][0], hi[k][1] + lo[k][1], hi[k][2] + lo[k][2], 0.0f);
    }
}

// One warp per flow point: FP64 sum of its partials in a fixed order, times 1/(8 pi mu).
__global__ void flow_reduce_kernel(const float4 *__restrict__ partial, int nf, int nsplit, double prefac,
                                   float *__restrict__ v) {
    const int lane = threadIdx.x & 31;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= nf) return;
    double a[3] = {0.0, 0.0, 0.0};
    for (int s = lane; s < nsplit; s += 32) {
        const float4 q = partial[static_cast<size_t>(i) * nsplit + s];
        a[0] += q.x;
        a[1] += q.y;
        a[2] += q.z;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[c] += __shfl_down_sync(0xffffffffu, a[c], o);
    if (lane == 0)
        for (int c = 0; c < 3; ++c) v[3 * i + c] = static_cast<float>(prefac * a[c]);
}

// Source records: segments [0, ns) from x [3ns] and f [6ns] (force, torque),
// then blobs [ns, ns + nb) from x [3nb] and f [3nb]; with bodies, the position
// of each source's body (segment j: body j / ns_per_body; blob k: k / nb_per_body).
__global__ void flow_pack_kernel(const float *xs, const float *fs, int ns, int ns_pb, const float *xb,
                                 const float *fb, int nb, int nb_pb, const float *xbod, float4 *sx, float4 *sf,
                                 float4 *st, float4 *sbod) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= ns + nb) return;
    int body = 0;
    if (j < ns) {
        sx[j] = make_float4(xs[3 * j], xs[3 * j + 1], xs[3 * j + 2], 0.0f);
        sf[j] = make_float4(fs[6 * j], fs[6 * j + 1], fs[6 * j + 2], 0.0f);
        st[j] = make_float4(fs[6 * j + 3], fs[6 * j + 4], fs[6 * j + 5], 0.0f);
        body = ns_pb > 0 ? j / ns_pb : 0;
    } else {
        const int k = j - ns;
        sx[j] = make_float4(xb[3 * k], xb[3 * k + 1], xb[3 * k + 2], 0.0f);
        sf[j] = make_float4(fb[3 * k], fb[3 * k + 1], fb[3 * k + 2], 0.0f);
        body = nb_pb > 0 ? k / nb_pb : 0;
    }
    if (xbod) sbod[j] = make_float4(xbod[3 * body], xbod[3 * body + 1], xbod[3 * body + 2], 0.0f);
}

struct FlowPlan {
    int ti, tiles, nsplit, split;
};

// Flow points per thread and source splits of nf points and nsrc sources: the choice with the least estimated
// time, waves x (per-block work), where a block's work is its sources times its points per thread plus a fixed
// cost (staging and epilogue) worth about 24 single-point sources.  More points per thread read each staged
// source less often (a source read from shared memory costs about 0.4 of a pair); more splits fill the SMs when
// the points are few.  The partials (nf x nsplit) stay within `cap`, the handle's buffer.
FlowPlan flow_plan(int nf, int nsrc, int num_sms, size_t cap) {
    FlowPlan best{};
    double best_cost = 1e300;
    const int max_tiles = std::max(1, (nsrc + kFlowTile - 1) / kFlowTile);
    for (int ti = 1; ti <= kFlowMaxTI; ti *= 2) {
        const int per = kFlowThreads * ti;
        const int tiles = std::max(1, (nf + per - 1) / per);
        const long long slots = static_cast<long long>(num_sms) * kFlowCtasPerSm;
        int last = 0;
        for (int cand = 1; cand <= max_tiles && cand <= 1024; ++cand) {
            const int split = kFlowTile * ((max_tiles + cand - 1) / cand);
            const int nsplit = (nsrc + split - 1) / split;
            if (nsplit == last) continue;
            last = nsplit;
            if (nsplit > 1 && static_cast<size_t>(nf) * nsplit > cap) break;
            const long long waves = (static_cast<long long>(tiles) * nsplit + slots - 1) / slots;
            const double cost = static_cast<double>(waves) * (split * (ti + 0.4) + 24.0);
            if (cost < best_cost * (1.0 - 1e-9)) {
                best_cost = cost;
                best = FlowPlan{ti, tiles, nsplit, split};
            }
        }
    }
    return best;
}

template <int TI>
void launch_flow_tiles(bool wall, bool net, dim3 grid, cudaStream_t st, const FlowParams &p, int ns) {
    if (wall && net) flow_tile_kernel<true, true, TI><<<grid, kFlowThreads, 0, st>>>(p, ns);
    else if (wall) flow_tile_kernel<true, false, TI><<<grid, kFlowThreads, 0, st>>>(p, ns);
    else if (net) flow_tile_kernel<false, true, TI><<<grid, kFlowThreads, 0, st>>>(p, ns);
    else flow_tile_kernel<false, false, TI><<<grid, kFlowThreads, 0, st>>>(p, ns);
}

template <typename T>
int falloc(T **p, size_t n) {
    *p = nullptr;
    CF_CUDA(cudaMalloc(reinterpret_cast<void **>(p), std::max<size_t>(n, 1) * sizeof(T)));
    return CF_OK;
}

int flow_run(cf_flow *h, const float *xf, int nf, const float *xs, const float *fs, int ns, int ns_pb,
             const float *xb, const float *fb, int nb, int nb_pb, const float *xbod, float *v, cudaStream_t st) {
    const int nsrc = ns + nb;
    if (nf == 0) return CF_OK;
    if (nsrc == 0) {
        CF_CUDA(cudaMemsetAsync(v, 0, sizeof(float) * 3 * nf, st));
        return CF_OK;
    }
    const bool net = h->cfg.remove_net_force != 0;
    flow_pack_kernel<<<(nsrc + 255) / 256, 256, 0, st>>>(xs, fs, ns, ns_pb, xb, fb, nb, nb_pb, net ? xbod : nullptr,
                                                         h->sx, h->sf, h->st, h->sb);
    CF_CHECK_LAUNCH("flow_pack_kernel");
    const FlowPlan pl = flow_plan(nf, nsrc, h->num_sms, h->partial_cap);
    CF_REQUIRE(static_cast<size_t>(nf) * pl.nsplit <= h->partial_cap, "cf_flow: scratch too small");
    FlowParams p{xf, h->sx, h->sf, h->st, h->sb, h->partial, nf, nsrc, pl.split, pl.nsplit};
    const dim3 grid(pl.tiles, pl.nsplit);
    const bool wall = nb_pb == 0;  // no blobs: half-space data (flow_field_evaluator.cu:75-78)
    if (pl.ti == 2) launch_flow_tiles<2>(wall, net, grid, st, p, ns);
    else launch_flow_tiles<1>(wall, net, grid, st, p, ns);
    CF_CHECK_LAUNCH("flow_tile_kernel");
    const double prefac = 1.0 / (8.0 * 3.14159265358979323846 * h->cfg.mu);
    flow_reduce_kernel<<<(nf + 7) / 8, 256, 0, st>>>(h->partial, nf, pl.nsplit, prefac, v);
    CF_CHECK_LAUNCH("flow_reduce_kernel");
    return CF_OK;
}

int flow_check(cf_flow *h, int nf, int ns, int ns_pb, int nb, int nb_pb, const char *who) {
    CF_REQUIRE(h, "%s: null handle", who);
    CF_REQUIRE(nf >= 0 && nf <= h->cfg.max_flow, "%s: n_flow %d outside [0, %d]", who, nf, h->cfg.max_flow);
    CF_REQUIRE(ns >= 0 && ns <= h->cfg.max_seg, "%s: n_seg %d outside [0, %d]", who, ns, h->cfg.max_seg);
    CF_REQUIRE(nb >= 0 && nb <= h->cfg.max_blob, "%s: n_blob %d outside [0, %d]", who, nb, h->cfg.max_blob);
    CF_REQUIRE(ns == 0 || (ns_pb >= 1 && ns % ns_pb == 0), "%s: n_seg must be a multiple of n_seg_per_body", who);
    CF_REQUIRE(nb == 0 || (nb_pb >= 1 && nb % nb_pb == 0), "%s: n_blob must be a multiple of n_blob_per_body", who);
    const int bodies = std::max(ns ? ns / ns_pb : 0, nb ? nb / nb_pb : 0);
    CF_REQUIRE(bodies <= h->max_bodies, "%s: %d bodies exceed max_bodies %d", who, bodies, h->max_bodies);
    return CF_OK;
}

}  // namespace
}  // namespace cufil

using namespace cufil;

extern "C" int cf_flow_destroy(cf_flow *h) {
    if (!h) return CF_OK;
    cudaSetDevice(h->cfg.device);
    for (void *p : {(void *)h->sx, (void *)h->sf, (void *)h->st, (void *)h->sb, (void *)h->partial})
        if (p) cudaFree(p);
    h->stage.release();
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return CF_OK;
}

extern "C" int cf_flow_create(const cf_flow_config *cfg, cf_flow **out) {
    clear_error();
    CF_REQUIRE(cfg && out, "cf_flow_create: null argument");
    *out = nullptr;
    CF_REQUIRE(cfg->max_flow >= 1 && cfg->max_seg >= 0 && cfg->max_blob >= 0 && cfg->max_bodies >= 1,
               "cf_flow_create: bad sizes (max_flow %d, max_seg %d, max_blob %d, max_bodies %d)", cfg->max_flow,
               cfg->max_seg, cfg->max_blob, cfg->max_bodies);
    CF_REQUIRE(cfg->mu > 0.0, "cf_flow_create: mu must be positive");
    CF_CUDA(cudaSetDevice(cfg->device));
    cf_flow *h = new (std::nothrow) cf_flow();
    if (!h) return set_error(CF_ENOMEM, "cf_flow_create: host allocation failed");
    h->cfg = *cfg;
    h->max_bodies = cfg->max_bodies;
    int rc = CF_OK;
    do {
        if ((rc = cuda_status(cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, cfg->device),
                              "cudaDeviceGetAttribute", __FILE__, __LINE__)))
            break;
        if ((rc = cuda_status(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "cudaStreamCreate",
                              __FILE__, __LINE__)))
            break;
        const size_t nsrc = static_cast<size_t>(cfg->max_seg) + cfg->max_blob;
        // one partial per point and split; flow_plan takes no more splits than fit
        h->partial_cap = static_cast<size_t>(2 * kFlowCtasPerSm * h->num_sms + 1) * kFlowThreads +
                         2 * static_cast<size_t>(cfg->max_flow);
        if ((rc = falloc(&h->sx, nsrc)) || (rc = falloc(&h->sf, nsrc)) || (rc = falloc(&h->st, nsrc)) ||
            (rc = falloc(&h->sb, nsrc)) || (rc = falloc(&h->partial, h->partial_cap)) ||
            (rc = cuda_status(h->stage.alloc(sizeof(float) * (6 * static_cast<size_t>(cfg->max_flow) +
                                                              9 * static_cast<size_t>(cfg->max_seg) +
                                                              6 * static_cast<size_t>(cfg->max_blob) +
                                                              3 * static_cast<size_t>(cfg->max_bodies))),
                              "staging buffer", __FILE__, __LINE__)))
            break;
    } while (0);
    if (rc != CF_OK) {
        cf_flow_destroy(h);
        return rc;
    }
    *out = h;
    return CF_OK;
}

extern "C" int cf_flow_velocities_device(cf_flow *h, const float *d_x_flow, int n_flow, const float *d_x_segs,
                                         const float *d_f_segs, int n_seg, int n_seg_per_body, const float *d_x_blobs,
                                         const float *d_f_blobs, int n_blob, int n_blob_per_body,
                                         const float *d_x_bodies, float *d_v_flow, void *stream) {
    clear_error();
    CF_TRY(flow_check(h, n_flow, n_seg, n_seg_per_body, n_blob, n_blob_per_body, "cf_flow_velocities_device"));
    CF_REQUIRE(!n_flow || (d_x_flow && d_v_flow), "cf_flow_velocities_device: missing flow-point buffers");
    CF_REQUIRE(!n_seg || (d_x_segs && d_f_segs), "cf_flow_velocities_device: missing segment buffers");
    CF_REQUIRE(!n_blob || (d_x_blobs && d_f_blobs), "cf_flow_velocities_device: missing blob buffers");
    CF_REQUIRE(!h->cfg.remove_net_force || d_x_bodies, "cf_flow_velocities_device: remove_net_force needs bodies");
    CF_CUDA(cudaSetDevice(h->cfg.device));
    return flow_run(h, d_x_flow, n_flow, d_x_segs, d_f_segs, n_seg, n_seg_per_body, d_x_blobs, d_f_blobs, n_blob,
                    n_blob_per_body, d_x_bodies, d_v_flow, static_cast<cudaStream_t>(stream));
}

extern "C" int cf_flow_velocities(cf_flow *h, const float *x_flow, int n_flow, const float *x_segs,
                                  const float *f_segs, int n_seg, int n_seg_per_body, const float *x_blobs,
                                  const float *f_blobs, int n_blob, int n_blob_per_body, const float *x_bodies,
                                  float *v_flow) {
    clear_error();
    CF_TRY(flow_check(h, n_flow, n_seg, n_seg_per_body, n_blob, n_blob_per_body, "cf_flow_velocities"));
    CF_REQUIRE(!n_flow || (x_flow && v_flow), "cf_flow_velocities: missing flow-point arrays");
    CF_REQUIRE(!n_seg || (x_segs && f_segs), "cf_flow_velocities: missing segment arrays");
    CF_REQUIRE(!n_blob || (x_blobs && f_blobs), "cf_flow_velocities: missing blob arrays");
    CF_REQUIRE(!h->cfg.remove_net_force || x_bodies, "cf_flow_velocities: remove_net_force needs bodies");
    CF_CUDA(cudaSetDevice(h->cfg.device));
    cudaStream_t st = h->stream;
    const int bodies = std::max(n_seg ? n_seg / n_seg_per_body : 0, n_blob ? n_blob / n_blob_per_body : 0);
    const size_t nf3 = 3 * static_cast<size_t>(n_flow), ns3 = 3 * static_cast<size_t>(n_seg),
                 nb3 = 3 * static_cast<size_t>(n_blob), nd3 = x_bodies ? 3 * static_cast<size_t>(bodies) : 0;
    h->stage.open();
    size_t at = 0;  // bytes
    cudaError_t e = cudaSuccess;
    auto put = [&](const float *src, size_t count) {
        if (e == cudaSuccess) e = h->stage.put(at, src, count * sizeof(float), st);
        float *d = h->stage.at<float>(at);
        at += count * sizeof(float);
        return d;
    };
    const float *dxf = put(x_flow, nf3), *dxs = put(x_segs, ns3), *dfs = put(f_segs, 2 * ns3), *dxb = put(x_blobs, nb3),
                *dfb = put(f_blobs, nb3), *dxd = put(x_bodies, nd3);
    CF_CUDA(e);
    CF_CUDA(h->stage.up(at, st));
    CF_TRY(flow_run(h, dxf, n_flow, dxs, dfs, n_seg, n_seg_per_body, dxb, dfb, n_blob, n_blob_per_body,
                    x_bodies ? dxd : nullptr, h->stage.at<float>(at), st));
    CF_CUDA(h->stage.down(at, nf3 * sizeof(float), st));
    CF_CUDA(cudaStreamSynchronize(st));
    CF_CUDA(h->stage.take(v_flow, at, nf3 * sizeof(float), st));
    return CF_OK;
}
