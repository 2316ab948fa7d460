// swim_engine.cuh -- cf_swim: one free rigid body carrying prescribed cilia,
// the reference's swimmer path (PRESCRIBED_CILIA with a body whose motion is
// solved for: BODY_VELOCITY_TYPE 0, BODY_OR_SURFACE_TYPE 2).  Included by sim.cu,
// whose beat kinematics it shares.
//
// Per step (cilia_sim_main.cu:405-716 with swimmer::initial_guess, swimmer.cpp:433-466):
//   body frame      filament frames q_body * q_ref (the filaments' own quaternions follow
//                   the body's rotation increments, filament.cpp:653-666), bases and blob
//                   positions from the body-frame references (swimmer.cpp:440-458);
//   kinematics      the Fulford-Blake beat in each filament's frame (kinematics_kernel);
//   precon matrix   swimmer::make_precon_mat (swimmer.cpp:1175-1349), the 6x6 body Schur
//                   matrix and its inverse, in FP64;
//   RHS             -q_phase, -q_angle rows (mobility_solver.cpp:284-420), zero elsewhere;
//   solve           right-preconditioned GMRES on the saddle system
//                   [3N lambda | 3B blob forces | V, Omega | N_fil phase rates | N_fil angle rates]
//                   (mobility_solver.cpp:2187-2669) with
//                     A: system_matrix_mult_new's body branch (:1887-2105): unbounded RPY over
//                        segments and blobs together, minus K V for every particle, the body's
//                        force and torque balance rows, and the filament rate rows;
//                     P: apply_preconditioner_new's body branch (:1244-1475);
//   body update     x += dt V, q = lie_exp(dt Omega) q (cilia_sim_main.cu:700-716).
// Everything runs on the device; the host only enqueues.  A GMRES iteration is eight
// launches (classical Gram-Schmidt with one re-orthogonalisation); the block that
// finishes the last of them does the Givens step and decides whether the solve goes
// on, and the kernels of an iteration enqueued past that point return at once, so
// the host enqueues one iteration ahead instead of waiting for each.  The pair
// products are the FP32 symmetric warp-tile kernel (rpy_kernels.cu).  A step of 256
// filaments on 2,562 blobs takes 1.33 ms, of which the pair products are about 0.5;
// with the host waiting for each iteration's dot products, the frames and the 6 x 6
// body matrix formed on the host and 19 launches an iteration it took 2.60 ms.
#pragma once

namespace cufil {
namespace swim {
// State of one solve.
struct SwimCtl {
    int run;         // 1 while GMRES iterates
    int apply;       // what the solve does to sol: 0 nothing, 1 adds the correction, 2 replaces sol by it, 3 zeroes sol
    int status;      // CF_OK, CF_NOT_CONVERGED, CF_NONFINITE
    int iters, zero_guess, singular;
    double norm_rhs, relres, inv_scale;
};
// What the host reads back: two control records in turn, the body's velocity and the wait flag.
struct SwimReport {
    SwimCtl ctl[2];
    double bv[6];
    int err;
};
}  // namespace swim
}  // namespace cufil

struct cf_swim {
    cf_swim_config cfg{};
    int device = 0, num_sms = CF_B200_SMS;
    cudaStream_t stream = nullptr;
    int F = 0, nseg = 0, N = 0, B = 0, n = 0, o_blob = 0, o_body = 0, o_phase = 0, o_angle = 0, max_iter = 0;
    cufil::SimDev d{};  // kinematics state (phases, frames, positions, velocity directions)
    std::vector<double> qref;    // [F][4] filament frames in the body frame (scalar first)
    std::vector<double> fil_ref;  // [3F] filament bases in the body frame
    std::vector<double> blob_ref; // [3B] blobs in the body frame
    double bx[3] = {0, 0, 0}, bq[4] = {1, 0, 0, 0}, bv[6] = {0, 0, 0, 0, 0, 0};
    double *d_qref = nullptr, *d_fil_ref = nullptr, *d_blob_ref = nullptr;  // the same on the device
    double *Rfil = nullptr, *xb = nullptr, *body = nullptr, *aux = nullptr, *kinv = nullptr;
    float4 *x4all = nullptr, *f4all = nullptr, *scratch = nullptr;
    size_t scratch_cap = 0;
    int *err = nullptr;
    double *rhs = nullptr, *sol = nullptr, *w = nullptr, *z = nullptr, *t = nullptr, *Q = nullptr;
    double *h1 = nullptr, *h2 = nullptr, *H = nullptr, *cs = nullptr, *sn = nullptr, *beta = nullptr, *y = nullptr;
    double *part = nullptr;           // block partials of the sums that span blocks
    unsigned int *counter = nullptr;  // their arrival counter (zero between launches)
    cufil::swim::SwimCtl *ctl = nullptr;
    cufil::swim::SwimReport *h_rep = nullptr;  // control records and body velocity read back: page-locked, or own_rep
    cufil::swim::SwimReport own_rep{};         // in the first step, where each read back waits
    cufil::PinnedBuffer pinned;
    cudaEvent_t ev[2] = {};
    int last_iters = 0, last_status = CF_OK;
    double last_relres = 0.0;
    bool stepped = false;
    std::vector<void *> allocations;
};

namespace cufil {
namespace swim {

// ------------------------------------------------------------ quaternions
// FP64 quaternions (scalar first), as src/general/quaternion.cpp defines them.
struct Quat {
    double s, v[3];
};

__host__ __device__ inline Quat qmul(const Quat &a, const Quat &b) {  // operator*= (quaternion.cpp:104-118)
    Quat r;
    r.s = a.s * b.s - (a.v[0] * b.v[0] + a.v[1] * b.v[1] + a.v[2] * b.v[2]);
    r.v[0] = a.s * b.v[0] + b.s * a.v[0] + a.v[1] * b.v[2] - a.v[2] * b.v[1];
    r.v[1] = a.s * b.v[1] + b.s * a.v[1] + a.v[2] * b.v[0] - a.v[0] * b.v[2];
    r.v[2] = a.s * b.v[2] + b.s * a.v[2] + a.v[0] * b.v[1] - a.v[1] * b.v[0];
    return r;
}

void qnormalise(Quat &q) {  // normalise_in_place (:183-187)
    const double nrm = std::sqrt(q.s * q.s + q.v[0] * q.v[0] + q.v[1] * q.v[1] + q.v[2] * q.v[2]);
    q.s /= nrm;
    for (double &c : q.v) c /= nrm;
}

void qsqrt_ortho(Quat &q) {  // sqrt_in_place_ortho (:197-223), including its guard near -1
    if (q.s < -0.999999) {
        q.s = -0.9999999;
        q.s = std::sqrt(0.5 * (1.0 + q.s));
        const double temp = 2.0 * q.s;
        for (double &c : q.v) c /= temp;
        const double qn = std::sqrt(q.s * q.s + q.v[0] * q.v[0] + q.v[1] * q.v[1] + q.v[2] * q.v[2]);
        q.s *= qn;
        for (double &c : q.v) c /= qn;
    } else {
        q.s = std::sqrt(0.5 * (1.0 + q.s));
        const double temp = 2.0 * q.s;
        for (double &c : q.v) c /= temp;
    }
    qnormalise(q);
}

void qnormal(const Quat &q, double n[3]) {  // normal (:271-277)
    n[0] = 2.0 * (q.v[0] * q.v[1] - q.s * q.v[2]);
    n[1] = 1.0 - 2.0 * (q.v[0] * q.v[0] + q.v[2] * q.v[2]);
    n[2] = 2.0 * (q.v[1] * q.v[2] + q.s * q.v[0]);
}

__host__ __device__ inline void qrot(const Quat &q, double R[9]) {  // rot_mat (:305-345), row-major
    const double x = q.v[0], y = q.v[1], zc = q.v[2], s = q.s;
    R[0] = 1.0 - 2.0 * y * y - 2.0 * zc * zc;
    R[4] = 1.0 - 2.0 * x * x - 2.0 * zc * zc;
    R[8] = 1.0 - 2.0 * x * x - 2.0 * y * y;
    R[3] = 2.0 * x * y + 2.0 * s * zc;
    R[1] = 2.0 * x * y - 2.0 * s * zc;
    R[6] = 2.0 * x * zc - 2.0 * s * y;
    R[2] = 2.0 * x * zc + 2.0 * s * y;
    R[5] = 2.0 * y * zc - 2.0 * s * x;
    R[7] = 2.0 * y * zc + 2.0 * s * x;
}

Quat qlie_exp(const double u[3]) {  // lie_exp (:500-523)
    const double th = std::sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    if (th < 1e-6) return Quat{1.0, {0.0, 0.0, 0.0}};
    const double cs = std::cos(0.5 * th), sn = std::sin(0.5 * th) / th;
    return Quat{cs, {sn * u[0], sn * u[1], sn * u[2]}};
}

// The frame of a filament whose base direction is dir in the body frame
// (filament.cpp:224-236, 368-400, 422-430 with TILT_ANGLE = 0): the rotation
// taking the reference x axis to dir, followed by the one that aligns the
// reference y axis with the polar direction (the projection of -e_z).
Quat filament_frame(const double *dir_in) {
    const double dn = std::sqrt(dir_in[0] * dir_in[0] + dir_in[1] * dir_in[1] + dir_in[2] * dir_in[2]);
    const double dir[3] = {dir_in[0] / dn, dir_in[1] / dn, dir_in[2] / dn};
    Quat qtemp{dir[0], {0.0, -dir[2], dir[1]}};
    qsqrt_ortho(qtemp);
    double bn[3];
    qnormal(qtemp, bn);
    double pol[3] = {0.0, 0.0, -1.0};
    const double dp = dir[0] * pol[0] + dir[1] * pol[1] + dir[2] * pol[2];
    for (int c = 0; c < 3; ++c) pol[c] -= dp * dir[c];
    const double np = std::sqrt(pol[0] * pol[0] + pol[1] * pol[1] + pol[2] * pol[2]);
    Quat q2{1.0, {0.0, 0.0, 0.0}};
    if (np > 0.0) {
        for (double &c : pol) c /= np;
        q2.s = pol[0] * bn[0] + pol[1] * bn[1] + pol[2] * bn[2];
        q2.v[0] = bn[1] * pol[2] - bn[2] * pol[1];
        q2.v[1] = bn[2] * pol[0] - bn[0] * pol[2];
        q2.v[2] = bn[0] * pol[1] - bn[1] * pol[0];
        qsqrt_ortho(q2);
    }
    return qmul(q2, qtemp);
}

// 6x6 inverse by Gauss-Jordan with partial pivoting (row-major, FP64); false if singular.
__device__ inline bool invert6(double *A) {
    double M[6][12];
    for (int i = 0; i < 6; ++i)
        for (int j = 0; j < 12; ++j) M[i][j] = j < 6 ? A[6 * i + j] : (j - 6 == i ? 1.0 : 0.0);
    for (int c = 0; c < 6; ++c) {
        int p = c;
        for (int r = c + 1; r < 6; ++r)
            if (fabs(M[r][c]) > fabs(M[p][c])) p = r;
        if (M[p][c] == 0.0 || !isfinite(M[p][c])) return false;
        if (p != c)
            for (int j = 0; j < 12; ++j) {
                const double t = M[p][j];
                M[p][j] = M[c][j];
                M[c][j] = t;
            }
        const double inv = 1.0 / M[c][c];
        for (int j = 0; j < 12; ++j) M[c][j] *= inv;
        for (int r = 0; r < 6; ++r)
            if (r != c) {
                const double f = M[r][c];
                if (f != 0.0)
                    for (int j = 0; j < 12; ++j) M[r][j] -= f * M[c][j];
            }
    }
    for (int i = 0; i < 6; ++i)
        for (int j = 0; j < 6; ++j) A[6 * i + j] = M[i][j + 6];
    return true;
}

// ------------------------------------------------------------ device side
constexpr double kSwimMobInv = 6.0 * 3.14159265358979323846;  // 6 pi mu a, mu = a = 1 (segments and blobs)

struct SwimParams {
    int F, nseg, N, B, o_blob, o_body, o_phase, o_angle;
    const double *xd, *kp, *ka, *gram;  // segment positions and velocity directions, per-filament (c11, c22, c12)
    const double *xb;                   // blob positions [3B]
    const double *body;                 // body centre [3]
    const double *aux;                  // per filament: v_phi, u_phi, v_theta, u_theta (12)
    const double *kinv;                 // inverse of the 6x6 body Schur matrix (row-major)
};

__device__ __forceinline__ void swim_diff(const SwimParams &p, int i, double r[3]) {
    const double *x = i < p.N ? p.xd + 3 * i : p.xb + 3 * (i - p.N);
    for (int c = 0; c < 3; ++c) r[c] = x[c] - p.body[c];
}

__device__ __forceinline__ long long swim_row(const SwimParams &p, int i) {
    return i < p.N ? 3LL * i : p.o_blob + 3LL * (i - p.N);
}

// Sums of NV values over a block of kSwT threads: value c's total in thread c (fixed order).
constexpr int kSwT = 128;
template <int NV>
__device__ __forceinline__ double block_sums(const double (&v)[NV], double (*sm)[NV]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        const double s = warp_sum(v[c]);
        if (lane == 0) sm[w][c] = s;
    }
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < NV)
        for (int q = 0; q < kSwT / 32; ++q) t += sm[q][threadIdx.x];
    return t;
}

// The particles of a block of the per-filament kernels: block m < F holds filament m, the blocks after them kSwT
// blobs each.
__device__ __forceinline__ void swim_range(const SwimParams &p, int blk, int &lo, int &hi) {
    if (blk < p.F) {
        lo = blk * p.nseg;
        hi = lo + p.nseg;
    } else {
        lo = p.N + (blk - p.F) * kSwT;
        hi = min(p.N + p.B, lo + kSwT);
    }
}

// Totals over the blocks of NV values each left in part[block][NV], by the block that arrives last: value c by warp
// c % (kSwT / 32), in a fixed order, into out[c] (shared).
template <int NV>
__device__ __forceinline__ bool swim_totals(double *part, unsigned int *counter, int *flag, double *out) {
    if (!arrive_last(counter, gridDim.x, flag)) return false;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c = w; c < NV; c += kSwT / 32) {
        double t = 0.0;
        for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) t += __ldcg(part + static_cast<size_t>(b) * NV + c);
        t = warp_sum(t);
        if (lane == 0) out[c] = t;
    }
    if (threadIdx.x == 0) *counter = 0u;
    __syncthreads();
    return true;
}

// Body frame of the current body state (swimmer::initial_guess, swimmer.cpp:433-466; the filaments' quaternions follow
// the body's): filament frames and bases, blob positions, body centre.
struct BodyState {
    double x[3], q[4];
};
__global__ void swim_frames_kernel(BodyState b, int F, int B, const double *qref, const double *fil_ref,
                                   const double *blob_ref, double *R, double *base, double *xb, double *body) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const Quat qb{b.q[0], {b.q[1], b.q[2], b.q[3]}};
    double Rb[9];
    qrot(qb, Rb);
    if (i < 3) body[i] = b.x[i];
    if (i < F) {
        const Quat qr{qref[4 * i], {qref[4 * i + 1], qref[4 * i + 2], qref[4 * i + 3]}};
        qrot(qmul(qb, qr), R + 9 * static_cast<size_t>(i));
    }
    const double *ref = i < F ? fil_ref + 3 * static_cast<size_t>(i) : blob_ref + 3 * static_cast<size_t>(i - F);
    double *out = i < F ? base + 3 * static_cast<size_t>(i) : xb + 3 * static_cast<size_t>(i - F);
    if (i < F + B)
        for (int c = 0; c < 3; ++c) out[c] = b.x[c] + Rb[3 * c] * ref[0] + Rb[3 * c + 1] * ref[1] + Rb[3 * c + 2] * ref[2];
}

// Start of a step after the kinematics: pair-kernel positions, the driving rows -q_phase, -(q_angle - spring term)
// (the other rows of the right-hand side stay zero), and swimmer::make_precon_mat (swimmer.cpp:1175-1349, dynamic
// phase and angle): the per-filament sums v_phi, u_phi, v_theta, u_theta and Gram entries that the preconditioner
// reuses, and the inverse of the 6x6 body Schur matrix
//   6 pi [ n I      S(d)^T ]  -  6 pi sum_m [v u]^T C_m^-1 [v u],   S(d) w = w x d,
//        [ S(d)  -S(d)S(d) ]
// whose particle sums are the first and second moments of d = x - x_body.  kinv is left untouched and ctl->singular set
// when the matrix cannot be inverted.
constexpr int kPreMoments = 9, kPreValues = kPreMoments + 21;  // sums of d and d d^T; lower triangle of the C terms
__global__ void __launch_bounds__(kSwT) swim_begin_kernel(SwimParams p, SimDev d, float4 *x4all, double *rhs, double *aux,
                                                          double *gram, double *kinv, double *part,
                                                          unsigned int *counter, SwimCtl *ctl) {
    __shared__ double sm[kSwT / 32][15];
    __shared__ double mom[kPreMoments + 15], tot[kPreValues];
    __shared__ int flag;
    int lo, hi;
    swim_range(p, blockIdx.x, lo, hi);
    const bool fil = static_cast<int>(blockIdx.x) < p.F;
    double m9[kPreMoments] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double f15[15] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // vp, up, vt, ut, c11, c22, c12
    for (int i = lo + threadIdx.x; i < hi; i += kSwT) {
        double r[3];
        swim_diff(p, i, r);
        for (int c = 0; c < 3; ++c) m9[c] += r[c];
        m9[3] += r[0] * r[0];
        m9[4] += r[1] * r[1];
        m9[5] += r[2] * r[2];
        m9[6] += r[0] * r[1];
        m9[7] += r[0] * r[2];
        m9[8] += r[1] * r[2];
        if (fil) {
            x4all[i] = d.x4[i];
            const double *a = p.kp + 3 * static_cast<size_t>(i), *b = p.ka + 3 * static_cast<size_t>(i);
            for (int c = 0; c < 3; ++c) {
                f15[c] += a[c];
                f15[6 + c] += b[c];
            }
            f15[3] += r[1] * a[2] - r[2] * a[1];
            f15[4] += r[2] * a[0] - r[0] * a[2];
            f15[5] += r[0] * a[1] - r[1] * a[0];
            f15[9] += r[1] * b[2] - r[2] * b[1];
            f15[10] += r[2] * b[0] - r[0] * b[2];
            f15[11] += r[0] * b[1] - r[1] * b[0];
            f15[12] += a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
            f15[13] += b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
            f15[14] += a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
        } else {
            const double *x = p.xb + 3 * static_cast<size_t>(i - p.N);
            x4all[i] = make_float4(static_cast<float>(x[0]), static_cast<float>(x[1]), static_cast<float>(x[2]), 0.0f);
        }
    }
    const double t15 = block_sums<15>(f15, sm);
    if (threadIdx.x < 15) mom[kPreMoments + threadIdx.x] = t15;
    __syncthreads();
    {
        double (*sm9)[kPreMoments] = reinterpret_cast<double (*)[kPreMoments]>(sm);
        const double t9 = block_sums<kPreMoments>(m9, sm9);
        if (threadIdx.x < kPreMoments) mom[threadIdx.x] = t9;
    }
    __syncthreads();
    double *mine = part + static_cast<size_t>(blockIdx.x) * kPreValues;
    if (threadIdx.x < kPreMoments) mine[threadIdx.x] = mom[threadIdx.x];
    if (threadIdx.x < 21) {  // entry (i, j), j <= i, of this filament's C term
        int i = 0, j = threadIdx.x;
        while (j > i) j -= ++i;
        double v = 0.0;
        if (fil) {
            const double *f = mom + kPreMoments;
            const double c11 = f[12], c22 = f[13], c12 = f[14], det = c11 * c22 - c12 * c12;
            const double i11 = c22 / det, i22 = c11 / det, i12 = -c12 / det;
            const double pi_ = f[i], pj = f[j], ti = f[6 + i], tj = f[6 + j];  // (v, u) of phi, then of theta
            v = pi_ * pj * i11 + pi_ * tj * i12 + ti * pj * i12 + ti * tj * i22;
        }
        mine[kPreMoments + threadIdx.x] = v;
    }
    if (fil) {
        const int m = blockIdx.x;
        if (threadIdx.x < 12) aux[12 * static_cast<size_t>(m) + threadIdx.x] = mom[kPreMoments + threadIdx.x];
        if (threadIdx.x < 3) gram[3 * static_cast<size_t>(m) + threadIdx.x] = mom[kPreMoments + 12 + threadIdx.x];
        if (threadIdx.x == 0) {
            const double w0 = d.omega0[m] * 0.5 / 3.14159265358979323846;
            double q_angle = cyclic_spline(d.phase[m], d.angle_refs, d.n_angle_refs) * w0;
            q_angle -= d.spring * d.omega0[m] * d.L * d.L * d.L * d.angle[m];
            rhs[p.o_phase + m] = -cyclic_spline(d.phase[m], d.phase_refs, d.n_phase_refs) * w0;
            rhs[p.o_angle + m] = -q_angle;
        }
    }
    if (!swim_totals<kPreValues>(part, counter, &flag, tot) || threadIdx.x != 0) return;
    double K[36];
    for (double &v : K) v = 0.0;
    const double s[3] = {tot[0], tot[1], tot[2]};
    const double mm[3][3] = {{tot[3], tot[6], tot[7]}, {tot[6], tot[4], tot[8]}, {tot[7], tot[8], tot[5]}};
    const double tr = tot[3] + tot[4] + tot[5];
    const double rc[3][3] = {{0.0, s[2], -s[1]}, {-s[2], 0.0, s[0]}, {s[1], -s[0], 0.0}};  // S(sum of d)
    for (int i = 0; i < 3; ++i) {
        K[7 * i] = static_cast<double>(p.N + p.B);
        for (int j = 0; j < 3; ++j) {
            K[6 * i + 3 + j] = rc[i][j];
            K[6 * (3 + i) + j] = -rc[i][j];
            K[6 * (3 + i) + 3 + j] = (i == j ? tr : 0.0) - mm[i][j];
        }
    }
    for (int i = 0, e = kPreMoments; i < 6; ++i)
        for (int j = 0; j <= i; ++j, ++e) {
            K[6 * i + j] -= tot[e];
            if (i != j) K[6 * j + i] -= tot[e];
        }
    for (double &v : K) v *= kSwimMobInv;
    if (invert6(K)) {
        for (int q = 0; q < 36; ++q) kinv[q] = K[q];
        ctl->singular = 0;
    } else {
        ctl->singular = 1;
    }
}

// Rows of A v that need v alone, and the pair kernel's forces: f4 = float(v), out[phase, angle] = -K^T lambda_m per
// filament, out[body] = minus the total force and torque (about the body centre) of every particle.
__device__ __forceinline__ void swim_tail_add(const SwimParams &p, int i, const double *f, double (&acc)[8]) {
    double r[3];
    swim_diff(p, i, r);
    acc[0] += f[0];
    acc[1] += f[1];
    acc[2] += f[2];
    acc[3] += r[1] * f[2] - r[2] * f[1];
    acc[4] += r[2] * f[0] - r[0] * f[2];
    acc[5] += r[0] * f[1] - r[1] * f[0];
    if (i < p.N)
        for (int c = 0; c < 3; ++c) {
            acc[6] += p.kp[3 * static_cast<size_t>(i) + c] * f[c];
            acc[7] += p.ka[3 * static_cast<size_t>(i) + c] * f[c];
        }
}
__device__ __forceinline__ void swim_tail_end(const SwimParams &p, const double (&acc)[8], double (*sm)[8], int *flag,
                                              double *out, double *part, unsigned int *counter, double *tot) {
    const double t = block_sums<8>(acc, sm);
    const int m = blockIdx.x;
    if (threadIdx.x < 6) part[static_cast<size_t>(m) * 6 + threadIdx.x] = t;
    else if (threadIdx.x < 8 && m < p.F) out[(threadIdx.x == 6 ? p.o_phase : p.o_angle) + m] = -t;
    if (swim_totals<6>(part, counter, flag, tot) && threadIdx.x < 6) out[p.o_body + threadIdx.x] = -tot[threadIdx.x];
}
__global__ void __launch_bounds__(kSwT) swim_tail_kernel(SwimParams p, const double *v, float4 *f4, double *out,
                                                         double *part, unsigned int *counter) {
    __shared__ double sm[kSwT / 32][8], tot[6];
    __shared__ int flag;
    chain_wait();
    int lo, hi;
    swim_range(p, blockIdx.x, lo, hi);
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = lo + threadIdx.x; i < hi; i += kSwT) {
        const double *f = v + swim_row(p, i);
        f4[i] = make_float4(static_cast<float>(f[0]), static_cast<float>(f[1]), static_cast<float>(f[2]), 0.0f);
        swim_tail_add(p, i, f, acc);
    }
    swim_tail_end(p, acc, sm, &flag, out, part, counter, tot);
}

// ---- preconditioner (apply_preconditioner_new, body branch, mobility_solver.cpp:1244-1475), two launches
// (a) q = src * scale (the new basis vector); per filament (-r_rate - K^T M^-1 r_1) through its 2x2 C^-1, left in the
// rate rows of z; over all blocks the body's -r_2 - K^T M^-1 r_1 - the filaments' B terms, then the 6x6 solve into the
// body rows of z.  gate: the launch does nothing where *gate is zero; ctl: scale and, for the first iteration after a
// discarded guess, rhs in place of src.
__global__ void __launch_bounds__(kSwT) swim_pre_a_kernel(SwimParams p, const int *gate, const SwimCtl *ctl,
                                                          const double *src, const double *rhs, double *q, double *z,
                                                          double *part, unsigned int *counter) {
    __shared__ double sm[kSwT / 32][8], t8[8], tot[6];
    __shared__ int flag;
    chain_wait();
    if (gate && *gate == 0) return;
    const double sc = ctl ? ctl->inv_scale : 1.0;
    if (rhs && ctl->zero_guess) src = rhs;
    int lo, hi;
    swim_range(p, blockIdx.x, lo, hi);
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = lo + threadIdx.x; i < hi; i += kSwT) {
        const long long row = swim_row(p, i);
        double f[3];
        for (int c = 0; c < 3; ++c) {
            const double v = src[row + c] * sc;
            q[row + c] = v;
            f[c] = kSwimMobInv * v;
        }
        swim_tail_add(p, i, f, acc);
    }
    const double t = block_sums<8>(acc, sm);
    if (threadIdx.x < 8) t8[threadIdx.x] = t;
    __syncthreads();
    const int m = blockIdx.x;
    if (threadIdx.x < 6) {
        double v = t8[threadIdx.x];
        if (m < p.F) {
            const double qp = src[p.o_phase + m] * sc, qa = src[p.o_angle + m] * sc;
            const double c11 = p.gram[3 * m], c22 = p.gram[3 * m + 1], c12 = p.gram[3 * m + 2];
            const double det = c11 * c22 - c12 * c12;
            const double i11 = c22 / det, i22 = c11 / det, i12 = -c12 / det;
            const double a = -qp - t8[6], b = -qa - t8[7];
            const double ph = i11 * a + i12 * b, an = i12 * a + i22 * b;
            const double *ax = p.aux + 12 * static_cast<size_t>(m);  // v_phi, u_phi, v_theta, u_theta
            v += ph * ax[threadIdx.x] + an * ax[6 + threadIdx.x];
            if (threadIdx.x == 0) {
                q[p.o_phase + m] = qp;
                q[p.o_angle + m] = qa;
                z[p.o_phase + m] = ph;
                z[p.o_angle + m] = an;
            }
        }
        part[static_cast<size_t>(m) * 6 + threadIdx.x] = v;
    }
    if (!swim_totals<6>(part, counter, &flag, tot)) return;
    if (threadIdx.x < 6) {
        const double r = src[p.o_body + threadIdx.x] * sc;
        q[p.o_body + threadIdx.x] = r;
        tot[threadIdx.x] = -r - tot[threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0.0;
        for (int c = 0; c < 6; ++c) v += p.kinv[6 * threadIdx.x + c] * tot[c];
        z[p.o_body + threadIdx.x] = v;
    }
}

// (b) the rates, divided by 6 pi mu a, minus C^-1 B^T of the body solution; s1 = M^-1 (r_1 + K s_2) on the particle
// rows.  With out, also the tail of A z (swim_tail_kernel).
__global__ void __launch_bounds__(kSwT) swim_pre_b_kernel(SwimParams p, const int *gate, const double *q, double *z,
                                                          float4 *f4, double *out, double *part, unsigned int *counter) {
    __shared__ double sm[kSwT / 32][8], tot[6];
    __shared__ int flag;
    chain_wait();
    if (gate && *gate == 0) return;
    int lo, hi;
    swim_range(p, blockIdx.x, lo, hi);
    const int m = blockIdx.x;
    double V[3], W[3], ph = 0.0, an = 0.0;
    for (int c = 0; c < 3; ++c) {
        V[c] = z[p.o_body + c];
        W[c] = z[p.o_body + 3 + c];
    }
    if (m < p.F) {
        const double c11 = p.gram[3 * m], c22 = p.gram[3 * m + 1], c12 = p.gram[3 * m + 2];
        const double det = c11 * c22 - c12 * c12;
        const double i11 = c22 / det, i22 = c11 / det, i12 = -c12 / det;
        const double *a = p.aux + 12 * static_cast<size_t>(m);
        double vpV = 0, vtV = 0, upW = 0, utW = 0;
        for (int c = 0; c < 3; ++c) {
            vpV += a[c] * V[c];
            upW += a[3 + c] * W[c];
            vtV += a[6 + c] * V[c];
            utW += a[9 + c] * W[c];
        }
        ph = z[p.o_phase + m] / kSwimMobInv - (i11 * vpV + i12 * vtV + i11 * upW + i12 * utW);
        an = z[p.o_angle + m] / kSwimMobInv - (i12 * vpV + i22 * vtV + i12 * upW + i22 * utW);
    }
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = lo + threadIdx.x; i < hi; i += kSwT) {
        const long long row = swim_row(p, i);
        double r[3];
        swim_diff(p, i, r);
        const double k[3] = {V[0] + W[1] * r[2] - W[2] * r[1], V[1] + W[2] * r[0] - W[0] * r[2],
                             V[2] + W[0] * r[1] - W[1] * r[0]};
        double f[3];
        for (int c = 0; c < 3; ++c) {
            double v = k[c];
            if (i < p.N) v += ph * p.kp[3 * static_cast<size_t>(i) + c] + an * p.ka[3 * static_cast<size_t>(i) + c];
            f[c] = kSwimMobInv * q[row + c] + kSwimMobInv * v;
            z[row + c] = f[c];
        }
        if (out) {
            f4[i] = make_float4(static_cast<float>(f[0]), static_cast<float>(f[1]), static_cast<float>(f[2]), 0.0f);
            swim_tail_add(p, i, f, acc);
        }
    }
    __syncthreads();  // every thread has read the rates as step (a) left them
    if (threadIdx.x == 0 && m < p.F) {
        z[p.o_phase + m] = ph;
        z[p.o_angle + m] = an;
    }
    if (out) swim_tail_end(p, acc, sm, &flag, out, part, counter, tot);
}

// Particle rows of A v, one warp each: the FP64 sum of the particle's pair partials and its self mobility, minus V + Omega x r, and for
// segments minus phi_dot k_phi + theta_dot k_theta.
__global__ void __launch_bounds__(256) swim_rows_kernel(SwimParams p, const int *gate, const float4 *__restrict__ partial,
                                                        int nb, const double *v, double *out) {
    chain_wait();
    if (gate && *gate == 0) return;
    const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= p.N + p.B) return;
    double o[3] = {0.0, 0.0, 0.0};
    const float4 *pt = partial + static_cast<size_t>(i) * nb;
    // eight reads of a lane in flight: bound by their latency (7,682 particles, 241 partials each: 10.2 us, one at a time
    // 13.1)
    constexpr int kDepth = 8;
    for (int s0 = lane; s0 < nb; s0 += 32 * kDepth) {
        float4 q[kDepth];
#pragma unroll
        for (int u = 0; u < kDepth; ++u)
            q[u] = s0 + 32 * u < nb ? __ldcs(pt + s0 + 32 * u) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < kDepth; ++u) {
            o[0] += q[u].x;
            o[1] += q[u].y;
            o[2] += q[u].z;
        }
    }
    for (int c = 0; c < 3; ++c) o[c] = kPairScale * warp_sum(o[c]);  // mu = 1
    if (lane != 0) return;
    double r[3];
    swim_diff(p, i, r);
    const double *V = v + p.o_body, *W = v + p.o_body + 3;
    const double wr[3] = {W[1] * r[2] - W[2] * r[1], W[2] * r[0] - W[0] * r[2], W[0] * r[1] - W[1] * r[0]};
    const long long row = swim_row(p, i);
    for (int c = 0; c < 3; ++c) o[c] += v[row + c] / kSwimMobInv - (V[c] + wr[c]);
    if (i < p.N) {
        const int m = i / p.nseg;
        const double ph = v[p.o_phase + m], an = v[p.o_angle + m];
        for (int c = 0; c < 3; ++c) o[c] -= ph * p.kp[3 * static_cast<size_t>(i) + c] + an * p.ka[3 * static_cast<size_t>(i) + c];
    }
    for (int c = 0; c < 3; ++c) out[row + c] = o[c];
}

// ---- Krylov vector kernels (rows [0, n))
// r0 = rhs - A x0 in place of A x0 in w; the block arriving last decides how the solve starts (mobility_solver.cpp:
// 2216-2424): zero right-hand side -> zero solution; a good guess is kept; a guess worse than zero is discarded.
__global__ void __launch_bounds__(kSwT) swim_start_kernel(const double *rhs, double *w, int n, double tol, SwimCtl *ctl,
                                                          double *beta, double *part, unsigned int *counter) {
    __shared__ double sm[kSwT / 32][2], tot[2];
    __shared__ int flag;
    chain_wait();
    double acc[2] = {0.0, 0.0};
    for (int i = blockIdx.x * kSwT + threadIdx.x; i < n; i += gridDim.x * kSwT) {
        const double b = rhs[i], r = b - w[i];
        w[i] = r;
        acc[0] += r * r;
        acc[1] += b * b;
    }
    const double t = block_sums<2>(acc, sm);
    if (threadIdx.x < 2) part[2 * static_cast<size_t>(blockIdx.x) + threadIdx.x] = t;
    if (!swim_totals<2>(part, counter, &flag, tot) || threadIdx.x != 0) return;
    double b0 = sqrt(tot[0]);
    const double nr = sqrt(tot[1]);
    ctl->run = 0;
    ctl->apply = 0;
    ctl->iters = 0;
    ctl->zero_guess = 0;
    ctl->status = CF_OK;
    ctl->norm_rhs = nr;
    ctl->relres = b0 / nr;
    if (ctl->singular) return;
    if (!isfinite(nr) || !isfinite(b0)) {
        ctl->status = CF_NONFINITE;
    } else if (nr == 0.0) {
        ctl->apply = 3;
        ctl->relres = 0.0;
    } else if (!(b0 <= tol * nr)) {
        if (b0 > nr) {
            ctl->zero_guess = 1;
            b0 = nr;
        }
        ctl->run = 1;
        ctl->inv_scale = 1.0 / b0;
        beta[0] = b0;
    }
}

// h[j] = <Q_j, w> for j < k1.  Block (c, j) sums the rows of chunk c with four independent accumulators; the block
// arriving last sums every j's chunks in a fixed order (part: k1 x kSwimChunks partials).
constexpr int kSwimChunks = 16;
__global__ void __launch_bounds__(256) swim_dots_kernel(const int *gate, const double *Q, long long ldq, const double *w,
                                                        int n, double *part, unsigned int *counter, double *h) {
    __shared__ double sm32[32];
    __shared__ int last;
    chain_wait();
    if (*gate == 0) return;
    const int c = blockIdx.x, j = blockIdx.y;
    const int chunk = (n + kSwimChunks - 1) / kSwimChunks;
    const int r0 = c * chunk, r1 = min(n, r0 + chunk);
    const double *q = Q + static_cast<long long>(j) * ldq;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int i = r0 + threadIdx.x;
    for (; i + 3 * 256 < r1; i += 4 * 256) {
        a0 += q[i] * w[i];
        a1 += q[i + 256] * w[i + 256];
        a2 += q[i + 512] * w[i + 512];
        a3 += q[i + 768] * w[i + 768];
    }
    for (; i < r1; i += 256) a0 += q[i] * w[i];
    const double sum = block_sum((a0 + a1) + (a2 + a3), sm32);
    if (threadIdx.x == 0) part[j * kSwimChunks + c] = sum;
    if (!arrive_last(counter, gridDim.x * gridDim.y, &last)) return;
    for (int jj = threadIdx.x; jj < static_cast<int>(gridDim.y); jj += blockDim.x) {
        double t = 0.0;
        for (int cc = 0; cc < kSwimChunks; ++cc) t += __ldcg(&part[jj * kSwimChunks + cc]);
        h[jj] = t;
    }
    if (threadIdx.x == 0) *counter = 0;
}

// w -= sum_j h[j] Q_j (j < k1).  In the final pass (h1 given) also |w|, and by the block arriving last the Givens step
// of column k1 - 1 of the Hessenberg matrix, h1 + h (mobility_solver.cpp:2462-2515), and the stopping decision.
struct SwimGivens {
    double *H, *cs, *sn, *beta;
    const double *h1;
    int ldh, max_iter;
    double tol;
};
__global__ void __launch_bounds__(kSwT) swim_sub_kernel(const int *gate, double *w, const double *Q, long long ldq,
                                                        const double *h, int k1, int n, SwimGivens g, SwimCtl *ctl,
                                                        double *part, unsigned int *counter) {
    __shared__ double sm[kSwT / 32][1], tot[1];
    __shared__ int flag;
    chain_wait();
    if (*gate == 0) return;
    const int i = blockIdx.x * kSwT + threadIdx.x;
    double acc[1] = {0.0};
    if (i < n) {
        double s0 = 0.0, s1 = 0.0;
        int j = 0;
        for (; j + 1 < k1; j += 2) {
            s0 += h[j] * Q[static_cast<long long>(j) * ldq + i];
            s1 += h[j + 1] * Q[static_cast<long long>(j + 1) * ldq + i];
        }
        if (j < k1) s0 += h[j] * Q[static_cast<long long>(j) * ldq + i];
        const double v = w[i] - (s0 + s1);
        w[i] = v;
        acc[0] = v * v;
    }
    if (!g.h1) return;
    const double t = block_sums<1>(acc, sm);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
    if (!swim_totals<1>(part, counter, &flag, tot)) return;
    double *col = g.H + static_cast<size_t>(k1 - 1) * g.ldh;  // column k1 - 1, rows 0 .. k1
    for (int r = threadIdx.x; r < k1; r += kSwT) col[r] = g.h1[r] + h[r];
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double qn = sqrt(tot[0]);
    ctl->iters = k1;
    if (!isfinite(qn)) {
        ctl->run = 0;
        ctl->status = CF_NONFINITE;
        ctl->relres = qn;
        return;
    }
    for (int r = 1; r < k1; ++r) {
        const double a = g.cs[r - 1] * col[r - 1] + g.sn[r - 1] * col[r];
        col[r] = g.cs[r - 1] * col[r] - g.sn[r - 1] * col[r - 1];
        col[r - 1] = a;
    }
    const double a = col[k1 - 1];
    double c, s;
    if (qn == 0.0) {
        c = 1.0;
        s = 0.0;
    } else if (fabs(qn) > fabs(a)) {
        const double tt = a / qn;
        s = 1.0 / sqrt(1.0 + tt * tt);
        c = tt * s;
    } else {
        const double tt = qn / a;
        c = (a > 0 ? 1.0 : -1.0) / sqrt(1.0 + tt * tt);
        s = tt * c;
    }
    g.cs[k1 - 1] = c;
    g.sn[k1 - 1] = s;
    col[k1 - 1] = c * a + s * qn;
    col[k1] = 0.0;
    const double bk = g.beta[k1 - 1];
    g.beta[k1] = -s * bk;
    g.beta[k1 - 1] = c * bk;
    const double rel = fabs(s * bk) / ctl->norm_rhs;
    ctl->relres = rel;
    ctl->inv_scale = qn != 0.0 ? 1.0 / qn : 1.0;
    if (rel <= g.tol || k1 == g.max_iter) {
        ctl->run = 0;
        ctl->status = rel <= g.tol ? CF_OK : CF_NOT_CONVERGED;
        ctl->apply = ctl->zero_guess ? 2 : 1;
    }
}

// H y = beta by one block, column oriented (mobility_solver.cpp:2520-2537).
__global__ void __launch_bounds__(256) swim_backsub_kernel(const SwimCtl *ctl, const double *H, int ldh,
                                                           const double *beta, double *y) {
    chain_wait();
    if (ctl->apply != 1 && ctl->apply != 2) return;
    const int k = ctl->iters;
    for (int r = threadIdx.x; r < k; r += blockDim.x) y[r] = beta[r];
    __syncthreads();
    for (int i = k - 1; i >= 0; --i) {
        const double *col = H + static_cast<size_t>(i) * ldh;
        if (threadIdx.x == 0) y[i] /= col[i];
        __syncthreads();
        const double yi = y[i];
        for (int r = threadIdx.x; r < i; r += blockDim.x) y[r] -= col[r] * yi;
        __syncthreads();
    }
}

// t = sum_j y_j Q_j
__global__ void __launch_bounds__(256) swim_combine_kernel(const SwimCtl *ctl, double *t, const double *Q, long long ldq,
                                                           const double *y, int n) {
    chain_wait();
    if (ctl->apply != 1 && ctl->apply != 2) return;
    const int k = ctl->iters;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s0 = 0.0, s1 = 0.0;
    int j = 0;
    for (; j + 1 < k; j += 2) {
        s0 += y[j] * Q[static_cast<long long>(j) * ldq + i];
        s1 += y[j + 1] * Q[static_cast<long long>(j + 1) * ldq + i];
    }
    if (j < k) s0 += y[j] * Q[static_cast<long long>(j) * ldq + i];
    t[i] = s0 + s1;
}

__global__ void swim_set_step_kernel(LoopCtl *lc, int nt) { lc->nt = nt; }

// sol as ctl->apply says, and the rates that the next step advances with; both stay as they are where the body matrix
// could not be inverted (no solve took place).
__global__ void swim_finish_kernel(SwimParams p, const SwimCtl *ctl, const double *z, double *sol, int n,
                                   double *phase_dot, double *angle_dot) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || ctl->singular) return;
    const int a = ctl->apply;
    double v = sol[i];
    if (a == 1) v += z[i];
    else if (a == 2) v = z[i];
    else if (a == 3) v = 0.0;
    sol[i] = v;
    if (i >= p.o_phase && i < p.o_phase + p.F) phase_dot[i - p.o_phase] = v;
    if (i >= p.o_angle && i < p.o_angle + p.F) angle_dot[i - p.o_angle] = v;
}

// ------------------------------------------------------------ host side
template <typename T>
int swim_alloc(cf_swim *h, T **p, size_t n) {
    *p = nullptr;
    void *q = nullptr;
    CF_CUDA(cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T)));
    h->allocations.push_back(q);
    *p = static_cast<T *>(q);
    return CF_OK;
}

template <typename T>
int swim_upload(cf_swim *h, T **p, const T *host, size_t n) {
    CF_TRY(swim_alloc(h, p, n));
    if (host && n) CF_CUDA(cudaMemcpy(*p, host, n * sizeof(T), cudaMemcpyHostToDevice));
    return CF_OK;
}

SwimParams swim_params(const cf_swim *h) {
    SwimParams p{};
    p.F = h->F;
    p.nseg = h->nseg;
    p.N = h->N;
    p.B = h->B;
    p.o_blob = h->o_blob;
    p.o_body = h->o_body;
    p.o_phase = h->o_phase;
    p.o_angle = h->o_angle;
    p.xd = h->d.xd;
    p.kp = h->d.kp;
    p.ka = h->d.ka;
    p.gram = h->d.gram;
    p.xb = h->xb;
    p.body = h->body;
    p.aux = h->aux;
    p.kinv = h->kinv;
    return p;
}

int swim_grid(int n) { return std::max(1, (n + 255) / 256); }
int swim_blocks(const cf_swim *h) { return h->F + (h->B + kSwT - 1) / kSwT; }

// Particle rows of out = A v once f4 holds v's forces (system_matrix_mult_new, body branch).
int swim_rows(cf_swim *h, const double *v, double *out, const int *gate) {
    cudaStream_t st = h->stream;
    const int np = h->N + h->B;
    RpyBlockDesc d{};
    d.wall = 0;
    d.vd = 3;
    d.fd = 3;
    d.self_set = 0;
    d.xt = h->x4all;
    d.nt = np;
    d.at = 1.0f;
    d.xs = h->x4all;
    d.fs = h->f4all;
    d.ts = nullptr;
    d.ns = np;
    d.as = 1.0f;
    d.mu = 1.0f;
    d.gate = gate;
    const RpyPlan plan = rpy_plan_for(d, h->num_sms);  // equal spheres on themselves: the symmetric kernel
    CF_TRY(rpy_launch_tiles(d, plan, h->scratch, h->err, st));
    CF_CUDA(launch_chained(swim_rows_kernel, dim3((np + 7) / 8), dim3(256), 0, st, swim_params(h), gate,
                           static_cast<const float4 *>(h->scratch), plan.nsplit, v, out));
    CF_CHECK_LAUNCH("swim_rows_kernel");
    return CF_OK;
}

// out = A v
int swim_matvec(cf_swim *h, const double *v, double *out) {
    CF_CUDA(launch_chained(swim_tail_kernel, dim3(swim_blocks(h)), dim3(kSwT), 0, h->stream, swim_params(h), v, h->f4all,
                           out, h->part, h->counter));
    CF_CHECK_LAUNCH("swim_tail_kernel");
    return swim_rows(h, v, out, nullptr);
}

// q = the vector preconditioned, z = P q; with out also the tail of A z.
int swim_precond(cf_swim *h, const int *gate, const SwimCtl *ctl, const double *src, const double *rhs, double *q,
                 double *z, double *out) {
    cudaStream_t st = h->stream;
    const SwimParams p = swim_params(h);
    const dim3 grid(swim_blocks(h));
    CF_CUDA(launch_chained(swim_pre_a_kernel, grid, dim3(kSwT), 0, st, p, gate, ctl, src, rhs, q, z, h->part, h->counter));
    CF_CHECK_LAUNCH("swim_pre_a_kernel");
    CF_CUDA(launch_chained(swim_pre_b_kernel, grid, dim3(kSwT), 0, st, p, gate, static_cast<const double *>(q), z, h->f4all,
                           out, h->part, h->counter));
    CF_CHECK_LAUNCH("swim_pre_b_kernel");
    return CF_OK;
}

int swim_sync(cf_swim *h) {
    CF_CUDA(cudaMemcpyAsync(&h->h_rep->err, h->err, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CF_CUDA(cudaStreamSynchronize(h->stream));
    if (h->h_rep->err) {
        CF_CUDA(cudaMemsetAsync(h->err, 0, sizeof(int), h->stream));
        return set_error(CF_TIMEOUT, "swim: a bounded device wait gave up (flags 0x%x)", h->h_rep->err);
    }
    return CF_OK;
}

// Right-preconditioned GMRES on A sol = rhs with the warm start in sol (mobility_solver.cpp:2187-2669), then the
// solution's update.  The control record of iteration i - 1 is looked at after iteration i was enqueued, so the device
// always has work queued; the at most one iteration enqueued past the end does nothing (its kernels see run = 0).
int swim_gmres(cf_swim *h) {
    const int n = h->n, M = h->max_iter, sub_grid = (n + kSwT - 1) / kSwT;
    cudaStream_t st = h->stream;
    const long long ldq = n;
    const int *run = &h->ctl->run;
    CF_TRY(swim_matvec(h, h->sol, h->w));
    CF_CUDA(launch_chained(swim_start_kernel, dim3(2 * h->num_sms), dim3(kSwT), 0, st, static_cast<const double *>(h->rhs),
                           h->w, n, h->cfg.gmres_tol, h->ctl, h->beta, h->part, h->counter));
    CF_CHECK_LAUNCH("swim_start_kernel");
    for (int it = 1; it <= M; ++it) {
        const double *src = h->w, *rhs = it == 1 ? h->rhs : nullptr, *Q = h->Q;
        double *q = h->Q + static_cast<long long>(it - 1) * ldq;
        CF_TRY(swim_precond(h, run, h->ctl, src, rhs, q, h->z, h->w));
        CF_TRY(swim_rows(h, h->z, h->w, run));
        const double *wv = h->w;
        for (int pass = 0; pass < 2; ++pass) {
            double *hh = pass == 0 ? h->h1 : h->h2;
            CF_CUDA(launch_chained(swim_dots_kernel, dim3(kSwimChunks, it), dim3(256), 0, st, run, Q, ldq, wv, n, h->part,
                                   h->counter, hh));
            CF_CHECK_LAUNCH("swim_dots_kernel");
            SwimGivens g{h->H, h->cs, h->sn, h->beta, pass == 0 ? nullptr : h->h1, M + 1, M, h->cfg.gmres_tol};
            CF_CUDA(launch_chained(swim_sub_kernel, dim3(sub_grid), dim3(kSwT), 0, st, run, h->w, Q, ldq,
                                   static_cast<const double *>(hh), it, n, g, h->ctl, h->part, h->counter));
            CF_CHECK_LAUNCH("swim_sub_kernel");
        }
        CF_CUDA(cudaMemcpyAsync(&h->h_rep->ctl[it & 1], h->ctl, sizeof(SwimCtl), cudaMemcpyDeviceToHost, st));
        CF_CUDA(cudaEventRecord(h->ev[it & 1], st));
        if (it > 1) {
            CF_CUDA(cudaEventSynchronize(h->ev[(it - 1) & 1]));
            if (!h->h_rep->ctl[(it - 1) & 1].run) break;
        }
    }
    const SwimCtl *ctl = h->ctl;
    CF_CUDA(launch_chained(swim_backsub_kernel, dim3(1), dim3(256), 0, st, ctl, static_cast<const double *>(h->H), M + 1,
                           static_cast<const double *>(h->beta), h->y));
    CF_CHECK_LAUNCH("swim_backsub_kernel");
    CF_CUDA(launch_chained(swim_combine_kernel, dim3(swim_grid(n)), dim3(256), 0, st, ctl, h->t,
                           static_cast<const double *>(h->Q), ldq, static_cast<const double *>(h->y), n));
    CF_CHECK_LAUNCH("swim_combine_kernel");
    CF_TRY(swim_precond(h, &h->ctl->apply, nullptr, h->t, nullptr, h->w, h->z, nullptr));
    CF_CUDA(launch_chained(swim_finish_kernel, dim3(swim_grid(n)), dim3(256), 0, st, swim_params(h),
                           ctl, static_cast<const double *>(h->z), h->sol, n,
                           h->d.phase_dot, h->d.angle_dot));
    CF_CHECK_LAUNCH("swim_finish_kernel");
    CF_CUDA(cudaMemcpyAsync(&h->h_rep->ctl[0], h->ctl, sizeof(SwimCtl), cudaMemcpyDeviceToHost, st));
    CF_CUDA(cudaMemcpyAsync(h->h_rep->bv, h->sol + h->o_body, 6 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CF_TRY(swim_sync(h));
    const SwimCtl &c = h->h_rep->ctl[0];
    h->last_iters = c.iters;
    h->last_relres = c.relres;
    h->last_status = c.status;
    return CF_OK;
}

void swim_release(cf_swim *h) {
    cudaSetDevice(h->device);
    for (void *p : h->allocations) cudaFree(p);
    h->allocations.clear();
    h->pinned.release();
    h->h_rep = nullptr;
    for (cudaEvent_t &e : h->ev) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    if (h->stream) cudaStreamDestroy(h->stream);
    h->stream = nullptr;
}

}  // namespace swim
}  // namespace cufil

using namespace cufil;
using namespace cufil::swim;

extern "C" int cf_swim_destroy(cf_swim *h) {
    if (!h) return CF_OK;
    swim_release(h);
    delete h;
    return CF_OK;
}

extern "C" int cf_swim_create(const cf_swim_config *cfg, cf_swim **out) {
    clear_error();
    CF_REQUIRE(cfg && out, "cf_swim_create: null argument");
    *out = nullptr;
    CF_REQUIRE(cfg->n_fil > 0 && cfg->n_seg >= 2 && cfg->n_seg <= 256 && cfg->n_blob >= 0,
               "cf_swim_create: need n_fil > 0, 2 <= n_seg <= 256, n_blob >= 0 (got %d, %d, %d)", cfg->n_fil,
               cfg->n_seg, cfg->n_blob);
    CF_REQUIRE(cfg->beat == CF_BEAT_FULFORD_BLAKE || cfg->beat == CF_BEAT_FULFORD_BLAKE_ORIGINAL,
               "cf_swim_create: unknown beat %d", cfg->beat);
    CF_REQUIRE(cfg->dt > 0 && cfg->seg_sep > 0 && cfg->gmres_tol > 0 && cfg->gmres_max_iter > 0,
               "cf_swim_create: dt, seg_sep, gmres_tol and gmres_max_iter must be positive");
    CF_REQUIRE(cfg->fil_refs && cfg->fil_dirs && (cfg->n_blob == 0 || cfg->blob_refs),
               "cf_swim_create: fil_refs, fil_dirs (and blob_refs when n_blob > 0) are required");
    CF_REQUIRE(cfg->gen_phase_force_refs && cfg->n_gen_phase_refs > 1 && cfg->gen_angle_force_refs &&
                   cfg->n_gen_angle_refs > 1,
               "cf_swim_create: the generalised-force tables are required (dynamic phase and angle)");
    const long long nsys = 3LL * cfg->n_fil * cfg->n_seg + 3LL * cfg->n_blob + 6 + 2LL * cfg->n_fil;
    CF_REQUIRE(nsys < (1LL << 28), "cf_swim_create: system too large");
    CF_CUDA(cudaSetDevice(cfg->device));
    cf_swim *h = new (std::nothrow) cf_swim();
    if (!h) return set_error(CF_ENOMEM, "cf_swim_create: host allocation failed");
    h->cfg = *cfg;
    h->device = cfg->device;
    h->F = cfg->n_fil;
    h->nseg = cfg->n_seg;
    h->N = cfg->n_fil * cfg->n_seg;
    h->B = cfg->n_blob;
    h->o_blob = 3 * h->N;
    h->o_body = h->o_blob + 3 * h->B;
    h->o_phase = h->o_body + 6;
    h->o_angle = h->o_phase + h->F;
    h->n = static_cast<int>(nsys);
    h->max_iter = std::min(h->n, cfg->gmres_max_iter);
    h->fil_ref.assign(cfg->fil_refs, cfg->fil_refs + 3 * static_cast<size_t>(h->F));
    if (h->B) h->blob_ref.assign(cfg->blob_refs, cfg->blob_refs + 3 * static_cast<size_t>(h->B));
    if (cfg->body_x0)
        for (int c = 0; c < 3; ++c) h->bx[c] = cfg->body_x0[c];
    if (cfg->body_q0) {
        Quat q{cfg->body_q0[0], {cfg->body_q0[1], cfg->body_q0[2], cfg->body_q0[3]}};
        qnormalise(q);
        h->bq[0] = q.s;
        for (int c = 0; c < 3; ++c) h->bq[1 + c] = q.v[c];
    }
    h->qref.resize(4 * static_cast<size_t>(h->F));
    for (int m = 0; m < h->F; ++m) {
        const Quat q = filament_frame(cfg->fil_dirs + 3 * m);
        h->qref[4 * m] = q.s;
        for (int c = 0; c < 3; ++c) h->qref[4 * m + 1 + c] = q.v[c];
    }
    int rc = CF_OK;
    do {
        if ((rc = cuda_status(cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, cfg->device),
                              "cudaDeviceGetAttribute", __FILE__, __LINE__)))
            break;
        if ((rc = cuda_status(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking), "cudaStreamCreate",
                              __FILE__, __LINE__)))
            break;
        SimDev &d = h->d;
        const int F = h->F, ns = h->nseg;
        d.B = 1;
        d.F = F;
        d.nseg = ns;
        d.N = h->N;
        d.dt = cfg->dt;
        d.L = cfg->seg_sep * (ns - 1);
        d.spring = cfg->spring_factor;
        d.s_tol = (cfg->s_tol_factor > 0 ? cfg->s_tol_factor : 0.1) / ns;
        d.beat = beat_table(cfg->beat);
        d.s_rows = cfg->s_values_ref ? cfg->s_ref_rows : 0;
        d.s_cols = cfg->s_values_ref ? cfg->s_ref_cols : 0;
        d.n_phase_refs = cfg->n_gen_phase_refs;
        d.n_angle_refs = cfg->n_gen_angle_refs;
        d.dyn_phase = d.dyn_angle = 1;
        std::vector<double> omega(F), ph(F, 0.0), an(F, 0.0), zeros(F, 0.0);
        for (int m = 0; m < F; ++m) {
            omega[m] = cfg->omega0 ? cfg->omega0[m] : 2.0 * 3.14159265358979323846;
            if (cfg->phase0) ph[m] = cfg->phase0[m];
            if (cfg->angle0) an[m] = cfg->angle0[m];
        }
        const size_t N = h->N, np = h->N + h->B, nv = h->n, mi = h->max_iter;
        // block partials: the begin kernel's sums, the dot products' chunks, the norms
        const size_t npart = std::max({static_cast<size_t>(swim_blocks(h)) * kPreValues, (mi + 1) * kSwimChunks,
                                       (nv + kSwT - 1) / kSwT, 4 * static_cast<size_t>(h->num_sms)});
        if ((rc = swim_upload(h, const_cast<double **>(&d.s_table), cfg->s_values_ref,
                              static_cast<size_t>(d.s_rows) * d.s_cols)) ||
            (rc = swim_upload(h, const_cast<double **>(&d.phase_refs), cfg->gen_phase_force_refs, d.n_phase_refs)) ||
            (rc = swim_upload(h, const_cast<double **>(&d.angle_refs), cfg->gen_angle_force_refs, d.n_angle_refs)) ||
            (rc = swim_upload(h, const_cast<double **>(&d.omega0), omega.data(), F)) ||
            (rc = swim_alloc(h, const_cast<double **>(&d.base), 3 * static_cast<size_t>(F))) ||
            (rc = swim_upload(h, &d.phase, ph.data(), F)) || (rc = swim_upload(h, &d.angle, an.data(), F)) ||
            (rc = swim_upload(h, &d.phase_dot, omega.data(), F)) ||
            (rc = swim_upload(h, &d.angle_dot, zeros.data(), F)) || (rc = swim_alloc(h, &d.x4, N)) ||
            (rc = swim_alloc(h, &d.xd, 3 * N)) || (rc = swim_alloc(h, &d.s_cur, N)) ||
            (rc = swim_alloc(h, &d.kp, 3 * N)) || (rc = swim_alloc(h, &d.ka, 3 * N)) ||
            (rc = swim_alloc(h, &d.gram, 3 * static_cast<size_t>(F))) || (rc = swim_alloc(h, &d.lc, 1)) ||
            (rc = swim_alloc(h, &h->Rfil, 9 * static_cast<size_t>(F))) ||
            (rc = swim_alloc(h, &h->xb, 3 * static_cast<size_t>(h->B))) || (rc = swim_alloc(h, &h->body, 3)) ||
            (rc = swim_alloc(h, &h->aux, 12 * static_cast<size_t>(F))) || (rc = swim_alloc(h, &h->kinv, 36)) ||
            (rc = swim_alloc(h, &h->x4all, np)) || (rc = swim_alloc(h, &h->f4all, np)) ||
            (rc = swim_alloc(h, &h->err, 1)) ||
            (rc = swim_upload(h, &h->d_qref, h->qref.data(), h->qref.size())) ||
            (rc = swim_upload(h, &h->d_fil_ref, h->fil_ref.data(), h->fil_ref.size())) ||
            (rc = swim_upload(h, &h->d_blob_ref, h->blob_ref.data(), h->blob_ref.size())) ||
            (rc = swim_alloc(h, &h->rhs, nv)) || (rc = swim_alloc(h, &h->sol, nv)) || (rc = swim_alloc(h, &h->w, nv)) ||
            (rc = swim_alloc(h, &h->z, nv)) || (rc = swim_alloc(h, &h->t, nv)) ||
            (rc = swim_alloc(h, &h->Q, static_cast<size_t>(h->max_iter + 1) * nv)) ||
            (rc = swim_alloc(h, &h->h1, mi + 1)) || (rc = swim_alloc(h, &h->h2, mi + 1)) ||
            (rc = swim_alloc(h, &h->H, (mi + 1) * (mi + 1))) || (rc = swim_alloc(h, &h->cs, mi + 1)) ||
            (rc = swim_alloc(h, &h->sn, mi + 1)) || (rc = swim_alloc(h, &h->beta, mi + 1)) || (rc = swim_alloc(h, &h->y, mi + 1)) ||
            (rc = swim_alloc(h, &h->part, npart)) || (rc = swim_alloc(h, &h->counter, 1)) ||
            (rc = swim_alloc(h, &h->ctl, 1)))
            break;
        if ((rc = cuda_status(cudaMemset(h->counter, 0, sizeof(unsigned int)), "cudaMemset", __FILE__, __LINE__)) ||
            (rc = cuda_status(cudaMemset(h->ctl, 0, sizeof(SwimCtl)), "cudaMemset", __FILE__, __LINE__)) ||
            (rc = cuda_status(cudaMemset(h->rhs, 0, sizeof(double) * nv), "cudaMemset", __FILE__, __LINE__)) ||
            (rc = cuda_status(cudaEventCreateWithFlags(&h->ev[0], cudaEventDisableTiming), "cudaEventCreate", __FILE__,
                              __LINE__)) ||
            (rc = cuda_status(cudaEventCreateWithFlags(&h->ev[1], cudaEventDisableTiming), "cudaEventCreate", __FILE__,
                              __LINE__)))
            break;
        d.Rfil = h->Rfil;
        h->h_rep = &h->own_rep;
        RpyBlockDesc bd{};
        bd.wall = 0;
        bd.vd = 3;
        bd.fd = 3;
        bd.nt = bd.ns = static_cast<int>(np);
        h->scratch_cap = rpy_plan_for(bd, h->num_sms).scratch_float4;
        if ((rc = swim_alloc(h, &h->scratch, h->scratch_cap))) break;
        if ((rc = cuda_status(cudaMemset(h->err, 0, sizeof(int)), "cudaMemset", __FILE__, __LINE__))) break;
        if ((rc = cuda_status(cudaMemset(h->sol, 0, sizeof(double) * nv), "cudaMemset", __FILE__, __LINE__))) break;
        LoopCtl lc{};
        if ((rc = cuda_status(cudaMemcpy(d.lc, &lc, sizeof(lc), cudaMemcpyHostToDevice), "cudaMemcpy", __FILE__,
                              __LINE__)))
            break;
        const size_t kin_smem = sizeof(double) * (2 * (10 * ns + 1) + ns);
        if (kin_smem > 48 * 1024 &&
            (rc = cuda_status(cudaFuncSetAttribute(kinematics_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(kin_smem)),
                              "cudaFuncSetAttribute", __FILE__, __LINE__)))
            break;
    } while (0);
    if (rc != CF_OK) {
        const std::string msg = cf_last_error();
        cf_swim_destroy(h);
        return set_error(rc, "%s", msg.c_str());
    }
    *out = h;
    return CF_OK;
}

// One implicit step of the swimmer (filament and swimmer initial_guess, compute_velocities, the body update).
extern "C" int cf_swim_step(cf_swim *h, int nt, int *iters, double *relres) {
    clear_error();
    CF_REQUIRE(h && nt >= 0, "cf_swim_step: bad arguments");
    CF_CUDA(cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    SimDev &d = h->d;
    void *locked = h->pinned.open(sizeof(SwimReport));
    h->h_rep = locked ? static_cast<SwimReport *>(locked) : &h->own_rep;
    BodyState body;
    for (int c = 0; c < 3; ++c) body.x[c] = h->bx[c];
    for (int c = 0; c < 4; ++c) body.q[c] = h->bq[c];
    swim_frames_kernel<<<swim_grid(h->F + h->B), 256, 0, st>>>(body, h->F, h->B, h->d_qref, h->d_fil_ref, h->d_blob_ref,
                                                               h->Rfil, const_cast<double *>(d.base), h->xb, h->body);
    CF_CHECK_LAUNCH("swim_frames_kernel");
    swim_set_step_kernel<<<1, 1, 0, st>>>(d.lc, nt);
    CF_CHECK_LAUNCH("swim_set_step_kernel");
    const int ns = h->nseg;
    const int threads = std::min(256, std::max(64, (3 * ns + 31) / 32 * 32));
    const size_t kin_smem = sizeof(double) * (2 * (10 * ns + 1) + ns);
    kinematics_kernel<<<h->F, threads, kin_smem, st>>>(d);
    CF_CHECK_LAUNCH("kinematics_kernel");
    const SwimParams p = swim_params(h);
    swim_begin_kernel<<<swim_blocks(h), kSwT, 0, st>>>(p, d, h->x4all, h->rhs, h->aux, d.gram, h->kinv, h->part,
                                                       h->counter, h->ctl);
    CF_CHECK_LAUNCH("swim_begin_kernel");
    CF_TRY(swim_gmres(h));
    if (h->h_rep->ctl[0].singular)
        return set_error(CF_NONFINITE, "cf_swim: the body's 6x6 preconditioner matrix is singular");
    h->stepped = true;
    for (int c = 0; c < 6; ++c) h->bv[c] = h->h_rep->bv[c];
    if (iters) *iters = h->last_iters;
    if (relres) *relres = h->last_relres;
    if (h->last_status == CF_NONFINITE)
        return set_error(CF_NONFINITE, "cf_swim: GMRES met a non-finite value (relative residual %.3e)",
                         h->last_relres);
    // explicit body update (cilia_sim_main.cu:700-716): x += dt V, q = lie_exp(dt Omega) q
    const double dt = h->cfg.dt;
    for (int c = 0; c < 3; ++c) h->bx[c] += dt * h->bv[c];
    const double uu[3] = {dt * h->bv[3], dt * h->bv[4], dt * h->bv[5]};
    const Quat q = qmul(qlie_exp(uu), Quat{h->bq[0], {h->bq[1], h->bq[2], h->bq[3]}});
    h->bq[0] = q.s;
    for (int c = 0; c < 3; ++c) h->bq[1 + c] = q.v[c];
    if (h->last_status == CF_NOT_CONVERGED)
        return set_error(CF_NOT_CONVERGED, "cf_swim: GMRES stopped at its cap: %d iterations, relative residual %.3e",
                         h->last_iters, h->last_relres);
    return CF_OK;
}

// State after the last step: per filament phase, angle and their rates [F] each; the body's
// position [3] and orientation [4] for the next step, and the velocity [6] (V, Omega) solved in the last step.
extern "C" int cf_swim_get_state(cf_swim *h, double *phase, double *angle, double *phase_dot, double *angle_dot,
                                 double *body_x, double *body_q, double *body_v) {
    clear_error();
    CF_REQUIRE(h, "null handle");
    CF_CUDA(cudaSetDevice(h->device));
    const size_t fb = sizeof(double) * h->F;
    cudaStream_t st = h->stream;
    if (phase) CF_CUDA(cudaMemcpyAsync(phase, h->d.phase, fb, cudaMemcpyDeviceToHost, st));
    if (angle) CF_CUDA(cudaMemcpyAsync(angle, h->d.angle, fb, cudaMemcpyDeviceToHost, st));
    if (phase_dot) CF_CUDA(cudaMemcpyAsync(phase_dot, h->d.phase_dot, fb, cudaMemcpyDeviceToHost, st));
    if (angle_dot) CF_CUDA(cudaMemcpyAsync(angle_dot, h->d.angle_dot, fb, cudaMemcpyDeviceToHost, st));
    CF_CUDA(cudaStreamSynchronize(st));
    if (body_x) std::memcpy(body_x, h->bx, sizeof(h->bx));
    if (body_q) std::memcpy(body_q, h->bq, sizeof(h->bq));
    if (body_v) std::memcpy(body_v, h->bv, sizeof(h->bv));
    return CF_OK;
}

// Segment positions [3N] and blob positions [3B] of the last step (FP64), and the solution's
// segment and blob forces [3N], [3B]; any pointer may be NULL.
extern "C" int cf_swim_get_particles(cf_swim *h, double *x_segs, double *x_blobs, double *f_segs, double *f_blobs) {
    clear_error();
    CF_REQUIRE(h, "null handle");
    CF_CUDA(cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    if (x_segs) CF_CUDA(cudaMemcpyAsync(x_segs, h->d.xd, sizeof(double) * 3 * h->N, cudaMemcpyDeviceToHost, st));
    if (x_blobs && h->B)
        CF_CUDA(cudaMemcpyAsync(x_blobs, h->xb, sizeof(double) * 3 * h->B, cudaMemcpyDeviceToHost, st));
    if (f_segs) CF_CUDA(cudaMemcpyAsync(f_segs, h->sol, sizeof(double) * 3 * h->N, cudaMemcpyDeviceToHost, st));
    if (f_blobs && h->B)
        CF_CUDA(cudaMemcpyAsync(f_blobs, h->sol + h->o_blob, sizeof(double) * 3 * h->B, cudaMemcpyDeviceToHost, st));
    CF_CUDA(cudaStreamSynchronize(st));
    return CF_OK;
}

// Velocity directions of the last step's kinematics (vel_dir_phase, vel_dir_angle) [3N] each.
extern "C" int cf_swim_get_directions(cf_swim *h, double *k_phase, double *k_angle) {
    clear_error();
    CF_REQUIRE(h && h->stepped, "cf_swim_get_directions: bad handle or no step yet");
    CF_CUDA(cudaSetDevice(h->device));
    const size_t b = sizeof(double) * 3 * h->N;
    if (k_phase) CF_CUDA(cudaMemcpyAsync(k_phase, h->d.kp, b, cudaMemcpyDeviceToHost, h->stream));
    if (k_angle) CF_CUDA(cudaMemcpyAsync(k_angle, h->d.ka, b, cudaMemcpyDeviceToHost, h->stream));
    CF_CUDA(cudaStreamSynchronize(h->stream));
    return CF_OK;
}

// A x and P x on host vectors of the system size, for the current geometry (after a step).
extern "C" int cf_swim_system_matvec(cf_swim *h, const double *in, double *out) {
    clear_error();
    CF_REQUIRE(h && in && out && h->stepped, "cf_swim_system_matvec: bad arguments or no step yet");
    CF_CUDA(cudaSetDevice(h->device));
    CF_CUDA(cudaMemcpyAsync(h->z, in, sizeof(double) * h->n, cudaMemcpyHostToDevice, h->stream));
    CF_TRY(swim_matvec(h, h->z, h->w));
    CF_CUDA(cudaMemcpyAsync(out, h->w, sizeof(double) * h->n, cudaMemcpyDeviceToHost, h->stream));
    return swim_sync(h);
}

extern "C" int cf_swim_apply_preconditioner(cf_swim *h, const double *in, double *out) {
    clear_error();
    CF_REQUIRE(h && in && out && h->stepped, "cf_swim_apply_preconditioner: bad arguments or no step yet");
    CF_CUDA(cudaSetDevice(h->device));
    CF_CUDA(cudaMemcpyAsync(h->t, in, sizeof(double) * h->n, cudaMemcpyHostToDevice, h->stream));
    CF_TRY(swim_precond(h, nullptr, nullptr, h->t, nullptr, h->w, h->z, nullptr));
    CF_CUDA(cudaMemcpyAsync(out, h->z, sizeof(double) * h->n, cudaMemcpyDeviceToHost, h->stream));
    return swim_sync(h);
}

extern "C" int cf_swim_system_size(cf_swim *h) { return h ? h->n : -1; }
