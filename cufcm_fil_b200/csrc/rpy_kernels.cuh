// rpy_kernels.cuh -- launch interface of the pairwise RPY block products.
//
// A block product V_t = M(t <- s) F_s is computed in two launches:
//   1. rpy_tile: grid (target tiles x source splits); each CTA stages its
//      source split (positions, forces, torques as float4) into shared memory
//      with one bulk async copy per array, then every thread sums the pair
//      blocks of its TI targets over the split in FP32 with blockwise
//      compensated (TwoSum) accumulation, and writes one partial per target.
//   2. rpy_reduce: sums the partials of each target over the splits in FP64
//      in a fixed order (deterministic), adds the wall self block, and writes
//      or accumulates the result in the caller's layout.
// The split count is chosen so that the grid fills every SM; the partials
// buffer (`scratch`) holds nt * nsplit * (VD/3) float4, target-major:
// partial[(i * nsplit + s) * (VD/3) + w], so the splits of one target are
// contiguous for the reduction.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

namespace cufil {

struct RpyBlockDesc {
    int wall;             // 1: Swan-Brady wall blocks, 0: unbounded
    int vd, fd;           // 3 or 6
    int self_set;         // targets and sources are the same particles
    const float4 *xt;     // target centres [nt] (w ignored)
    int nt;
    float at;             // target radius (unbounded only)
    const float4 *xs;     // source centres [ns]
    const float4 *fs;     // source forces [ns]
    const float4 *ts;     // source torques [ns] (fd == 6)
    int ns;
    float as;             // source radius (unbounded only)
    float mu;             // viscosity (unbounded only)
    const int *gate;      // may be null; the symmetric 3x3 kernel does nothing where *gate is zero
};

struct RpyPlan {
    int sym;       // 1: symmetric warp-tile kernel (a set on itself)
    int n6;        // symmetric: the first n6 particles have torques and spins
    int nb;        // symmetric: 32-particle tiles
    bool packed;      // symmetric: what the items are (rpy_sym_items); false with torques
    long long items;  // symmetric: work items
    int grid;      // symmetric: CTAs
    int ti;        // targets per thread
    int tiles;     // target tiles (gridDim.x)
    int nsplit;    // source splits (gridDim.y)
    int split;     // sources per split
    size_t smem;   // dynamic shared memory bytes of the tile kernel
    size_t scratch_float4;  // float4 entries of the partials buffer
};

// Number of float4 entries needed in the partials buffer for any product with
// at most nt_max targets (sizing helper for allocators).
size_t rpy_scratch_float4(int nt_max, int ns_max, int vd, int num_sms);

RpyPlan rpy_plan(int nt, int ns, int vd, int fd, int num_sms);
// Same with at most max_nsplit source splits (bounded partials buffer); the
// split count never drops below ceil(ns / 2048).
RpyPlan rpy_plan_capped(int nt, int ns, int vd, int fd, int num_sms, int max_nsplit);
// Plan of the symmetric kernel for n particles acting on themselves, the first n6 with torques and spins.  Its partials
// are target-major: particle i < n6 has nb pairs (velocity, spin) at 2 nb i, particle i >= n6 nb velocities at
// 2 nb n6 + nb (i - n6).
RpyPlan rpy_plan_sym(int n, int n6, int num_sms);

// The partials of the force-only symmetric kernels are 8 pi (without a wall 8 pi mu) times the velocities; who sums them
// applies this.  Those with torques are velocities and spins, without a wall in lengths of a power of two near a radius far from 1
// (rpy_set_product scales back); neither holds the self blocks.
constexpr double kPairScale = 1.0 / (8.0 * 3.14159265358979323846);

// The full product of one particle set on itself through the symmetric kernel: segments [0, n_seg) (with torques and
// spins when seg_dof is 6) followed by blobs, the wall or equal radii `a`.  Velocities into v_segs [6 n_seg] (spins zero
// for seg_dof 3) and v_blobs [3 (n - n_seg)].
struct RpySetDesc {
    int wall, seg_dof, n_seg, n;
    const float4 *x, *f, *t;  // [n], [n], [n_seg]
    float a, mu;
};
// Whether that is the faster way for n particles, n6 of them with torques, and its partials stay bounded.
bool rpy_set_symmetric(int n, int n6);
int rpy_set_product(const RpySetDesc &d, float4 *scratch, size_t scratch_cap, float *v_segs, float *v_blobs, int num_sms,
                    cudaStream_t st);
// The plan rpy_block_product uses for d (symmetric when d allows it).
RpyPlan rpy_plan_for(const RpyBlockDesc &d, int num_sms);

// Configures the tile-kernel instantiation used by (d, plan) so that later
// launches may be captured into a CUDA graph.
int rpy_prepare(const RpyBlockDesc &d, const RpyPlan &plan);

// Launches the tile kernel; partials land in `scratch`.
int rpy_launch_tiles(const RpyBlockDesc &d, const RpyPlan &plan, float4 *scratch, int *dev_err,
                     cudaStream_t st);

// Batched symmetric wall products (segments on segments, 3x3) of B independent
// particle sets stored back to back.  Per array b: particles [seg0[b], seg0[b]+n[b])
// of x/f, nb[b] = ceil(n[b]/32) tiles, partials at partial + poff[b] laid out
// slot-major, [tile * n[b] + i], and rpy_sym_items(nb[b], packed) work items [item0[b], item0[b+1]) (item0[B] == items).
struct SymBatchParams {
    const float4 *x;
    const float4 *f;
    float4 *partial;
    const int *seg0, *n, *nb;
    const long long *poff, *item0;
    const int *active;  // may be null: every array active
    int B;
    bool packed;        // what the items are (rpy_sym_items)
    long long items;
};
int rpy_launch_sym_batch(const SymBatchParams &p, int grid, cudaStream_t st);
// Work items of a force-only set of nb tiles: 32 targets x 64 sources in packed arithmetic, or pairs of tiles.
__host__ __device__ constexpr long long rpy_sym_items(int nb, bool packed) {
    return packed ? static_cast<long long>((nb + 1) / 2) * ((nb + 1) / 2 + 1) : static_cast<long long>(nb) * (nb + 1) / 2;
}
// Whether a launch over that many pairs of tiles takes the packed units.  Below about thirteen an SM the SMs are not full
// and the launch lasts as long as one unit, which a pair of tiles, half the work, makes shorter; the results are the same
// bit for bit.  A step by pairs and packed, us: one array of 4 cilia (6 pairs) 209 and 217, of 30 (190) 226 and 236, of 48
// (465) 231 and 240, 100 arrays of 6 (1,000) 347 and 362, 8 of 30 (1,520) 258 and 264; one of 100 (2,016) 244 and 241, 4 of
// 64 (3,280) 279 and 264.
constexpr bool rpy_sym_packed(long long tile_pairs, int num_sms) { return tile_pairs > 13LL * num_sms; }

// Output modes of the reduction.
enum RpyOut : int { kOutWrite = 0, kOutAdd = 1 };

// Reduces partials into out_f[i*stride + c] (float) for c < vd; components
// vd..stride-1 are zeroed in write mode (the reference writes all six
// entries of a segment velocity, cuda_functions.cu:460-469).
// With dev_err given, every output of the launch is a quiet NaN when that
// word is non-zero (a tile block gave up waiting for its sources).  A symmetric
// plan is refused: its partials have other factors and lack the self blocks
// (kPairScale); rpy_set_product sums them, or a kernel of the caller's.
int rpy_launch_reduce_f32(const RpyBlockDesc &d, const RpyPlan &plan, const float4 *scratch, float *out_f,
                          int stride, int mode, cudaStream_t st, const int *dev_err = nullptr);

// Tries of the tile kernel's first bounded wait for its staged sources
// (cf_set_wait_limit); the default is the full limit.
unsigned rpy_wait_limit();

// The full product of a small set of force-only particles (the wall, or equal radii) in one launch, straight from and to
// the reference's layouts: segments x [3 n_seg], f [6 n_seg], v [6 n_seg] (spins zero), blobs x, f, v [3 n_blob].
// It leaves the set's float4 records in x and force, as pack_sets_to_float4 does.
constexpr int kRpyDirectMax = 1280;  // largest n_seg + n_blob (see rpy_kernels.cu)
int rpy_direct_product(int wall, const float *x_segs, const float *f_segs, const float *x_blobs, const float *f_blobs,
                       int n_seg, int n_blob, float a, float mu, float *v_segs, float *v_blobs, float4 *x, float4 *force,
                       cudaStream_t st);

// Packing helpers between the reference's AoS host layouts and float4 arrays.
int pack_xyz_to_float4(const float *aos3, float4 *out, int n, cudaStream_t st);
int pack_ft6_to_float4(const float *aos6, float4 *force, float4 *torque, int n, cudaStream_t st);
// Both of the above for one particle set (positions [3n], forces + torques [6n]) in one launch.
int pack_set_to_float4(const float *aos3, const float *aos6, float4 *x, float4 *force, float4 *torque, int n,
                       cudaStream_t st);

// Segments then blobs (either may be empty) from the reference's layouts into consecutive float4 records, in one launch.
int pack_sets_to_float4(const float *x_segs, const float *f_segs, const float *x_blobs, const float *f_blobs, int n_seg,
                        int n_blob, float4 *x, float4 *force, float4 *torque, cudaStream_t st);

// Full product V_t (=|+=) M F_s with the right staging; convenience wrapper.
int rpy_block_product(const RpyBlockDesc &d, float4 *scratch, size_t scratch_cap, int *dev_err, float *out_f,
                      int stride, int mode, int num_sms, cudaStream_t st);

}  // namespace cufil
