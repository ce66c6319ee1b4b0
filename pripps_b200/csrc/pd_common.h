// Internal types shared by the host planner (pd_plan.cpp) and the device
// kernels (pd_kernels.cu) of libpripps_debye.
//
// Data layout in HBM, per request:
//   * atoms are re-ordered into "classes" (species, or species × hydration
//     weight when few distinct weights exist) and each class is padded to a
//     multiple of PD_GRANULE = 32 atoms, so that every warp-row of 32 i-atoms
//     belongs to one class; padded atoms are inert (gvalid masks them);
//   * coordinates are stored as float4 {x, y, z, w} (FP32 form) or double4
//     (FP64 form), centred on the frame centroid; w carries the per-atom
//     hydration weight in the weighted mode and is unused otherwise;
//   * a tile ("job") is (frame, i-block of PD_IBLOCK atoms, contiguous j range
//     of real atoms of ONE class, q-block of K grid points); it covers the
//     pairs (i, j) with j > i;
//   * the PD_WARPS warps of a tile keep their warp-reduced FP64 partial sums
//     for the K q-points in shared memory; at the end of the tile the warps of
//     one atom class are added in warp order and written to one FP64 slot per
//     distinct class of the i-block (usually one); a second kernel adds the
//     slots of every (class pair, q) in a fixed order, so the result does not
//     depend on which SM ran which tile.
#pragma once

#include <cstdint>

#ifndef __CUDACC__
struct float4 { float x, y, z, w; };
struct double4 { double x, y, z, w; };
#else
#include <cuda_runtime.h>
#endif

constexpr int PD_GRANULE = 32;                    // atoms per warp-row
constexpr int PD_WARPS = 4;                       // warps per tile CTA
constexpr int PD_THREADS = PD_GRANULE * PD_WARPS; // 128 threads
constexpr int PD_IBLOCK = PD_THREADS;             // i-atoms per tile

// Mode of the pair accumulation.
//   PD_MODE_CLASS:    one accumulator, Σ sin(q r)/r per class pair; every
//                     per-atom factor is a per-class constant.
//   PD_MODE_WEIGHTED: two accumulators, Σ sin(q r)/r and Σ w_j sin(q r)/r, for
//                     hydration weights that vary within a species.
enum PdMode : int32_t { PD_MODE_CLASS = 0, PD_MODE_WEIGHTED = 1 };

struct PdJob {
    int32_t req;    // request index within the launch
    int32_t frame;  // frame of the request
    int32_t i0;     // first padded i index (multiple of PD_IBLOCK)
    int32_t j0, j1; // padded j range [j0, j1): real atoms of one class; of a plan without
                    // tiles: the job's ordinal in its frame, and the frame's jobs
    int32_t qb;     // q-block index
    // bits 0..47: first output slot of this tile; bits 48..55: the slot of
    // each warp relative to it, 2 bits per warp (warp w at bits 48 + 2w).
    // Warps of one class share a slot; slot numbers follow the first warp
    // of each class, so warp 0 always has relative slot 0.
    int64_t slot;
};
static_assert(sizeof(PdJob) == 32, "PdJob layout");
constexpr int PD_SLOT_MAP_SHIFT = 48;
constexpr int64_t PD_SLOT_MASK = (int64_t{1} << PD_SLOT_MAP_SHIFT) - 1;

// Bits of the per-request device status word (PdReqDev::status).
constexpr int32_t PD_DEV_WAIT_EXPIRED = 1;  // a bounded wait for a bulk copy gave up

// PdReqDev::flags
constexpr int32_t PD_REQF_TEST_EXPIRE = 1;  // test hook: the launch's first tile skips its copy

// Per-frame constants, written on the device once the frame's radius is known.
//
// n_grp > 0: the frame runs in the direction form (amplitudes over a
// quadrature of the sphere, pd_moments.cuh). Its work units are (atom chunk,
// moment block, group of 32 directions); the request's jobs share them by
// ordinal.
//
// Else n_mom > 0: moment form of the pairs. Every pair's sinc(q r) is expanded in
// cos(n φ), sin(φ/2) = r/d, n < n_mom, and the tiles sum the moments instead of the
// grid points. A tile's nqb jobs are then n_mblk moment blocks times n_parts
// parts of its j range (job qb: block qb mod n_mblk, part qb / n_mblk; the jobs
// past n_mblk·n_parts are idle).
//
// Else the grid points are summed directly.
struct PdFrameDev {
    double radius;   // largest atom distance from the centroid (Å)
    double d;        // pairs: expansion length, a little over 2·radius (Å)
    double inv_d2;   // 1/d²
    double r1;       // directions: expansion length, a little over the radius (Å)
    int32_t n_mom;   // moments, a multiple of 8; 0: no moment form
    int32_t n_mblk;  // moment blocks of pd_moment_block(K) moments
    int32_t n_parts;
    int32_t n_grp;   // this rank's groups of 32 directions; 0: no direction form
    int32_t n_amp;   // moments of the direction form, a multiple of 8
    int32_t n_node;  // values of q that the class-pair sums are formed at (direction form):
                     // Chebyshev nodes of the q range, or (FP64) the grid points
    int32_t pad_[2];
};
static_assert(sizeof(PdFrameDev) == 64, "PdFrameDev layout");

// Atoms [j0, j1) (padded indices) of one class: a work unit of the direction form.
struct PdChunk {
    int32_t cls, j0, j1, pad_;
};

// Moments per job of a kernel shape with q-block K: at most K (they share its
// slots) and what the accumulators of the shape's register budget hold.
constexpr int pd_moment_block(int K) {
    return K >= 128 ? 128 : (K >= 64 ? 64 : 32);
}
// The moment form is bounded to this many moments (q_max·d up to about 900).
constexpr int PD_MAX_MOMENTS = 512;

// The direction form: at most this many moments (q_max·radius up to about 220),
// and the shared memory of the kernel that sums the class pairs.
constexpr int PD_MAX_DIR_MOMENTS = 256;
constexpr int PD_DIR_SMEM = 200 * 1024;
// Nodes of directions that the class pairs' products are charged at least: with fewer the
// kernel that forms them has SMs to spare.
constexpr double PD_DIR_LEAST = 12000.0;
// Atoms that a chunk of the FP64 form is charged for: a block's 128 threads take an atom
// each and add up their moments, whatever the chunk holds (per direction, 19 to 3,345
// atoms in 1 to 60 chunks: as long as n_atoms + 80 to 116 per chunk).
constexpr double PD_DIR_CHUNK64 = 130.0;
constexpr int PD_DIR_DIRS = 8;  // directions of a work unit
// Moments of its first block (FP32, FP64) and of each later one.
constexpr int PD_DIR_MBLOCK = 128, PD_DIR_MBLOCK64 = 64;

// When a frame may run in the moment form (block = 0, the FP64 form: never).
struct PdMomentRule {
    double qmax;          // last grid point
    int32_t block;        // moments per job, pd_moment_block(K)
    int32_t nqb;          // jobs per tile
    int32_t max_moments;  // more do not fit
    int32_t fp64;
    // Cost of a pair: all grid points, the moment form per moment and per block (the
    // cheaper one sums the pairs), and the grid points in the directions' unit.
    double grid_cost, mom_cost, mom_block_cost, grid_dir_cost;
    // What is charged beyond the pairs: their tiles, at the grid points a thread's chain of
    // atoms, with moments the longer chain of short kernels; and for each node of a direction the products of the class pairs.
    double tile_cost, grid_latency, mom_latency, dir_pair_cost;
    // direction form (dir_cap = 0: never)
    int32_t dir_block;    // moments per unit
    int32_t dir_cap;      // directions the frame's table holds (a multiple of 32)
    int32_t grp_cap;      // direction groups of this rank that the sums hold
    int32_t amp_cap;      // moments
    int32_t node_cap;     // Chebyshev nodes, or (FP64) the grid points
    int32_t n_chunk, n_cls, nv2;  // nv2: 1, or 2 with sums weighted by w (weighted mode)
    int32_t rank, world;
    int64_t slot_cap;     // doubles per frame for the chunks' sums
    int64_t n_atoms;
    double n_tile_pairs;  // pairs of a frame that the tiles sum (not a lattice set's own)
    int32_t nq;
    int32_t dir_only;     // the plan has no tiles: every frame takes the direction form
};

// Sizes the direction kernels share.
struct PdAmpShape {
    int32_t n_chunk, n_cls, nv2, nq;
    int32_t dir_cap, grp_cap, amp_cap, node_cap;
    int32_t node_tile;  // nodes per block of the sums' kernel (a multiple of 4)
    int32_t sum_smem;   // its shared memory in doubles
    int32_t rank, world, dir_block;
    int64_t slot_cap;
};

// Sizes of the slot reduction and the profile kernel.
struct PdReduceShape {
    int32_t n_pairs, nq, K, nqb;
    int32_t block;        // moments per job
    int32_t width;        // row length of the sums: grid points or moments
    int32_t n_z;          // 128-value blocks per row
    int32_t n_chunk;      // blocks that share a slot list
    int32_t max_moments;  // moments or nodes
    int32_t node_cap;     // nodes or grid points (direction form)
    int32_t dir_only;     // no tiles (a frame without directions has no result: NaN)
    int32_t fp64;         // directions are summed at the grid points, not at nodes
    int64_t slots_per_frame;
};

// Per-request descriptor read by the pair kernels.
struct PdReqDev {
    const float4 *atoms32;    // [n_frames][n_pad] (FP32 form)
    const double4 *atoms64;   // [n_frames][n_pad] (FP64 form)
    const int32_t *gvalid;    // [n_pad / 32] valid atoms per granule
    const double *qv;         // [nq] grid (FP64 form reads it directly)
    double *slots;            // [n_slots][nv][K]
    double *dir_slots;        // [n_frames][slot_cap] (direction form)
    const PdFrameDev *frames; // [n_frames]
    const double4 *dirs;      // [n_frames][dir_cap] direction/(2·r1) and quadrature weight
    const PdChunk *chunks;    // [n_chunk]
    int32_t *status;          // PD_DEV_* bits, OR-ed in by the pair kernel
    double qmin, dq;          // grid origin and step
    int32_t n_pad;
    int32_t nq;
    int32_t K;
    int32_t mode;
    int32_t flags;            // PD_REQF_* bits
    int32_t pad_;
    PdAmpShape amp;
};

// Per-class constants for the combine kernel.
struct PdClassDev {
    int32_t species;
    int32_t lat;   // lattice set whose pair counts give the class's self pair sum, or -1
    double n;   // atoms in the class
    double w;   // hydration weight (class mode)
    double w1;  // Σ w_i over the class (weighted mode)
    double w2;  // Σ w_i² over the class (weighted mode)
};

// Per-class-pair constants: classes (a <= b) and the q = 0 pair sums
// (sinc = 1 for every pair): count, Σ w_i, Σ w_j, Σ w_i w_j.
struct PdPairDev {
    int32_t a, b;
    double q0[4];
};

// A lattice set of one class: its points are origin + spacing·(i, j, k); the
// class's self pair sums come from the exact pair count per integer squared
// offset n = |Δ(i, j, k)|², hist[hist_off + n], n < n_bins.
struct PdLatDev {
    double origin[3];
    double spacing;
    int32_t ext[3];
    int32_t cls;       // class index
    int32_t start;     // padded index of the class's first point
    int32_t n;         // points of the class
    int32_t pair;      // class-pair index (cls, cls)
    int32_t n_bins;    // max n + 1
    int64_t hist_off;  // first bin in the histogram array
};

// One CTA of the pair-count kernel: lattice `lat`, i points [i0, i0 + 128)
// of the class (relative to its start), j points [j0, j1), pairs with j > i.
struct PdLatTile {
    int32_t lat, i0, j0, j1;
};
static_assert(sizeof(PdLatTile) == 16, "PdLatTile layout");

// Direct transform at lattice vectors on lines: a segment of consecutive vectors
// n0 + j·δ. The members are entries of a point's phase table (the distinct |indices| of
// each axis): those of the start n0 and of the step δ; the sign bit is set where
// the index is negative.
struct PdLine {
    int32_t x, y, z, sx, sy, sz;
};
