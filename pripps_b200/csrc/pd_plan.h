// Host planner: turns a pd_request into the device layout and tile list.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "pd_common.h"
#include "pripps_debye.h"

namespace pd {

// At most this many (species, hydration weight) classes use the one-
// accumulator class mode; more distinct weights switch to the weighted mode.
constexpr int PD_MAX_CLASSES = 48;
// Lattice sets per request, and the largest squared grid diagonal (bins of
// its pair-count histogram).
constexpr uint32_t PD_MAX_LATTICES = 8;
constexpr int64_t PD_MAX_LATTICE_BINS = int64_t{1} << 24;
// Pair-count tiles: 128 i points × up to 8192 j points.
constexpr int PD_LAT_IBLOCK = 128;
constexpr int PD_LAT_JCHUNK = 8192;

struct Tuning {
    int K = 64;     // q-block length
    int TJ = 2048;  // j atoms per tile
    int NP = 2;     // pairs per thread per pass (FP32 form; 1 for FP64)
};

struct Plan {
    // request shape
    int64_t n_atoms = 0;
    int32_t nq = 0;
    int32_t n_frames = 1;
    int32_t n_species = 0;
    int precision = 0;
    bool has_exc = false, has_hyd = false;
    int mode = PD_MODE_CLASS;
    int nv = 1;  // values per slot entry: 1 (class) or 4 (weighted)
    bool test_expire = false;  // PD_FLAG_TEST_EXPIRED_WAIT
    Tuning tun;
    double qmin = 0, qmax = 0, dq = 0;
    std::vector<double> qv;

    // classes and layout
    int n_cls = 0, n_pairs = 0;
    std::vector<PdClassDev> cls;
    std::vector<PdPairDev> pairs;
    std::vector<int32_t> cls_start;  // padded start of each class region
    int32_t n_pad = 0;
    std::vector<int32_t> perm;    // [n_pad] source atom or -1
    std::vector<int32_t> gvalid;  // [n_pad/32]
    std::vector<int32_t> gclass;  // [n_pad/32] class or -1

    // tiles (execution order) and the deterministic reduction lists
    std::vector<PdJob> jobs;        // all frames
    int64_t jobs_per_frame = 0;
    int64_t slots_per_frame = 0;
    int nqb = 0;
    std::vector<int64_t> lptr;  // [n_pairs * nqb + 1]
    std::vector<int64_t> lidx;  // slot indices within a frame
    PdMomentRule mom{};     // when a frame takes the moment form
    PdReduceShape red{};    // sizes of the slot reduction
    // direction form: atom chunks (longest first), the chunks of each class in
    // chunk order, and the sizes its device arrays are given
    std::vector<PdChunk> chunks;
    std::vector<int32_t> cls_ptr, cls_chunk;
    PdAmpShape amp{};
    double radius_hint = -1.0;  // largest distance from the centroid, < 0: not known
    // Host coordinates whose exact radius makes the direction form the cheaper
    // one: no tiles, slots or lists; the jobs only carry the direction units.
    bool dir_only = false;
    bool no_directions = false;  // given up (drop_directions); a shard's share inherits it
    bool compact = false;        // the least memory (make_compact)
    double dir_work = 0.0;   // FP32 lane operations of a frame's directions
    double dir_cost = 0.0;   // and of its class pairs' products: the form's
    int64_t dir_units = 0;   // its work units
    double job_cost = 0.0;   // relative cost of a job (dir_only)
    double pair_bytes = 0.0; // at least what the tiles' plan would take (dir_only)
    uint32_t rank = 0, world = 1;
    uint64_t pairs_covered = 0; // per frame, unordered pairs over all tiles

    // lattice sets (class mode, one frame): their self pairs are counted per
    // integer squared offset instead of running through the pair tiles
    std::vector<PdLatDev> lat;
    std::vector<PdLatTile> lat_tiles;
    int64_t lat_bins = 0;
};

// Whether every one of n values is finite (no early exit: a few values per cycle).
bool all_finite(const double *x, uint64_t n);

// Validate a request; fills msg and returns a PD_E* code on failure.
int validate_request(const pd_request *req, bool device_pointers, std::string &msg);

// Default shape when no tuned entry exists.
Tuning default_tuning(int64_t n_atoms, int64_t nq, int precision, int64_t n_frames = 1);
// The instantiated kernel shape a requested one runs as in a mode (the q
// block and pairs per thread adjusted where that shape has no kernel).
Tuning fit_tuning(int precision, int mode, Tuning t);

// The moment rule and reduction sizes of a plan whose tiles and lists stand
// (again after a shard cut them).
void set_reduction(Plan &P);

// A rank's share of a plan for a tile-sharded solve: every world-th tile of
// the cost-ordered job list, with only the slots those tiles write (numbered
// in their original order) and the reduction lists cut to them.
int shard_plan(const Plan &full, uint32_t rank, uint32_t world, Plan &out);

// Build the plan from host-side species and weights (hyd may be NULL).
// count_pairs fills Plan::pairs_covered (an O(N · tiles per block) host loop
// that only pd_plan_inspect needs). radius_hint sizes the direction form's arrays: the
// largest distance of an atom from its frame's centroid, or < 0 when the
// coordinates are not known yet (a generous estimate from the atom count).
// With allow_dir_only the hint is the exact radius (a little more is fine), and
// a plan whose frames all take the direction form gets no tiles.
int build_plan(const pd_request *req, const uint32_t *species_host, const double *weights_host,
               const Tuning &tun, Plan &plan, std::string &msg, bool count_pairs = false,
               double radius_hint = -1.0, bool allow_dir_only = false);

// Largest distance of an atom from its frame's centroid (host coordinates), not
// below the same taken with the centroid summed in another order.
double max_radius(const double *xyz, int64_t n_atoms, int64_t n_frames);

// Give up the direction form (a request that only fits without its arrays), also in
// every shard of the plan: the ranks' partial sums are of one form.
void drop_directions(Plan &P);

// The least device memory that the request can run in: pairs, no more moments than
// grid points, every slot list summed by one block.
void make_compact(Plan &P);

}  // namespace pd
