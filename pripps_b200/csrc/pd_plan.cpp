// Host planner of the Debye backend: classes, padded layout, tiles and the
// fixed-order reduction lists (see pd_common.h for the layout).
#include "pd_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <utility>

#include "pd_kernels.h"
#include "pd_tuning.h"

namespace pd {

__attribute__((optimize("O3"))) bool all_finite(const double *x, uint64_t n) {
    // 0·x is 0 for finite x and NaN otherwise; eight independent sums
    double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint64_t i = 0;
    for (; i + 8 <= n; i += 8)
        for (int k = 0; k < 8; ++k) s[k] += 0.0 * x[i + k];
    for (; i < n; ++i) s[0] += 0.0 * x[i];
    for (int k = 1; k < 8; ++k) s[0] += s[k];
    return s[0] == 0.0;
}

__attribute__((optimize("O3"))) static uint32_t max_species(const uint32_t *x, uint64_t n) {
    uint32_t m = 0;
    for (uint64_t i = 0; i < n; ++i) m = m > x[i] ? m : x[i];
    return m;
}

int validate_request(const pd_request *req, bool device_pointers, std::string &msg) {
    if (!req) {
        msg = "request is NULL";
        return PD_EINVAL;
    }
    if (req->n_atoms == 0) {
        msg = "n_atoms must be >= 1";
        return PD_EINVAL;
    }
    if (req->n_atoms > (1ull << 30)) {
        msg = "n_atoms exceeds 2^30";
        return PD_EINVAL;
    }
    if (req->nq == 0 || req->nq > (1ull << 24)) {
        msg = "nq must be in [1, 2^24]";
        return PD_EINVAL;
    }
    if (req->n_species == 0) {
        msg = "n_species must be >= 1";
        return PD_EINVAL;
    }
    if (req->precision != PD_FP32_FP64RED && req->precision != PD_FP64) {
        msg = "precision must be PD_FP32_FP64RED or PD_FP64";
        return PD_EINVAL;
    }
    if (!req->xyz || !req->species || !req->ff_atoms) {
        msg = "xyz, species and ff_atoms are required";
        return PD_EINVAL;
    }
    if (req->hyd_weights && !req->ff_water) {
        msg = "ff_water is required when hyd_weights is given";
        return PD_EINVAL;
    }
    if ((req->flags & ~PD_FLAG_TEST_EXPIRED_WAIT) != 0) {
        msg = "flags must be 0 (or PD_FLAG_TEST_EXPIRED_WAIT)";
        return PD_EINVAL;
    }
    if (req->n_lattices > PD_MAX_LATTICES || (req->n_lattices && !req->lattices)) {
        msg = "n_lattices must be <= " + std::to_string(PD_MAX_LATTICES) +
              " with a lattices array";
        return PD_EINVAL;
    }
    for (uint32_t l = 0; l < req->n_lattices; ++l) {
        const pd_lattice &L = req->lattices[l];
        if (L.species >= req->n_species || L.reserved || L.reserved2 ||
            !(std::isfinite(L.spacing) && L.spacing > 0.0) || !std::isfinite(L.origin[0]) ||
            !std::isfinite(L.origin[1]) || !std::isfinite(L.origin[2]) || L.extent[0] < 1 ||
            L.extent[1] < 1 || L.extent[2] < 1 || L.extent[0] > (1u << 16) ||
            L.extent[1] > (1u << 16) || L.extent[2] > (1u << 16)) {
            msg = "lattice " + std::to_string(l) +
                  ": species < n_species, spacing > 0, finite origin, extents in [1, 65536] "
                  "and zero reserved fields required";
            return PD_EINVAL;
        }
        const double e0 = L.extent[0] - 1.0, e1 = L.extent[1] - 1.0, e2 = L.extent[2] - 1.0;
        if (e0 * e0 + e1 * e1 + e2 * e2 >= static_cast<double>(PD_MAX_LATTICE_BINS)) {
            msg = "lattice " + std::to_string(l) + " is too large: its squared diagonal exceeds " +
                  std::to_string(PD_MAX_LATTICE_BINS) + " grid steps²";
            return PD_EINVAL;
        }
        for (uint32_t m = 0; m < l; ++m)
            if (req->lattices[m].species == L.species) {
                msg = "two lattices name species " + std::to_string(L.species);
                return PD_EINVAL;
            }
    }
    if (req->n_lattices && req->n_frames > 1) {
        msg = "lattice sets need a single frame";
        return PD_EINVAL;
    }
    if (!std::isfinite(req->qmin) || !std::isfinite(req->qmax) || req->qmin < 0.0 ||
        req->qmax < req->qmin) {
        msg = "q range must satisfy 0 <= qmin <= qmax (finite)";
        return PD_EINVAL;
    }
    const uint64_t nf = req->n_frames ? req->n_frames : 1;
    if (nf > (1u << 20)) {
        msg = "n_frames exceeds 2^20";
        return PD_EINVAL;
    }
    if (device_pointers) return PD_OK;
    // Host buffers: check the values the planner and the kernels rely on.
    const uint64_t n = req->n_atoms;
    // (whole-array scans first; the loops only name the offending entry)
    if (max_species(req->species, n) >= req->n_species) {
        uint64_t i = 0;
        while (req->species[i] < req->n_species) ++i;
        msg = "species id " + std::to_string(req->species[i]) + " at atom " + std::to_string(i) +
              " is >= n_species";
        return PD_EINVAL;
    }
    if (!all_finite(req->xyz, n * 3 * nf)) {
        uint64_t i = 0;
        while (std::isfinite(req->xyz[i])) ++i;
        msg = "non-finite coordinate at index " + std::to_string(i);
        return PD_EINVAL;
    }
    const uint64_t nt = static_cast<uint64_t>(req->n_species) * req->nq;
    if (!all_finite(req->ff_atoms, nt) ||
        (req->ff_excluded && !all_finite(req->ff_excluded, nt))) {
        msg = "non-finite form-factor table entry";
        return PD_EINVAL;
    }
    if (req->hyd_weights) {
        if (!all_finite(req->hyd_weights, n)) {
            msg = "non-finite hydration weight";
            return PD_EINVAL;
        }
        if (!all_finite(req->ff_water, req->nq)) {
            msg = "non-finite water form factor";
            return PD_EINVAL;
        }
    }
    if (req->frame_weights) {
        double s = 0.0;
        for (uint64_t f = 0; f < nf; ++f) {
            if (!std::isfinite(req->frame_weights[f])) {
                msg = "non-finite frame weight";
                return PD_EINVAL;
            }
            s += req->frame_weights[f];
        }
        // trajectory_average rejects a sum that is zero or not normal
        // (src/trajectory.rs:234-238).
        if (!std::isnormal(std::fabs(s))) {
            msg = "frame weights sum to zero or a non-normal value; cannot normalize";
            return PD_EINVAL;
        }
    }
    return PD_OK;
}

static int next_pow2(int64_t v) {
    int p = 1;
    while (p < v && p < (1 << 30)) p <<= 1;
    return p;
}

Tuning fit_tuning(int precision, int mode, Tuning t) {
    // Two accumulators per q (weighted mode) allow q blocks up to 64 (there
    // four pairs per thread measured fastest: at the grid points, 814 ms on 100,000
    // atoms with per-atom hydration weights against 835 ms with two); FP64 runs
    // one pair per pass.
    if (precision == PD_FP64) {
        t.NP = 1;
    } else if (!valid_shape(precision, mode, t.K, t.NP)) {
        if (mode == PD_MODE_WEIGHTED) {
            t.K = t.K > 32 ? 64 : 32;
            t.NP = t.K == 64 ? 4 : 2;
        } else {
            t.NP = t.K == 32 ? 4 : 2;
        }
    }
    return t;
}

Tuning default_tuning(int64_t n_atoms, int64_t nq, int precision, int64_t n_frames) {
    Tuning t;
    if (precision == PD_FP64) {
        t.K = 32;
        t.NP = 1;
        t.TJ = std::clamp(next_pow2(n_atoms / 16), 256, 4096);
        return t;
    }
    // Measured on B200 with the grid points summed one by one (class mode; structures
    // of these sizes that are not long sum directions, which have no such shape): K = 128
    // with 4 pairs per thread (three CTAs per SM, seeds computed at the top of each
    // pass) is the fastest shape from ~4k atoms up — 100,000 atoms 546.7 ms against
    // 561.5 ms with 2 pairs — and K = 64 with 4 pairs below; a j chunk of about N/8
    // atoms balances tile count against per-tile overhead. The last q-block of a grid
    // runs only the 16-point chunks that lie on it, so a long block wastes at most
    // 15 grid points per request. (These are the shapes of buckets the tuning
    // table does not name.)
    if (n_atoms < 4000) {
        t.K = 64;
        t.NP = 4;
    } else {
        t.K = 128;
        t.NP = 4;
    }
    if (nq <= 32) {
        t.K = 32;
        t.NP = 4;
    }
    // j chunk: about N/8 atoms, halved while a solve would have fewer than
    // ~6 tiles per resident CTA of a B200 (148 SMs × 3): the longest-first
    // tile order then ends with short tiles on every SM. Measured at the grid points
    // (pair kernel + slot reduction): 10,000 atoms, nq 500: 3.82 / 3.51 /
    // 3.54 / 3.74 ms at 2,048 / 1,024 / 512 / 256; 20,000 atoms, nq 512:
    // 13.24 / 12.78 / 12.89 ms at 4,096 / 2,048 / 1,024; 100,000 atoms, nq
    // 1,000: 589.5 / 592.5 ms at 16,384 / 4,096.
    t.TJ = std::clamp(next_pow2(n_atoms / 8), 256, 16384);
    const double iblocks = static_cast<double>((n_atoms + 127) / 128);
    const double nqb = static_cast<double>((nq + t.K - 1) / t.K);
    const double frames = static_cast<double>(std::max<int64_t>(n_frames, 1));
    while (t.TJ > 256 &&
           iblocks * std::ceil(static_cast<double>(n_atoms) / t.TJ) * 0.5 * nqb * frames <
               6.0 * 148 * 3)
        t.TJ /= 2;
    return t;
}

// Index of a (species, weight) key among at most max_keys distinct ones in
// first-seen order, or -1 for one too many: a table of 256 places, probed from
// a multiplicative hash (at most 48 keys, so a probe rarely steps on). Equality
// of the weights as numbers: adding +0 gives both zeros one bit pattern.
struct KeySet {
    std::vector<std::pair<uint32_t, double>> seen;
    int16_t at[256];
    int max_keys;
    explicit KeySet(int max) : max_keys(max) {
        static_assert(PD_MAX_CLASSES < 128, "places of the key table");
        std::fill(at, at + 256, int16_t{-1});
        seen.reserve(max);
    }
    int find(uint32_t species, double w) {
        const double z = w + 0.0;
        uint64_t bits;
        std::memcpy(&bits, &z, 8);
        uint64_t h = ((bits ^ (uint64_t{species} << 32) ^ species) * 0x9E3779B97F4A7C15ull) >> 56;
        for (;; h = (h + 1) & 255) {
            const int k = at[h];
            if (k < 0) break;
            if (seen[k].first == species && seen[k].second == w) return k;
        }
        if (static_cast<int>(seen.size()) == max_keys) return -1;
        at[h] = static_cast<int16_t>(seen.size());
        seen.emplace_back(species, w);
        return at[h];
    }
};

int request_mode(const pd_request *req, const uint32_t *species, const double *weights) {
    if (!req->hyd_weights || !weights) return PD_MODE_CLASS;
    KeySet keys(PD_MAX_CLASSES);
    for (uint64_t i = 0; i < req->n_atoms; ++i)
        if (keys.find(species[i], weights[i]) < 0) return PD_MODE_WEIGHTED;
    return PD_MODE_CLASS;
}

// The distinct (species, weight) keys of the atoms in ascending order and
// each atom's index among them; false as soon as there are more than
// max_keys. Weights are finite (validated), so equality is the map order's
// equivalence.
static bool weight_class_keys(int64_t n, const uint32_t *species, const double *w,
                              int max_keys, std::vector<std::pair<uint32_t, double>> &keys,
                              std::vector<int32_t> &atom_key) {
    KeySet set(max_keys);
    for (int64_t i = 0; i < n; ++i) {
        const int k = set.find(species[i], w[i]);
        if (k < 0) return false;
        atom_key[i] = k;
    }
    const auto &seen = set.seen;
    std::vector<int32_t> order(seen.size()), rank(seen.size());
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return seen[a] < seen[b]; });
    keys.resize(seen.size());
    for (size_t r = 0; r < order.size(); ++r) {
        rank[order[r]] = static_cast<int32_t>(r);
        keys[r] = seen[order[r]];
    }
    for (int64_t i = 0; i < n; ++i) atom_key[i] = rank[atom_key[i]];
    return true;
}

// One key per species present (weight 0), in ascending species order.
static void species_class_keys(int64_t n, const uint32_t *species, int32_t n_species,
                               std::vector<std::pair<uint32_t, double>> &keys,
                               std::vector<int32_t> &atom_key) {
    std::vector<int32_t> rank(n_species, -1);
    for (int64_t i = 0; i < n; ++i) rank[species[i]] = 0;
    keys.clear();
    for (int32_t sp = 0; sp < n_species; ++sp)
        if (rank[sp] >= 0) {
            rank[sp] = static_cast<int32_t>(keys.size());
            keys.emplace_back(static_cast<uint32_t>(sp), 0.0);
        }
    for (int64_t i = 0; i < n; ++i) atom_key[i] = rank[species[i]];
}

static bool direction_only(Plan &P);
static void set_chunks(Plan &P);

int build_plan(const pd_request *req, const uint32_t *species, const double *w,
               const Tuning &tun, Plan &P, std::string &msg, bool count_pairs,
               double radius_hint, bool allow_dir_only) {
    P = Plan();
    P.radius_hint = radius_hint;
    P.n_atoms = static_cast<int64_t>(req->n_atoms);
    P.nq = static_cast<int32_t>(req->nq);
    P.n_frames = static_cast<int32_t>(req->n_frames ? req->n_frames : 1);
    P.n_species = static_cast<int32_t>(req->n_species);
    P.precision = static_cast<int>(req->precision);
    P.has_exc = req->ff_excluded != nullptr;
    P.has_hyd = req->hyd_weights != nullptr;
    P.test_expire = (req->flags & PD_FLAG_TEST_EXPIRED_WAIT) != 0;
    P.tun = tun;
    if (!valid_q_block(P.precision, tun.K) || tun.TJ < 32 || tun.TJ % 32 != 0 ||
        tun.NP < 1 || tun.NP > 4) {
        msg = "invalid tuning (q block " + std::to_string(tun.K) + ", j chunk " +
              std::to_string(tun.TJ) + ")";
        return PD_EINVAL;
    }
    P.qmin = req->qmin;
    P.qmax = req->qmax;
    // Grid exactly as linear_q_values (src/q_sampler.rs:24-29).
    const double denom = static_cast<double>(P.nq > 1 ? P.nq - 1 : 1);
    P.qv.resize(P.nq);
    for (int k = 0; k < P.nq; ++k)
        P.qv[k] = P.qmin + (P.qmax - P.qmin) * static_cast<double>(k) / denom;
    P.dq = (P.qmax - P.qmin) / denom;

    const int64_t n = P.n_atoms;
    // ---- classes: species, or (species, weight) while few distinct weights;
    // numbered in ascending (species, weight) order
    std::vector<std::pair<uint32_t, double>> keys;
    std::vector<int32_t> atom_cls(n);
    const bool by_weight =
        P.has_hyd && weight_class_keys(n, species, w, PD_MAX_CLASSES, keys, atom_cls);
    if (!by_weight) species_class_keys(n, species, P.n_species, keys, atom_cls);
    P.mode = (P.has_hyd && !by_weight) ? PD_MODE_WEIGHTED : PD_MODE_CLASS;
    P.nv = P.mode == PD_MODE_WEIGHTED ? 4 : 1;
    P.tun = fit_tuning(P.precision, P.mode, P.tun);
    const int c = static_cast<int>(keys.size());
    P.n_cls = c;
    P.cls.assign(c, PdClassDev{});
    for (int ci = 0; ci < c; ++ci) {
        P.cls[ci].species = static_cast<int32_t>(keys[ci].first);
        P.cls[ci].w = keys[ci].second;
    }
    // ---- lattice sets: one class each, class mode only
    std::vector<int> lat_of_cls(c, -1);
    P.lat.clear();
    for (uint32_t l = 0; l < req->n_lattices; ++l) {
        const pd_lattice &L = req->lattices[l];
        int found = -1, count = 0;
        for (int k = 0; k < c; ++k)
            if (P.cls[k].species == static_cast<int32_t>(L.species)) {
                found = k;
                ++count;
            }
        if (count == 0) continue;  // no point of the species: nothing to sum
        if (count > 1 || P.mode != PD_MODE_CLASS) {
            msg = "the points of lattice species " + std::to_string(L.species) +
                  " must share one hydration weight (and the request have at most " +
                  std::to_string(PD_MAX_CLASSES) + " species × weight classes)";
            return PD_EINVAL;
        }
        PdLatDev d{};
        for (int a = 0; a < 3; ++a) {
            d.origin[a] = L.origin[a];
            d.ext[a] = static_cast<int32_t>(L.extent[a]);
        }
        d.spacing = L.spacing;
        d.cls = found;
        const int64_t e0 = L.extent[0] - 1, e1 = L.extent[1] - 1, e2 = L.extent[2] - 1;
        d.n_bins = static_cast<int32_t>(e0 * e0 + e1 * e1 + e2 * e2 + 1);
        lat_of_cls[found] = static_cast<int>(P.lat.size());
        P.lat.push_back(d);
    }
    std::vector<int64_t> count(c, 0);
    for (int64_t i = 0; i < n; ++i) ++count[atom_cls[i]];
    // ---- padded layout
    P.cls_start.assign(c, 0);
    int64_t cur = 0;
    for (int k = 0; k < c; ++k) {
        P.cls_start[k] = static_cast<int32_t>(cur);
        const int64_t nk = count[k];
        cur += (nk + PD_GRANULE - 1) / PD_GRANULE * PD_GRANULE;
    }
    cur = (cur + PD_IBLOCK - 1) / PD_IBLOCK * PD_IBLOCK;
    if (cur > (int64_t{1} << 31) - PD_IBLOCK) {
        msg = "padded atom count overflows";
        return PD_EINVAL;
    }
    P.n_pad = static_cast<int32_t>(cur);
    P.perm.assign(P.n_pad, -1);
    const int ng = P.n_pad / PD_GRANULE;
    P.gvalid.assign(ng, 0);
    P.gclass.assign(ng, -1);
    {
        std::vector<int32_t> next(P.cls_start);
        for (int64_t i = 0; i < n; ++i)
            P.perm[next[atom_cls[i]]++] = static_cast<int32_t>(i);
    }
    for (int k = 0; k < c; ++k) {
        const int64_t nk = count[k];
        double s1 = 0, s2 = 0;
        if (P.has_hyd)
            for (int64_t r = 0; r < nk; ++r) {
                const double wr = w[P.perm[P.cls_start[k] + r]];
                s1 += wr;
                s2 += wr * wr;
            }
        P.cls[k].lat = lat_of_cls[k];
        P.cls[k].n = static_cast<double>(nk);
        P.cls[k].w1 = s1;
        P.cls[k].w2 = s2;
        for (int64_t g = 0; g < (nk + PD_GRANULE - 1) / PD_GRANULE; ++g) {
            const int gi = P.cls_start[k] / PD_GRANULE + static_cast<int>(g);
            P.gclass[gi] = k;
            P.gvalid[gi] = static_cast<int32_t>(std::min<int64_t>(PD_GRANULE, nk - g * PD_GRANULE));
        }
    }
    // ---- class pairs (a <= b) and their exact q = 0 sums
    std::vector<int> pair_index(static_cast<size_t>(c) * c, -1);
    for (int a = 0; a < c; ++a)
        for (int b = a; b < c; ++b) {
            PdPairDev pd{};
            pd.a = a;
            pd.b = b;
            const double na = P.cls[a].n, nb = P.cls[b].n;
            if (a != b) {
                pd.q0[0] = na * nb;
                pd.q0[1] = P.cls[a].w1 * nb;
                pd.q0[2] = na * P.cls[b].w1;
                pd.q0[3] = P.cls[a].w1 * P.cls[b].w1;
            } else {
                pd.q0[0] = na * (na - 1.0) / 2.0;
                // Σ_{i<j} w_i and Σ_{i<j} w_j in padded order within the class.
                double ti = 0, tj = 0, tij = 0, pre = 0;
                const int64_t nk = P.has_hyd ? count[a] : 0;
                for (int64_t r = 0; r < nk; ++r) {
                    const double wr = w[P.perm[P.cls_start[a] + r]];
                    ti += wr * static_cast<double>(nk - 1 - r);
                    tj += wr * static_cast<double>(r);
                    tij += wr * pre;
                    pre += wr;
                }
                pd.q0[1] = ti;
                pd.q0[2] = tj;
                pd.q0[3] = tij;
            }
            pair_index[a * c + b] = static_cast<int>(P.pairs.size());
            P.pairs.push_back(pd);
        }
    P.n_pairs = static_cast<int>(P.pairs.size());
    // lattice layout: class range, self pair, histogram bins, count tiles
    {
        int64_t off = 0;
        for (size_t l = 0; l < P.lat.size(); ++l) {
            PdLatDev &d = P.lat[l];
            d.start = P.cls_start[d.cls];
            d.n = static_cast<int32_t>(P.cls[d.cls].n);
            d.pair = pair_index[d.cls * c + d.cls];
            d.hist_off = off;
            off += d.n_bins;
        }
        P.lat_bins = off;
    }

    // ---- pair-count tiles of the lattice sets
    P.lat_tiles.clear();
    for (size_t l = 0; l < P.lat.size(); ++l) {
        const PdLatDev &d = P.lat[l];
        // j chunks that give every SM a few tiles where the set is small (a thread counts
        // its chunk one after the other: 7,200 points in chunks of 8,192 points 400 us)
        const int64_t even = static_cast<int64_t>(d.n) * d.n / (2 * PD_LAT_IBLOCK * 592);
        const int32_t chunk = static_cast<int32_t>(
            std::clamp<int64_t>((even + 255) & ~int64_t{255}, 256, PD_LAT_JCHUNK));
        for (int32_t i0 = 0; i0 < d.n; i0 += PD_LAT_IBLOCK)
            for (int32_t j0 = i0; j0 < d.n; j0 += chunk)
                if (std::min(d.n, j0 + chunk) - 1 > i0)
                    P.lat_tiles.push_back(
                        PdLatTile{static_cast<int32_t>(l), i0, j0, std::min(d.n, j0 + chunk)});
    }

    set_chunks(P);
    const int K = P.tun.K, TJ = P.tun.TJ;
    P.nqb = (P.nq + K - 1) / K;
    if (allow_dir_only && radius_hint >= 0.0 && direction_only(P)) return PD_OK;

    // ---- tiles of one frame, in creation order
    struct Tile {
        int32_t i0, j0, j1, cls;
    };
    std::vector<Tile> tiles;
    const int nblocks = P.n_pad / PD_IBLOCK;
    for (int ib = 0; ib < nblocks; ++ib) {
        const int32_t i0 = ib * PD_IBLOCK;
        int min_cls = -1;
        for (int wv = 0; wv < PD_WARPS; ++wv) {
            const int g = ib * PD_WARPS + wv;
            if (P.gvalid[g] > 0) {
                min_cls = P.gclass[g];
                break;
            }
        }
        if (min_cls < 0) continue;
        for (int k = min_cls; k < c; ++k) {
            const int32_t cend = P.cls_start[k] + static_cast<int32_t>(count[k]);
            const int32_t s0 = std::max(i0, P.cls_start[k]);
            if (cend - 1 <= i0) continue;  // no j > the block's first atom
            if (lat_of_cls[k] >= 0) {
                // a lattice class's self pairs come from its pair counts: drop
                // the tiles whose i atoms all belong to it
                bool all_k = true;
                for (int wv = 0; wv < PD_WARPS; ++wv) {
                    const int g = ib * PD_WARPS + wv;
                    if (P.gvalid[g] > 0 && P.gclass[g] != k) all_k = false;
                }
                if (all_k) continue;
            }
            for (int32_t j0 = s0; j0 < cend; j0 += TJ)
                tiles.push_back(Tile{i0, j0, std::min(cend, j0 + TJ), k});
        }
    }
    P.jobs_per_frame = static_cast<int64_t>(tiles.size()) * P.nqb;
    if (P.jobs_per_frame * P.n_frames > (int64_t{1} << 31) - 1) {
        msg = "too many tiles for one launch; use a larger j chunk";
        return PD_EINVAL;
    }
    // Slots: the warps of one class in an i-block share one slot (the kernel
    // adds them in warp order at the end of the tile); a padding warp (no
    // valid atom, all-zero sums) joins slot 0. Reduction lists: (pair,
    // q-block) -> slots in creation order.
    std::vector<std::vector<int64_t>> lists(static_cast<size_t>(P.n_pairs) * P.nqb);
    std::vector<PdJob> frame_jobs;
    frame_jobs.reserve(P.jobs_per_frame);
    uint64_t covered = 0;
    int64_t next_slot = 0;
    for (const Tile &t : tiles) {
        int rel[PD_WARPS];
        int cls_of_slot[PD_WARPS];
        int nslot = 0;
        int64_t map = 0;
        for (int wv = 0; wv < PD_WARPS; ++wv) {
            const int g = t.i0 / PD_GRANULE + wv;
            const int a = P.gvalid[g] > 0 ? P.gclass[g] : -1;
            int s = -1;
            for (int u = 0; u < nslot && s < 0; ++u)
                if (cls_of_slot[u] == a) s = u;
            if (s < 0 && a < 0 && nslot > 0) s = 0;  // padding joins slot 0
            if (s < 0) {
                s = nslot;
                cls_of_slot[nslot++] = a;
            }
            rel[wv] = s;
            map |= static_cast<int64_t>(s) << (PD_SLOT_MAP_SHIFT + 2 * wv);
        }
        for (int qb = 0; qb < P.nqb; ++qb) {
            PdJob jb{};
            jb.req = 0;
            jb.frame = 0;
            jb.i0 = t.i0;
            jb.j0 = t.j0;
            jb.j1 = t.j1;
            jb.qb = qb;
            jb.slot = next_slot | map;
            frame_jobs.push_back(jb);
            bool listed[PD_WARPS] = {false, false, false, false};
            for (int wv = 0; wv < PD_WARPS; ++wv) {
                const int g = t.i0 / PD_GRANULE + wv;
                const int a = P.gclass[g];
                if (a < 0 || P.gvalid[g] == 0 || a > t.cls) continue;
                if (a == t.cls && lat_of_cls[a] >= 0) continue;  // from the pair counts
                const int64_t ilo = static_cast<int64_t>(g) * PD_GRANULE;
                const int64_t ihi = ilo + P.gvalid[g];  // exclusive
                if (t.j1 - 1 <= ilo) continue;          // every j <= every i
                if (!listed[rel[wv]]) {
                    lists[static_cast<size_t>(pair_index[a * c + t.cls]) * P.nqb + qb].push_back(
                        next_slot + rel[wv]);
                    listed[rel[wv]] = true;
                }
                if (qb == 0 && count_pairs) {
                    // Σ_{i in [ilo, ihi)} max(0, j1 − max(j0, i + 1)): the i
                    // below j0 − 1 see the whole range, the others an
                    // arithmetic series j1 − 1 − i
                    const int64_t j0 = t.j0, j1 = t.j1;
                    const int64_t a_end = std::min(ihi, j0 - 1);
                    if (a_end > ilo) covered += static_cast<uint64_t>((a_end - ilo) * (j1 - j0));
                    const int64_t b0 = std::max(ilo, j0 - 1), b1 = std::min(ihi, j1 - 1);
                    if (b1 > b0)  // terms j1 − 1 − b0 down to j1 − b1
                        covered += static_cast<uint64_t>(((j1 - 1 - b0) + (j1 - b1)) * (b1 - b0) / 2);
                }
            }
            next_slot += nslot;
        }
    }
    P.slots_per_frame = next_slot;
    if (P.slots_per_frame * P.n_frames >= (int64_t{1} << (PD_SLOT_MAP_SHIFT - 1))) {
        msg = "too many tile slots for one request";
        return PD_EINVAL;
    }
    for (const PdLatDev &d : P.lat)
        covered += static_cast<uint64_t>(d.n) * static_cast<uint64_t>(d.n - 1) / 2;
    P.pairs_covered = covered;
    P.lptr.assign(static_cast<size_t>(P.n_pairs) * P.nqb + 1, 0);
    for (size_t e = 0; e < lists.size(); ++e) P.lptr[e + 1] = P.lptr[e] + lists[e].size();
    P.lidx.reserve(P.lptr.back());
    for (auto &l : lists) P.lidx.insert(P.lidx.end(), l.begin(), l.end());

    // Execution order: longest tiles first (j length), stable; replicated
    // per frame with frame-offset slots. A tile's q-block jobs are
    // consecutive in creation order and of one length, so sorting the tiles
    // gives the order a stable sort of the jobs would.
    std::vector<int64_t> order(tiles.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int64_t x, int64_t y) {
        return (tiles[x].j1 - tiles[x].j0) > (tiles[y].j1 - tiles[y].j0);
    });
    P.jobs.reserve(frame_jobs.size() * P.n_frames);
    for (int64_t o : order) {
        for (int qb = 0; qb < P.nqb; ++qb) {
            for (int f = 0; f < P.n_frames; ++f) {
                PdJob jb = frame_jobs[o * P.nqb + qb];
                jb.frame = f;
                jb.slot += static_cast<int64_t>(f) * P.slots_per_frame;
                P.jobs.push_back(jb);
            }
        }
    }
    set_reduction(P);
    return PD_OK;
}

__attribute__((optimize("O3"))) double max_radius(const double *xyz, int64_t n, int64_t n_frames) {
    double best = 0.0;
    for (int64_t f = 0; f < n_frames; ++f) {
        const double *p = xyz + 3 * n * f;
        // four atoms at a time in twelve sums: vector additions
        double s[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}, c[12], far = 0.0;
        int64_t i = 0;
        for (; i + 4 <= n; i += 4)
            for (int a = 0; a < 12; ++a) s[a] += p[3 * i + a];
        for (; i < n; ++i)
            for (int a = 0; a < 3; ++a) s[a] += p[3 * i + a];
        for (int a = 0; a < 3; ++a) {
            c[a] = ((s[a] + s[a + 3]) + (s[a + 6] + s[a + 9])) / static_cast<double>(n);
            c[a + 3] = c[a + 6] = c[a + 9] = c[a];
            far = std::max(far, std::fabs(c[a]));
        }
        double m[4] = {0, 0, 0, 0};
        for (i = 0; i + 4 <= n; i += 4) {
            double t[12];
            for (int a = 0; a < 12; ++a) {
                t[a] = p[3 * i + a] - c[a];
                t[a] *= t[a];
            }
            for (int k = 0; k < 4; ++k) {
                const double r2 = t[3 * k] + t[3 * k + 1] + t[3 * k + 2];
                m[k] = m[k] > r2 ? m[k] : r2;
            }
        }
        for (; i < n; ++i) {
            const double x = p[3 * i] - c[0], y = p[3 * i + 1] - c[1], z = p[3 * i + 2] - c[2];
            m[0] = std::max(m[0], x * x + y * y + z * z);
        }
        const double r2 = std::max(std::max(m[0], m[1]), std::max(m[2], m[3]));
        best = std::max(best, std::sqrt(r2) * (1.0 + 1e-6) + 1e-9 * far);
    }
    return best;
}

// Terms of a Bessel series of argument z, as direction_order on the device, and of
// the interpolation nodes.
static double series_order(double z, bool fp64) {
    return fp64 ? z + 15.0 * std::cbrt(0.5 * z) + 5.0 : z + 8.0 * std::cbrt(0.5 * z) + 2.0;
}
static double node_order(double z) { return z + 13.0 * std::cbrt(0.5 * z) + 3.0; }

// Atom chunks of the direction form, longest first. A longer chunk means fewer sums
// to hold and to add up, a shorter one more units to share: 2.5 units for each of 592
// blocks (four per SM, what the kernel for up to 64 moments holds; the one for more holds
// three and the FP64 one two), at least 1,024 atoms and at most 16,384, with the
// directions of a globule of the request's atom count (its coordinates would be
// better, but then a solve's rounding would depend on when they are known). Measured,
// whole execution in µs with chunks of 512 / 1,024 / 2,048 / 4,096 / 16,384 atoms: 3,000
// atoms 77 / 75 / 83 / 83 / 83, 10,000 atoms 101 / 102 / 101 / 112 / 144, 20,000 atoms 503 /
// 457 / 443 / 441 / 468, 100,000 atoms 5,165 / 4,599 / 4,346 / 4,229 / 4,155.
static void set_chunks(Plan &P) {
    const double n = static_cast<double>(P.n_atoms);
    const double z = 2.0 * P.qmax * std::cbrt(n * 17.0 * 3.0 / (4.0 * M_PI));
    const double top = series_order(z, P.precision == PD_FP64);
    const double want = 0.4 * n * P.n_frames * (0.2 * top * top / PD_DIR_DIRS) / 592.0;
    const int64_t len = want < 1024.0 ? 1024 : (want < 16384.0 ? static_cast<int64_t>(want) : 16384);
    P.chunks.clear();
    P.cls_chunk.clear();
    for (int k = 0; k < P.n_cls; ++k) {
        const int64_t nk = static_cast<int64_t>(P.cls[k].n), parts = (nk + len - 1) / len;
        for (int64_t t = 0; t < parts; ++t)
            P.chunks.push_back(PdChunk{k, P.cls_start[k] + static_cast<int32_t>(nk * t / parts),
                                       P.cls_start[k] + static_cast<int32_t>(nk * (t + 1) / parts),
                                       0});
    }
    std::stable_sort(P.chunks.begin(), P.chunks.end(), [](const PdChunk &x, const PdChunk &y) {
        return x.j1 - x.j0 > y.j1 - y.j0;
    });
    P.cls_ptr.assign(P.n_cls + 1, 0);
    for (const PdChunk &ck : P.chunks) ++P.cls_ptr[ck.cls + 1];
    std::partial_sum(P.cls_ptr.begin(), P.cls_ptr.end(), P.cls_ptr.begin());
    P.cls_chunk.resize(P.chunks.size());
    std::vector<int32_t> next(P.cls_ptr.begin(), P.cls_ptr.end() - 1);
    for (size_t t = 0; t < P.chunks.size(); ++t)
        P.cls_chunk[next[P.chunks[t].cls]++] = static_cast<int32_t>(t);
}

// A plan without tiles, where the frames' exact radius (radius_hint, the largest
// one) is known and the direction form is the cheaper one by pd_pack's own
// comparison: planning and upload of the tiles, slots and lists were 4.7 of the
// 10 ms of a 100,000-atom solve, 0.14 of 0.3 ms at 3,000 atoms. The sizes hold for
// every frame: the counts of rings, ring points, moments and nodes grow with the
// radius. False (and the tiles follow) where the tiles' plan might be refused.
static bool direction_only(Plan &P) {
    const double frames = P.n_frames, K = P.tun.K;
    const double tiles = static_cast<double>(P.n_pad / PD_IBLOCK) *
                         (P.n_cls + static_cast<double>(P.n_pad) / P.tun.TJ);
    const double jobs = tiles * P.nqb, slots = jobs * PD_WARPS;
    if (jobs * frames > 2147483647.0 ||
        slots * frames >= static_cast<double>(int64_t{1} << (PD_SLOT_MAP_SHIFT - 1)))
        return false;
    P.jobs_per_frame = 2;  // (any: this rank has jobs of every frame)
    P.lptr.assign(static_cast<size_t>(P.n_pairs) * P.nqb + 1, 0);
    P.dir_only = true;
    set_reduction(P);
    double pair_cost = P.mom.grid_dir_cost, latency = P.mom.grid_latency;
    if (P.mom.block > 0) {
        const double d = std::max(2.0 * 1.03 * P.radius_hint, 1e-6);
        const double z = P.qmax * d;  // the moments of pd_pack's pair form
        const double m = z + 9.7 * std::cbrt(0.5 * z) + 3.5;
        const double m8 =
            m < 1e6 ? static_cast<double>((static_cast<int64_t>(0.5 * m) + 8) & ~int64_t{7}) : 1e6;
        const double blocks = std::ceil(m8 / P.mom.block);
        if (m8 <= P.mom.max_moments && blocks <= P.nqb &&
            P.mom.mom_cost * m8 + P.mom.mom_block_cost * blocks < P.mom.grid_cost) {
            pair_cost = 56.0 * blocks + 1.5 * m8;
            latency = P.mom.mom_latency;
        }
    }
    pair_cost *= P.mom.n_tile_pairs;
    pair_cost += P.mom.tile_cost + latency;
    const bool use = P.amp.dir_cap > 0 && P.dir_cost < pair_cost;
    if (!use) {
        P.dir_only = false;
        return false;
    }
    const double row = std::max<double>(P.nq, PD_MAX_MOMENTS) + 128.0;
    P.pair_bytes = frames * (slots * P.nv * K * 8.0 + jobs * sizeof(PdJob)) + slots * 8.0 +
                   17.0 * frames * P.n_pairs * P.nv * row * 8.0 +
                   static_cast<double>(P.lat_bins) * 8.0 + (1 << 20);
    // Jobs: shares of the frame's units for the serving loop's steps (a whole
    // plan's blocks take the units by number instead).
    const int64_t per = std::min<int64_t>(
        P.dir_units, std::max<int64_t>(1, (1024 + P.n_frames - 1) / P.n_frames));
    P.jobs_per_frame = per;
    P.job_cost = P.dir_work / (3.0 * static_cast<double>(per));
    if (P.precision == PD_FP64) P.job_cost *= 2.0;
    P.jobs.resize(static_cast<size_t>(per) * P.n_frames);
    for (int64_t o = 0; o < per; ++o)
        for (int f = 0; f < P.n_frames; ++f) {
            PdJob &jb = P.jobs[static_cast<size_t>(o) * P.n_frames + f];
            jb = PdJob{};
            jb.frame = f;
            jb.j0 = static_cast<int32_t>(o);
            jb.j1 = static_cast<int32_t>(per);
        }
    return true;
}

// Sizes of the direction form for frames of up to the hinted radius (pd_pack
// decides per frame, with the same formulas, whether it fits and pays).
static void set_directions(Plan &P) {
    P.amp = PdAmpShape{};
    P.amp.nq = P.nq;
    P.amp.dir_block = P.precision == PD_FP64 ? PD_DIR_MBLOCK64 : PD_DIR_MBLOCK;
    P.amp.rank = static_cast<int32_t>(P.rank);
    P.amp.world = static_cast<int32_t>(P.world);
    P.amp.n_cls = P.n_cls;
    P.amp.nv2 = P.mode == PD_MODE_WEIGHTED ? 2 : 1;
    P.amp.n_chunk = static_cast<int32_t>(P.chunks.size());
    // Below 150 atoms the moments of the pairs are cheaper than the directions. In FP64 a
    // grid point costs a double sin and a chain of them per atom (whole solves, 100
    // points, pairs / directions: 8 atoms 71 / 59 us, 16 atoms 88 / 59, 100 atoms 233 /
    // 59): only a handful of atoms stay pairs, whose sums have no quadrature. The jobs
    // carry the work units, so every rank needs jobs of every frame. The test hook (of
    // the FP32 form) needs the pair tiles.
    const int64_t fewest = P.precision == PD_FP64 ? 12 : 150;
    if (P.no_directions || P.n_atoms < fewest ||
        P.jobs_per_frame < 2 * static_cast<int64_t>(P.world) ||
        (P.world > 1 && P.n_frames > 1) || (P.test_expire && P.precision != PD_FP64))
        return;
    // unknown coordinates: 20 cubic Angstrom per atom, elongated up to about 2.5 : 1
    const double radius =
        P.radius_hint >= 0.0
            ? P.radius_hint
            : 1.9 * std::cbrt(static_cast<double>(P.n_atoms) * 20.0 * 3.0 / (4.0 * M_PI));
    const bool fp64 = P.precision == PD_FP64;
    auto order = [&](double z) { return series_order(z, fp64); };
    const double z = 2.0 * radius * P.qmax;
    const double r1 = std::max(1.03 * radius, 1e-6);  // (as pd_pack bounds it)
    const double top = order(z), mo = order(r1 * P.qmax);
    if (!(top < 500.0) || !(mo < PD_MAX_DIR_MOMENTS - 8.0)) return;
    const int h = static_cast<int>(top * 0.25) + 1;
    int64_t S = 0;
    for (int i = 0; i < h; ++i)  // rings at nearly the Gauss angles, one point to spare each
        S += std::max(4, static_cast<int>(order(z * std::sin(M_PI * (i + 0.75) / (2 * h + 0.5)))) + 2);
    const int64_t groups = (S + 31) / 32, mine = (groups + P.world - 1) / P.world;
    const int64_t m8 = (static_cast<int64_t>(mo) + 8) & ~int64_t{7};
    const double zn = 2.0 * r1 * P.qmax;
    const int64_t nodes = fp64 ? P.nq : static_cast<int64_t>(0.5 * node_order(zn)) + 1;
    // The sums' kernel: a block's shared memory holds the coefficients and the
    // amplitudes of every class at a tile of nodes (16, or fewer while that leaves
    // SMs without a block), and the moments of as many classes as fit; up to
    // 110 KB (two blocks per SM) unless one class's moments need more.
    const int64_t ncv = static_cast<int64_t>(P.n_cls) * P.amp.nv2;
    int64_t tile = 16;
    while (tile > 4 && (S + 31) / 32 * ((nodes + tile - 1) / tile) * P.n_frames < 296) tile /= 2;
    while (tile > 4 && m8 * (tile + 32) + ncv * tile * 64 > PD_DIR_SMEM / 8) tile -= 4;
    const int64_t least = m8 * (tile + 32) + ncv * tile * 64;
    if (least > PD_DIR_SMEM / 8) return;
    P.amp.sum_smem = static_cast<int32_t>(std::max(
        least, std::min<int64_t>(110 * 1024 / 8, m8 * tile + ncv * (tile * 64 + m8 * 32))));
    const int64_t slots = P.amp.n_chunk * P.amp.nv2 * mine * m8 * 32;
    const int64_t parts = mine * P.n_pairs * P.nv * nodes;
    if (std::max(slots, parts) * 8 * P.n_frames > (int64_t{4} << 30)) return;
    P.amp.dir_cap = static_cast<int32_t>(groups * 32);
    P.amp.grp_cap = static_cast<int32_t>(mine);
    P.amp.amp_cap = static_cast<int32_t>(std::min<int64_t>(m8, PD_MAX_DIR_MOMENTS));
    P.amp.node_cap = static_cast<int32_t>(nodes);
    P.amp.node_tile = static_cast<int32_t>(tile);
    P.amp.slot_cap = slots;
    const double ablk = static_cast<double>((m8 + P.amp.dir_block - 1) / P.amp.dir_block);
    P.dir_work = static_cast<double>(S) *
                 ((static_cast<double>(P.n_atoms) + (fp64 ? PD_DIR_CHUNK64 * P.amp.n_chunk : 0.0)) *
                      P.amp.nv2 * (44.0 * ablk - 30.0 + 1.25 * m8) +
                  4.0 * P.n_cls * static_cast<double>(m8) * static_cast<double>(nodes));
    P.dir_cost = P.dir_work + P.mom.dir_pair_cost *
                                  std::max(static_cast<double>(S) * static_cast<double>(nodes),
                                           PD_DIR_LEAST);
    P.dir_units = static_cast<int64_t>(P.amp.n_chunk) * P.amp.nv2 *
                  static_cast<int64_t>(ablk) * mine * (32 / PD_DIR_DIRS);
}

void drop_directions(Plan &P) {
    P.no_directions = true;
    set_reduction(P);
}

void make_compact(Plan &P) {
    P.no_directions = P.compact = true;
    set_reduction(P);
}

void set_reduction(Plan &P) {
    PdMomentRule &m = P.mom;
    m = PdMomentRule{};
    m.qmax = P.qmax;
    m.nqb = P.nqb;
    m.fp64 = P.precision == PD_FP64 ? 1 : 0;
    m.block = m.fp64 ? 0 : pd_moment_block(P.tun.K);
    m.max_moments = static_cast<int32_t>(
        std::min<int64_t>({PD_MAX_MOMENTS, static_cast<int64_t>(P.nqb) * m.block,
                           P.compact ? P.nq : PD_MAX_MOMENTS}) & ~int64_t{7});
    if (m.max_moments < 8) m.block = 0;
    // As measured, whole solves of 3,000 to 20,000 atoms, FP32, in units of 83 % of the
    // FFMA peak: 3 lane operations per grid point (in 16s) and 55 for each q-block's
    // seeds, against 1.25 per moment and 140 for a block of 128 (sequences and flush);
    // weighted mode (two sums per value) 4 and 55 against 2.1 and 200 for a block of 64.
    // Grid points / moments: a rod of 5,000 atoms, 160 moments, 150 points 511 / 414 us,
    // 300 points 819 / 414, weighted 708 / 757 and 1,040 / 757; 20,000 atoms, 208 moments,
    // 150 points 5.5 / 4.4 ms, weighted 7.8 / 10.0 and, 300 points, 12.3 / 10.0. The
    // directions' own operations run at 57 % of the peak (FP64: 23 %), hence the
    // factor 0.7. FP64: a grid point costs a double sin, 110 operations, for whole
    // q-blocks.
    const double points = static_cast<double>((P.nq + 15) & ~15);
    if (m.fp64) {
        m.grid_dir_cost = 0.23 * 110.0 * P.nqb * P.tun.K;
    } else {
        const bool weighted = P.mode == PD_MODE_WEIGHTED;
        m.grid_cost = (weighted ? 4.0 : 3.0) * points + 55.0 * P.nqb;
        m.mom_cost = weighted ? 2.1 : 1.25;
        m.mom_block_cost = weighted ? 72.0 + 2.0 * m.block : 60.0 + 0.625 * m.block;
        m.grid_dir_cost = 0.7 * m.grid_cost;
    }
    // Beyond the pairs: each tile's jobs, with moments a longer chain of short kernels
    // (1e7), and at the grid points a thread's pass over a class's atoms, which is a chain
    // (FP32 8e7: 800 atoms, 1 to 16 points, 111 us, directions 75; FP64 4 us per atom of
    // the largest class: 100 atoms of one class 490 us, directions 67, of eight classes
    // 140 and 77) and which a batch's frames run side by side. On the other side the
    // class pairs' products at each node of each direction, an FP64 contraction of 2 to
    // 7 ps for each. The constants are a fit to whole solves of both forms, 20 to 15,000
    // atoms, 1 to 100 species, 2 to 600 points, 1 to 40 frames: the form chosen is slower
    // than the other by more than 10 % in about 130 of 2,840 cases. Pairs / directions, us: FP64, weighted, 300
    // atoms of 16 species, 300 points 300 / 1,720, 1,000 atoms of 30, 60 points 430 / 940,
    // 40 frames of 100 atoms of 9, 30 points 251 / 1,108; FP32, 10,000 atoms of 60, 60
    // points 950 / 1,980, 10 frames of 2,000 atoms of 30, 150 points 590 / 1,420, 2,000
    // atoms of 84, 1,000 points 4,170 / 770.
    const double all_pairs = 0.5 * static_cast<double>(P.n_atoms) * P.n_atoms;
    m.n_tile_pairs = all_pairs;
    for (const PdLatDev &d : P.lat)
        m.n_tile_pairs -= 0.5 * static_cast<double>(d.n) * d.n;
    const double tiles = 0.5 * static_cast<double>(P.n_pad / PD_IBLOCK) *
                             (P.n_cls + static_cast<double>(P.n_pad) / P.tun.TJ) *
                             (m.n_tile_pairs / all_pairs) + 1.0;
    double largest = 0.0;
    for (const PdClassDev &c : P.cls) largest = std::max(largest, c.n);
    m.tile_cost = 1.2e6 * tiles * P.nqb;
    // (In FP32 a frame's form, whose rounding shows, does not follow its batch's size.)
    m.grid_latency = m.fp64 ? 2e7 * std::min(largest, 256.0) / P.n_frames : 8e7;
    m.mom_latency = 1e7;
    m.dir_pair_cost = (m.fp64 ? 30.0 : 100.0) * P.n_pairs * P.nv;
    set_directions(P);
    m.dir_block = P.amp.dir_block;
    m.dir_cap = P.amp.dir_cap;
    m.grp_cap = P.amp.grp_cap;
    m.amp_cap = P.amp.amp_cap;
    m.node_cap = P.amp.node_cap;
    m.n_chunk = P.amp.n_chunk;
    m.n_cls = P.amp.n_cls;
    m.nv2 = P.amp.nv2;
    m.rank = P.amp.rank;
    m.world = P.amp.world;
    m.slot_cap = P.amp.slot_cap;
    m.n_atoms = P.n_atoms;
    m.nq = P.nq;
    m.dir_only = P.dir_only ? 1 : 0;
    PdReduceShape &r = P.red;
    r = PdReduceShape{};
    r.n_pairs = P.n_pairs;
    r.nq = P.nq;
    r.K = P.tun.K;
    r.nqb = P.nqb;
    r.block = m.block;
    r.max_moments = m.block ? m.max_moments : 0;
    r.n_z = (std::max(P.nq, r.max_moments) + 127) / 128;
    if (!m.fp64) r.max_moments = std::max(r.max_moments, P.amp.node_cap);
    r.node_cap = P.amp.node_cap;
    r.dir_only = m.dir_only;
    r.fp64 = m.fp64;
    r.width = std::max(P.nq, r.max_moments);
    // A block adds its share of a class pair's slot list serially: lists of
    // more than a few hundred entries are shared by up to 16 blocks (one
    // frame; the frames of a batch fill the GPU by themselves).
    int64_t longest = 0;
    for (int p = 0; p < P.n_pairs; ++p)
        longest = std::max(longest, P.lptr[static_cast<size_t>(p + 1) * P.nqb] -
                                        P.lptr[static_cast<size_t>(p) * P.nqb]);
    r.n_chunk = P.n_frames > 1 || P.compact ? 1
                               : static_cast<int32_t>(
                                     std::min<int64_t>(std::max<int64_t>(longest / 256, 1), 16));
    r.slots_per_frame = P.slots_per_frame;
}

int shard_plan(const Plan &full, uint32_t rank, uint32_t world, Plan &out) {
    out = full;
    if (world <= 1) return PD_OK;
    if (rank >= world) return PD_EINVAL;
    const int64_t spf = full.slots_per_frame;
    std::vector<int64_t> remap(static_cast<size_t>(spf), -1);
    auto local_of = [&](const PdJob &jb) {
        return (jb.slot & PD_SLOT_MASK) - static_cast<int64_t>(jb.frame) * spf;
    };
    auto nslot_of = [](const PdJob &jb) {
        int n = 1;
        for (int w = 0; w < PD_WARPS; ++w)
            n = std::max(n, 1 + static_cast<int>((jb.slot >> (PD_SLOT_MAP_SHIFT + 2 * w)) & 3));
        return n;
    };
    out.rank = rank;
    out.world = world;
    out.jobs.clear();
    for (size_t t = rank; t < full.jobs.size(); t += world) {
        const PdJob &jb = full.jobs[t];
        const int64_t loc = local_of(jb);
        for (int s = 0; s < nslot_of(jb); ++s) remap[static_cast<size_t>(loc + s)] = 0;
        out.jobs.push_back(jb);
    }
    // this rank's slots, numbered in their original order (list order kept)
    int64_t k = 0;
    for (auto &r : remap)
        if (r >= 0) r = k++;
    out.slots_per_frame = k;
    for (PdJob &jb : out.jobs) {
        const int64_t loc = local_of(jb);
        jb.slot = (jb.slot & ~PD_SLOT_MASK) |
                  (static_cast<int64_t>(jb.frame) * k + remap[static_cast<size_t>(loc)]);
    }
    out.lidx.clear();
    out.lptr.assign(full.lptr.size(), 0);
    for (size_t e = 0; e + 1 < full.lptr.size(); ++e) {
        for (int64_t x = full.lptr[e]; x < full.lptr[e + 1]; ++x) {
            const int64_t r = remap[static_cast<size_t>(full.lidx[static_cast<size_t>(x)])];
            if (r >= 0) out.lidx.push_back(r);
        }
        out.lptr[e + 1] = static_cast<int64_t>(out.lidx.size());
    }
    set_reduction(out);
    return PD_OK;
}

}  // namespace pd
