// Host-callable launchers of the device kernels (pd_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pd_common.h"

namespace pd {

bool valid_q_block(int precision, int K);
bool valid_shape(int precision, int mode, int K, int NP);
int pairs_blocks_per_sm(int precision, int K, int NP, int mode);
// Set the launch attributes of every FP32 pair-kernel shape on the current
// device (their shared-memory opt-in), so that no later launch — one inside a
// stream capture included — has to.
cudaError_t prepare_pair_kernels();

// `after` of a launcher: the operation before it on the stream is one of these kernels
// (chain_launch in pd_launch.cuh).
//
// n_jobs points to the tile count in device memory (read once per CTA).
// plan_frames > 0: the jobs are those of one request (reqs[0]) with that many
// frames, all of them (counter: two zeroed ints); 0: any jobs of any requests
// (one).
cudaError_t launch_pairs(int precision, int K, int NP, int mode, const PdJob *jobs,
                         const int *n_jobs, const PdReqDev *reqs, int *counter, int plan_frames,
                         int grid, cudaStream_t st, bool after = false);
// The direction form's first stage, for the frames that take it; the other arguments
// are those of launch_pairs (plan_frames > 0 uses the second counter). A variant holds
// up to its number of moments (directions_variant of the most a frame may have).
int directions_variant(int precision, int32_t n_amp);
int directions_blocks_per_sm(int variant);
cudaError_t launch_directions(int variant, const PdJob *jobs, const int *n_jobs,
                              const PdReqDev *reqs, int *counter, int plan_frames, int grid,
                              cudaStream_t st, bool after = false);
// Blocks per frame of the centroid kernel (3 partial sums each).
int32_t centroid_blocks(int64_t n_atoms);
// Centres the frames, packs their atoms in the classes' order and sets the frames'
// constants; clears `status` if given. cent_done, done and rad2 (one per frame) must
// be zero. `launches`: how many kernels it took.
cudaError_t launch_pack(const double *xyz, const double *weights, const int32_t *perm,
                        int64_t n_atoms, int32_t n_pad, int32_t n_frames, double *part,
                        unsigned int *cent_done, double *centroid, int32_t *status, float4 *out32,
                        double4 *out64, const PdMomentRule &rule, unsigned long long *rad2,
                        unsigned int *done, PdFrameDev *frames, double4 *dirs, double2 *node_tab,
                        cudaStream_t st, int *launches);
// The quadrature rules of the direction form on the current device (before any
// launch_pack there, and before a stream capture).
cudaError_t prepare_direction_rules();
// Direction form: class-pair sums at the nodes, or at the grid points qv if given, from
// the chunks' moments, into red (does nothing for frames in the other forms). part holds grp_cap·pairs·nv·
// node_cap doubles per frame, done one zeroed counter per node tile and frame.
cudaError_t launch_direction_sums(const double *slots, const double4 *dirs,
                                  const PdFrameDev *frames, const PdAmpShape &sh, double qmax,
                                  const double *qv, int32_t n_frames, const PdClassDev *cls,
                                  const PdPairDev *pairs,
                                  int32_t n_pairs, const int32_t *cls_ptr,
                                  const int32_t *cls_chunk, int32_t width,
                                  int add_exact, double *part, unsigned int *done, double *red,
                                  cudaStream_t st, bool after = false);
// Slot sums (red: [frame][pair][nv][width]); with n_chunk > 1, chunk_sums holds
// 128·nv·n_chunk doubles and done one zeroed counter per (frame, pair, n_z).
cudaError_t launch_reduce(const double *slots, const int64_t *lptr, const int64_t *lidx,
                          const PdPairDev *pairs, const double *qv, const PdFrameDev *frames,
                          const PdReduceShape &sh, int32_t nv, int32_t n_frames, int residual_form,
                          int add_exact, double *chunk_sums, unsigned int *done, double *red,
                          cudaStream_t st, bool after = false);
cudaError_t launch_profiles(const double *red, const double *lat_sums, const PdClassDev *cls,
                            const PdPairDev *pairs, int32_t n_cls, const PdReduceShape &sh,
                            int32_t nv, int32_t n_frames, const double *qv,
                            const PdFrameDev *frames, const double2 *node_tab, const double *ffA,
                            const double *ffC, const double *ffW, int add_diag, double qmax, const int *err,
                            double *terms, cudaStream_t st, bool after = false);
// Lattice sets: integer coordinates of their points and the exact pair count
// per squared offset (after pack), then their self pair sums, sums[lattice][q].
cudaError_t launch_lattice(const double *xyz, const int32_t *perm, const PdLatDev *lat_dev,
                           const PdLatDev *lat_host, int n_lat, const PdLatTile *tiles,
                           int64_t n_tiles, int4 *idx, unsigned long long *hist, int64_t n_bins,
                           int *err, cudaStream_t st);
cudaError_t launch_lattice_sums(const unsigned long long *hist, const PdLatDev *lat, int n_lat,
                                const double *qv, int32_t nq, int add_exact, const int *err,
                                double *sums, cudaStream_t st);
cudaError_t launch_frame_mean(const double *terms, const double *fw, int32_t n_frames, int32_t nq,
                              double *out, cudaStream_t st, bool normalize = true, bool after = false);
// Direct transform: (Re A, Im A, |A|², Σ_m |F_m|²) per q-vector for points
// in molecules of mol_size (n_points a multiple of it). part holds
// direct_chunks(n_points, mol_size, n_vec) × n_vec × 5 doubles; the launch
// has direct_blocks(…) blocks (at most 2^31 - 1).
cudaError_t launch_direct(const double *xyz, const uint32_t *kind, const double *weight,
                          const double *ff, int32_t n_kinds, const double *qvec, int64_t n_vec,
                          int64_t n_points, int64_t mol_size, double *part, int64_t part_chunks,
                          double *out, cudaStream_t st);
int64_t direct_chunks(int64_t n_points, int64_t mol_size, int64_t n_vec);
// Direct transform at lattice vectors q = 2π·hkl/box from per-point phase
// tables (indices |h|, |k|, |l| <= nmax, with direct_table_points(nmax) >= 1);
// same part and out layouts as launch_direct.
int direct_table_points(int32_t nmax);
cudaError_t launch_direct_table(const double *xyz, const uint32_t *kind, const double *weight,
                                const double *ff, const int32_t *hkl, int32_t nmax,
                                const double box[3], int64_t n_vec, int64_t n_points,
                                int64_t mol_size, double *part, int64_t part_chunks, double *out,
                                cudaStream_t st);
int64_t direct_blocks(int64_t n_points, int64_t mol_size, int64_t n_vec);
// Direct transform at lattice vectors on lines of PD_DLINE_J (16) consecutive ones
// (see pd_direct_lines): points grouped by kind within each molecule, ff
// [n_kinds][16][n_line], index the distinct indices of the three axes; part holds
// 32·n_line doubles per chunk, out 4 per vector (j·n_line + line).
int direct_line_points(int32_t n_entries);
void direct_line_layout(int64_t n_points, int64_t mol_size, int32_t n_line, int64_t *chunk,
                        int64_t *spm);
// Points of each molecule sorted by kind, in pieces of a few thousand (n_kinds <= 44).
cudaError_t launch_direct_sort(const double *xyz, const uint32_t *kind, const double *weight,
                               int64_t n_points, int64_t mol_size, int32_t n_kinds,
                               double *xyz_out, uint32_t *kind_out, double *weight_out,
                               cudaStream_t st);
cudaError_t launch_direct_lines(const double *xyz, const uint32_t *kind, const double *weight,
                                const double *ff, const PdLine *lines, const int32_t *index,
                                const int32_t n_index[3], const double box[3], int32_t n_line,
                                int64_t n_points, int64_t mol_size, int64_t chunk, int64_t spm,
                                double *part, double *out, cudaStream_t st);
// Form-factor tables [n_ff][nq] on the uniform grid; *bad = index + 1 of a
// form factor whose range misses a grid point (0 if none).
cudaError_t launch_ff_eval(const int32_t *desc, const double *range, const double *params,
                           int32_t n_ff, double qmin, double qmax, int64_t nq, int *bad,
                           double *out, cudaStream_t st);
cudaError_t launch_stream_accumulate(const double *batch, double scale, int32_t n, double *acc,
                                     cudaStream_t st);
cudaError_t launch_ffma_probe(float *out, int iters, int grid, int block, bool packed,
                              cudaStream_t st);

}  // namespace pd
