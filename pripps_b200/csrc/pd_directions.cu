// Direction form, first stage: Σ_j T_n(n·r_j/r1) over the atoms of a chunk, in
// each direction of the quadrature (pd_moments.cuh), for the sums of the class
// pairs that follow.
#include <algorithm>

#include "pd_kernels.h"
#include "pd_launch.cuh"
#include "pd_moments.cuh"

namespace pd {

// Atoms a thread sums in FP32 for its direction before the CTA's sums go, in FP64,
// into the unit's slot. The low moments are coherent sums, whose rounding shows at the
// deep minima: 100,000 atoms, largest error of a profile point 1.8e-6 with 512 atoms,
// 3.3e-7 with 128 and 2.0e-7 with 64 (the pair form 4.3e-7), in 4.08, 4.20 and 4.31 ms.
constexpr int PD_DIR_RUN = 128;
// Atoms staged at once: two buffers of 16 KB, filled by asynchronous copies (a
// thread's pass over a block is shorter than a read from L2).
template <class Atom>
constexpr int dir_block() { return 16384 / static_cast<int>(sizeof(Atom)); }
static_assert(PD_DIR_RUN * PD_DIR_LANES % dir_block<float4>() == 0, "a run is whole blocks");

template <int MAXM>
constexpr int dir_smem_bytes() {
    return 2 * 16384 + PD_WARPS * MAXM * PD_DIR_DIRS * static_cast<int>(sizeof(float));
}
constexpr int DIR_SMEM64 =
    2 * 16384 + PD_WARPS * PD_DIR_MBLOCK64 * PD_DIR_DIRS * static_cast<int>(sizeof(double));

// A work unit, u-th of the frame's n_chunk·nv2·n_ablk·4·n_grp: one chunk (weighted or
// not) and moment block in 8 directions, a quarter of a group. The longest chunks come
// first, the directions are innermost.
struct DirUnit {
    const void *at;      // the frame's atoms
    const double4 *dir;  // its 8 directions
    double *out;
    int c0, c1;          // the chunk
    int n_amp, mb;
    bool ok, weighted;
};

__device__ __forceinline__ unsigned dir_unit_count(int n_chunk, int nv2, int n_ablk, int n_grp) {
    return static_cast<unsigned>(n_chunk) * nv2 * n_ablk * n_grp * (32 / PD_DIR_DIRS);
}

template <class Atom>
__device__ __forceinline__ void dir_unit_set(DirUnit &d, const PdReqDev &rq, const PdChunk *chunks,
                                             int frame, int n_grp, int n_amp, unsigned u) {
    constexpr unsigned PER = 32 / PD_DIR_DIRS;
    const int mblock = sizeof(Atom) == sizeof(double4) ? PD_DIR_MBLOCK64 : PD_DIR_MBLOCK;
    const unsigned n_ablk = (n_amp + mblock - 1) / mblock, nv2 = rq.amp.nv2;
    const unsigned sub = u % PER;
    u /= PER;
    const unsigned grp = u % n_grp;
    u /= n_grp;
    d.mb = n_ablk > 1 ? static_cast<int>(u % n_ablk) : 0;
    if (n_ablk > 1) u /= n_ablk;
    const unsigned v = nv2 > 1 ? u & 1 : 0;
    const unsigned chunk = nv2 > 1 ? u >> 1 : u;
    const PdChunk ck = chunks[chunk];
    d.c0 = ck.j0;
    d.c1 = ck.j1;
    d.weighted = v != 0;
    d.n_amp = n_amp;
    const Atom *at;
    if constexpr (sizeof(Atom) == sizeof(double4))
        at = rq.atoms64;
    else
        at = rq.atoms32;
    d.at = at + static_cast<size_t>(frame) * rq.n_pad;
    d.dir = rq.dirs + static_cast<int64_t>(frame) * rq.amp.dir_cap +
            (static_cast<int64_t>(grp) * rq.amp.world + rq.amp.rank) * 32 + sub * PD_DIR_DIRS;
    d.out = rq.dir_slots + static_cast<int64_t>(frame) * rq.amp.slot_cap +
            ((static_cast<int64_t>(chunk) * nv2 + v) * n_grp + grp) * n_amp * 32 +
            sub * PD_DIR_DIRS;
    d.ok = true;
}

__device__ __forceinline__ void dir_copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

// Atoms j0 … j1 − 1 into dst (one group of copies, also when there are none).
template <class Atom>
__device__ __forceinline__ void dir_stage(Atom *dst, const Atom *at, int j0, int j1) {
    constexpr int P = sizeof(Atom) / 16;
    const char *src = reinterpret_cast<const char *>(at + j0);
    for (int k = threadIdx.x; k < (j1 - j0) * P; k += PD_THREADS)
        dir_copy16(reinterpret_cast<char *>(dst) + 16 * k, src + 16 * k);
}
// A unit's first block and its directions.
template <class Atom>
__device__ __forceinline__ void dir_stage_first(Atom *dst, double4 *dir, const DirUnit &n) {
    dir_stage(dst, static_cast<const Atom *>(n.at), n.c0, min(n.c1, n.c0 + dir_block<Atom>()));
    if (threadIdx.x < 2 * PD_DIR_DIRS)
        dir_copy16(reinterpret_cast<char *>(dir) + 16 * threadIdx.x,
                   reinterpret_cast<const char *>(n.dir) + 16 * threadIdx.x);
}
__device__ __forceinline__ void dir_stage_end() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The sums of a warp's four atom lanes (lane / 8), reduce-scattered: afterwards
// atom lane a holds acc[t], a·NT/4 <= t < (a + 1)·NT/4, in acc[0 .. NT/4).
template <int NT>
__device__ __forceinline__ void direction_scatter(float2 (&v)[NT], int lane) {
#pragma unroll
    for (int lev = 0; lev < 2; ++lev) {
        const int o = 16 >> lev, h = (NT >> lev) / 2;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float2 lo = v[k], hi = v[k + h];
            const float2 keep = up ? hi : lo;
            const float2 send = up ? lo : hi;
            v[k] = __fadd2_rn(keep, make_float2(__shfl_xor_sync(0xffffffffu, send.x, o),
                                                __shfl_xor_sync(0xffffffffu, send.y, o)));
        }
    }
}

// One work unit with KM moments (LATER: of a later block). A lane is one of 8
// directions for every 16th atom of the chunk, so 128 threads share 8·KM sums: few
// enough units fill the GPU with short loops on small structures, and the slots stay
// small. A run's sums of the 16 atom lanes meet by shuffles and in shared memory and
// are added to the slot in warp order, in FP64. The unit's first block and directions
// are on their way into buffer b and dir when it starts, and it starts those of the
// next unit behind its own last block; returns the next unit's buffer.
//
// Bound: the FP32 pipe, 10 lane operations for eight moments and 14 for an atom's
// start. KM is the moment count itself up to the next 8 or 16 (no branch between
// the groups of eight), two atoms at a time up to 96 moments. TAG keeps the
// kernels' register limits apart.
template <class Atom, int KM, bool LATER, int TAG>
__device__ __noinline__ int dir_unit_run(const DirUnit &un, const DirUnit &next,
                                         Atom *__restrict__ buf, int b,
                                         const double4 *__restrict__ dir,
                                         double4 *__restrict__ next_dir) {
    constexpr bool F64 = sizeof(Atom) == sizeof(double4);
    constexpr int NT = KM / 2, BLOCK = dir_block<Atom>();
    constexpr int RUN = F64 ? (1 << 30) : PD_DIR_RUN * PD_DIR_LANES;
    constexpr int MBLOCK = F64 ? PD_DIR_MBLOCK64 : PD_DIR_MBLOCK;
    const Atom *at = static_cast<const Atom *>(un.at);
    const int c0 = un.c0, c1 = un.c1, n_amp = un.n_amp, mb = LATER ? un.mb : 0;
    const bool weighted = un.weighted;
    double *__restrict__ out = un.out;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nj = LATER ? min(KM, n_amp - mb * MBLOCK) >> 3 : KM / 8;
    const int at0 = static_cast<int>(threadIdx.x) / PD_DIR_DIRS, dl = lane % PD_DIR_DIRS;
    const int rows = min(nj * 4, (n_amp - mb * MBLOCK) >> 1);
    for (int r0 = c0; r0 < c1;) {
        const int r1 = RUN < c1 - r0 ? r0 + RUN : c1;
        if constexpr (F64) {
            double acc[KM];
#pragma unroll
            for (int e = 0; e < KM; ++e) acc[e] = 0.0;
            for (int j0 = r0; j0 < r1; j0 += BLOCK, b ^= 1) {
                const int j1 = min(c1, j0 + BLOCK);
                if (j1 < c1)
                    dir_stage(buf + (b ^ 1) * BLOCK, at, j1, min(c1, j1 + BLOCK));
                else if (next.ok)
                    dir_stage_first(buf + (b ^ 1) * BLOCK, next_dir, next);
                dir_stage_end();
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();
                if constexpr (LATER)
                    direction_range_later_f64<KM>(buf + b * BLOCK, dir[dl], weighted, at0, j1 - j0,
                                                  nj, mb, acc);
                else
                    direction_range_f64<KM, (KM <= 48)>(buf + b * BLOCK, dir[dl], weighted, at0,
                                                        j1 - j0, acc);
                __syncthreads();  // the block is read before its buffer is refilled
            }
            double *part = reinterpret_cast<double *>(buf + 2 * BLOCK);  // [warp][e][8]
#pragma unroll
            for (int e = 0; e < KM; ++e) {
                double a = acc[e];
                a += __shfl_xor_sync(0xffffffffu, a, 8);
                a += __shfl_xor_sync(0xffffffffu, a, 16);
                if (lane < PD_DIR_DIRS) part[(warp * KM + e) * PD_DIR_DIRS + lane] = a;
            }
            __syncthreads();
            for (int k = threadIdx.x; k < rows * PD_DIR_DIRS; k += PD_THREADS) {
                const int d = k % PD_DIR_DIRS, i = k / PD_DIR_DIRS;
                double x = 0.0, y = 0.0;
#pragma unroll
                for (int w = 0; w < PD_WARPS; ++w) {
                    const double *c = part + (w * KM + 2 * i) * PD_DIR_DIRS + d;
                    x += c[0];
                    y += c[PD_DIR_DIRS];
                }
                if constexpr (LATER)
                    direction_put_later(out, mb * MBLOCK, i >> 2, i & 3, d, x, y, true);
                else
                    direction_put(out, i >> 2, i & 3, d, x, y, true);
            }
        } else {
            float2 acc[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = make_float2(0.0f, 0.0f);
            for (int j0 = r0; j0 < r1; j0 += BLOCK, b ^= 1) {
                const int j1 = min(c1, j0 + BLOCK);
                if (j1 < c1)
                    dir_stage(buf + (b ^ 1) * BLOCK, at, j1, min(c1, j1 + BLOCK));
                else if (next.ok)
                    dir_stage_first(buf + (b ^ 1) * BLOCK, next_dir, next);
                dir_stage_end();
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();
                const double4 D = dir[dl];
                const float3 dv = make_float3(static_cast<float>(D.x), static_cast<float>(D.y),
                                              static_cast<float>(D.z));
                if constexpr (LATER)
                    direction_range_later<KM>(buf + b * BLOCK, dv, weighted, at0, j1 - j0, nj, mb,
                                              acc);
                else
                    direction_range<KM, (KM <= 96)>(buf + b * BLOCK, dv, weighted, at0, j1 - j0,
                                                    acc);
                __syncthreads();  // the block is read before its buffer is refilled
            }
            float *sums = reinterpret_cast<float *>(buf + 2 * BLOCK);  // [warp][e][8]
            const int a = lane / PD_DIR_DIRS;
            float *o = sums + warp * KM * PD_DIR_DIRS + dl;
            direction_scatter<NT>(acc, lane);
#pragma unroll
            for (int t = 0; t < NT / 4; ++t) {
                // row e ^ a: the four atom lanes write different banks
                const int e = 2 * (a * (NT / 4) + t);
                o[(e ^ a) * PD_DIR_DIRS] = acc[t].x;
                o[((e + 1) ^ a) * PD_DIR_DIRS] = acc[t].y;
            }
            __syncthreads();
            for (int k = threadIdx.x; k < rows * PD_DIR_DIRS; k += PD_THREADS) {
                const int d = k % PD_DIR_DIRS, i = k / PD_DIR_DIRS;  // i = 4·jj + t
                const int al = i / (NT / 4);
                double x = 0.0, y = 0.0;
#pragma unroll
                for (int w = 0; w < PD_WARPS; ++w) {
                    const float *c = sums + w * KM * PD_DIR_DIRS + d;
                    x += static_cast<double>(c[((2 * i) ^ al) * PD_DIR_DIRS]);
                    y += static_cast<double>(c[((2 * i + 1) ^ al) * PD_DIR_DIRS]);
                }
                if constexpr (LATER)
                    direction_put_later(out, mb * MBLOCK, i >> 2, i & 3, d, x, y, r0 == c0);
                else
                    direction_put(out, i >> 2, i & 3, d, x, y, r0 == c0);
            }
        }
        r0 = r1;
        __syncthreads();  // sums are rewritten by the next run
    }
    return b;
}

template <class Atom, int MAXM>
__device__ __forceinline__ int dir_unit(const DirUnit &un, const DirUnit &next,
                                        Atom *__restrict__ buf, int b, const double4 *dir,
                                        double4 *next_dir) {
    const int M = un.n_amp;
#define PD_DIR_CASE(KM)        \
    if (MAXM >= KM && M <= KM) \
        return dir_unit_run<Atom, KM, false, MAXM>(un, next, buf, b, dir, next_dir);
    if (un.mb == 0) {
        if constexpr (sizeof(Atom) == sizeof(float4)) { PD_DIR_CASE(16) }
        PD_DIR_CASE(24) PD_DIR_CASE(32) PD_DIR_CASE(40) PD_DIR_CASE(48) PD_DIR_CASE(56)
        if constexpr (MAXM > 64) { PD_DIR_CASE(64) PD_DIR_CASE(80) PD_DIR_CASE(96) PD_DIR_CASE(112) }
        return dir_unit_run<Atom, MAXM, false, MAXM>(un, next, buf, b, dir, next_dir);
    }
    // (the 64-moment FP32 kernel is not launched where frames may have more)
    if constexpr (MAXM > 64 || sizeof(Atom) == sizeof(double4))
        return dir_unit_run<Atom, MAXM, true, MAXM>(un, next, buf, b, dir, next_dir);
    return b;
#undef PD_DIR_CASE
}

// Persistent blocks. plan_frames > 0: the units of every frame of one request
// (reqs[0]) are taken by number (counter[1]); 0: the jobs of any requests, each a
// share of its frame's units (every j1-th from j0 on). Frames in the other forms
// are passed over. Thread 0 draws the numbers and describes the next unit while the
// block sums the current one; a plan's frames (512 at a time) and chunks are kept in
// shared memory for that.
constexpr int DIR_FRAMES = 512, DIR_CHUNKS = 64;

template <class Atom, int MAXM>
__device__ __forceinline__ void dir_units(const PdJob *__restrict__ jobs,
                                          const int *__restrict__ n_jobs_ptr,
                                          const PdReqDev *__restrict__ reqs,
                                          int *__restrict__ counter, int plan_frames,
                                          Atom *__restrict__ buf) {
    __shared__ DirUnit s_unit[2];
    __shared__ __align__(16) double4 s_dir[2][PD_DIR_DIRS];
    __shared__ PdChunk s_chunk[DIR_CHUNKS];
    __shared__ unsigned s_end[DIR_FRAMES], s_warp[PD_WARPS];  // units of the frames up to each
    __shared__ int s_shape[DIR_FRAMES];                       // n_grp · 512 + n_amp
    constexpr int MBLOCK = sizeof(Atom) == sizeof(double4) ? PD_DIR_MBLOCK64 : PD_DIR_MBLOCK;
    // the units that next_unit describes (thread 0 only; false: no more), one after
    // the other
    auto run = [&](auto next_unit) {
        if (threadIdx.x == 0) s_unit[0].ok = next_unit(s_unit[0]);
        __syncthreads();
        if (!s_unit[0].ok) return;
        int p = 0, b = 0;
        dir_stage_first(buf, s_dir[0], s_unit[0]);
        dir_stage_end();
        for (;; p ^= 1) {
            if (threadIdx.x == 0) s_unit[p ^ 1].ok = next_unit(s_unit[p ^ 1]);
            __syncthreads();
            b = dir_unit<Atom, MAXM>(s_unit[p], s_unit[p ^ 1], buf, b, s_dir[p], s_dir[p ^ 1]);
            if (!s_unit[p ^ 1].ok) break;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    };
    if (plan_frames > 0) {
        const PdReqDev &rq = reqs[0];
        const int n_chunk = rq.amp.n_chunk, nv2 = rq.amp.nv2;
        for (int k = threadIdx.x; k < min(n_chunk, DIR_CHUNKS); k += PD_THREADS)
            s_chunk[k] = rq.chunks[k];
        const PdChunk *chunks = n_chunk <= DIR_CHUNKS ? s_chunk : rq.chunks;
        unsigned cur = 0, base = 0;  // (cur: thread 0)
        if (threadIdx.x == 0) cur = static_cast<unsigned>(atomicAdd(&counter[1], 1));
        for (int f0 = 0; f0 < plan_frames; f0 += DIR_FRAMES) {
            const int nf = min(DIR_FRAMES, plan_frames - f0);
            constexpr int PER = DIR_FRAMES / PD_THREADS;
            unsigned own[PER], sum = 0;  // PER frames of each thread, then an inclusive scan
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const int f = threadIdx.x * PER + k;
                int n_grp = 0, n_amp = 0;
                if (f < nf) {
                    n_grp = rq.frames[f0 + f].n_grp;
                    n_amp = rq.frames[f0 + f].n_amp;
                }
                if (n_grp > 0)
                    sum += dir_unit_count(n_chunk, nv2, (n_amp + MBLOCK - 1) / MBLOCK, n_grp);
                own[k] = sum;
                s_shape[f] = n_grp * 512 + n_amp;
            }
            const int lane = threadIdx.x & 31;
            unsigned scan = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned v = __shfl_up_sync(0xffffffffu, scan, o);
                if (lane >= o) scan += v;
            }
            if (lane == 31) s_warp[threadIdx.x >> 5] = scan;
            __syncthreads();
            unsigned before = base + scan - sum, total = base;
#pragma unroll
            for (int w = 0; w < PD_WARPS; ++w) {
                if (w < static_cast<int>(threadIdx.x >> 5)) before += s_warp[w];
                total += s_warp[w];
            }
#pragma unroll
            for (int k = 0; k < PER; ++k) s_end[threadIdx.x * PER + k] = before + own[k];
            __syncthreads();
            int f = 0;
            run([&](DirUnit &d) {
                if (cur >= total) return false;
                while (cur >= s_end[f]) ++f;
                dir_unit_set<Atom>(d, rq, chunks, f0 + f, s_shape[f] / 512, s_shape[f] % 512,
                                   cur - (f ? s_end[f - 1] : base));
                cur = static_cast<unsigned>(atomicAdd(&counter[1], 1));
                return true;
            });
            base = total;
            __syncthreads();  // the tables are read
        }
        return;
    }
    const int n_jobs = *n_jobs_ptr;
    PdJob jb{};
    unsigned u = 0, n_units = 0;
    int n_grp = 0, n_amp = 0;
    run([&](DirUnit &d) {
        while (u >= n_units) {
            const int jid = atomicAdd(counter, 1);
            if (jid >= n_jobs) return false;
            jb = jobs[jid];
            const PdReqDev &rq = reqs[jb.req];
            n_grp = rq.frames[jb.frame].n_grp;
            n_amp = rq.frames[jb.frame].n_amp;
            n_units = n_grp == 0 ? 0
                                 : dir_unit_count(rq.amp.n_chunk, rq.amp.nv2,
                                                  (n_amp + MBLOCK - 1) / MBLOCK, n_grp);
            u = jb.j0;
        }
        const PdReqDev &rq = reqs[jb.req];
        dir_unit_set<Atom>(d, rq, rq.chunks, jb.frame, n_grp, n_amp, u);
        u += jb.j1;
        return true;
    });
}

template <int MAXM>
__global__ void __launch_bounds__(PD_THREADS, MAXM <= 64 ? 4 : 3)
    pd_directions_fp32(const PdJob *__restrict__ jobs, const int *__restrict__ n_jobs_ptr,
                       const PdReqDev *__restrict__ reqs, int *__restrict__ counter,
                       int plan_frames) {
    chain_enter();
    extern __shared__ __align__(128) float4 s_buf[];
    dir_units<float4, MAXM>(jobs, n_jobs_ptr, reqs, counter, plan_frames, s_buf);
}

__global__ void __launch_bounds__(PD_THREADS, 2)
    pd_directions_fp64(const PdJob *__restrict__ jobs, const int *__restrict__ n_jobs_ptr,
                       const PdReqDev *__restrict__ reqs, int *__restrict__ counter,
                       int plan_frames) {
    chain_enter();
    extern __shared__ __align__(128) float4 s_buf[];
    dir_units<double4, PD_DIR_MBLOCK64>(jobs, n_jobs_ptr, reqs, counter, plan_frames,
                                        reinterpret_cast<double4 *>(s_buf));
}

namespace {
template <class Kernel>
int prepared_blocks(Kernel k, int smem) {
    if (smem > 0 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
                        cudaSuccess)
        return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, PD_THREADS, smem) != cudaSuccess)
        return 0;
    return n;
}
}  // namespace

int directions_variant(int precision, int32_t n_amp) {
    return precision == 1 ? 0 : (n_amp <= 64 ? 64 : 128);
}

int directions_blocks_per_sm(int variant) {
    if (variant == 0) return prepared_blocks(pd_directions_fp64, DIR_SMEM64);
    if (variant == 64) return prepared_blocks(pd_directions_fp32<64>, dir_smem_bytes<64>());
    return prepared_blocks(pd_directions_fp32<128>, dir_smem_bytes<128>());
}

cudaError_t launch_directions(int variant, const PdJob *jobs, const int *n_jobs,
                              const PdReqDev *reqs, int *counter, int plan_frames, int grid,
                              cudaStream_t st, bool after) {
    if (variant == 0)
        return chain_launch(after, pd_directions_fp64, grid, PD_THREADS, DIR_SMEM64, st, jobs,
                            n_jobs, reqs, counter, plan_frames);
    if (variant == 64)
        return chain_launch(after, pd_directions_fp32<64>, grid, PD_THREADS, dir_smem_bytes<64>(),
                            st, jobs, n_jobs, reqs, counter, plan_frames);
    return chain_launch(after, pd_directions_fp32<128>, grid, PD_THREADS, dir_smem_bytes<128>(), st,
                        jobs, n_jobs, reqs, counter, plan_frames);
}

}  // namespace pd
