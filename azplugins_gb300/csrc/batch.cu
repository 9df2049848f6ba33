// batch.cu -- many independent systems advanced together (azp_batch).
//
// S replicas of uneven size, each with its own periodic box, pair parameters and
// RNG seed, are packed into one particle array (replica r owns the index range
// [off_r, off_r + N_r) after every re-sort) and advanced by ONE fused force +
// Langevin launch per timestep for all replicas together, replayed from a CUDA
// graph; a list rebuild for all replicas runs as a graph conditional node when
// any particle of any replica moved more than r_buff / 2.
//
// Replicas never see each other: every replica has its own cell grid (global
// cell index = the replica's cell offset + its local cell), so candidate cells of
// a particle belong to its own replica only. Positions of replica r are stored as
// fixed-point fractions of ITS box, so the integer difference is its minimum
// image. Tags are per replica (0 .. N_r - 1) and the seed is the replica's: each
// replica draws exactly the noise it would draw run alone.
//
// One particle type per replica; pair potentials as in the single-system engine
// (the arithmetic of evaluators.cuh, FP32 forces with FP64 integration or FP64).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <new>
#include <utility>
#include <vector>

#include "celllist.cuh"
#include "evaluators.cuh"
#include "integrate.cuh"
#include "pair.cuh"
#include "scan.cuh"

namespace azp
{
struct SysInfo {
    double L[3], Linv[3], lo[3], hi[3], fscale[3];
    float sfix[3];
    float list_lo, list_hi;   // FP32 list prefilter thresholds
    double rlistsq;           // exact list decision
    double rcutsq;
    uint32_t cell_off;
    int dim[3];
    int reach[3];
    double cscale[3];         // dim / L
    uint32_t seed;
    uint32_t off, n;          // the replica's particles: [off, off + n)
    uint32_t far_cells;       // every axis has 2 reach + 3 cells or more (k_b_nlist)
    float recf[PAIR_TBL];     // rec and rcutsq as the FP32 step reads them
    float rcutf;
    double rec[PAIR_TBL];     // pair kernel record + cut record (one type)
};

constexpr int BATCH_BLOCK = 256;      // default threads per block of the fused step
constexpr int BATCH_BLOCK_MAX = 512;  // largest block azp_batch_set_block accepts

// ---------------------------------------------------------------- rebuild kernels
__global__ void k_b_zero(uint32_t* __restrict__ p, uint32_t n, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = 0u;
}

__device__ __forceinline__ int b_cell_coord(double x, double lo, double scale, int dim)
{
    int c = (int)floor((x - lo) * scale);
    if (c < 0) c += dim;
    if (c >= dim) c -= dim;
    return min(max(c, 0), dim - 1);
}

__global__ void k_b_assign(const double4_32a* __restrict__ pos, const uint16_t* __restrict__ sys, uint32_t N,
                           const SysInfo* __restrict__ info, uint32_t* __restrict__ cell_of,
                           uint32_t* __restrict__ slot, uint32_t* __restrict__ cell_count,
                           const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const SysInfo& si = info[sys[i]];
    const double4_32a p = pos[i];
    const int cx = b_cell_coord(p.x, si.lo[0], si.cscale[0], si.dim[0]);
    const int cy = b_cell_coord(p.y, si.lo[1], si.cscale[1], si.dim[1]);
    const int cz = b_cell_coord(p.z, si.lo[2], si.cscale[2], si.dim[2]);
    const uint32_t c = si.cell_off + ((uint32_t)cz * si.dim[1] + cy) * si.dim[0] + cx;
    cell_of[i] = c;
    slot[i] = atomicAdd(&cell_count[c], 1u);
}

__global__ void k_b_scatter(const uint32_t* __restrict__ cell_of, const uint32_t* __restrict__ slot,
                            const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ members, uint32_t N,
                            const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    members[cell_start[cell_of[i]] + slot[i]] = i;
}

// each cell's members sorted by index (deterministic order): one warp per 32
// consecutive cells, a lane per cell for small cells, the whole warp for crowded ones
__global__ void __launch_bounds__(kSortWarps * 32) k_b_cell_sort(const uint32_t* __restrict__ cell_start,
                                                                 uint32_t* __restrict__ members, uint32_t ncell,
                                                                 const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    __shared__ uint32_t s_rows[kSortWarps][kMaxSortedCell];
    sort_cells_warp(cell_start, members, ncell, s_rows[threadIdx.x >> 5], blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
}

__global__ void __launch_bounds__(kSortWarps * 32) k_b_cell_sort_crowded(const uint32_t* __restrict__ cell_start,
                                                                         uint32_t* __restrict__ members,
                                                                         uint32_t ncell,
                                                                         const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    __shared__ uint32_t s_rows[kSortWarps][kMaxSortedCell];
    sort_cell_per_warp(cell_start, members, ncell, s_rows[threadIdx.x >> 5], blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
}

struct BPerm {
    const uint32_t* members;
    double4_32a *pos, *t_pos, *vel, *t_vel;
    double *accel, *t_accel;
    int *image, *t_image;
    uint32_t *tag, *t_tag;
    uint16_t *sys, *t_sys;
    uint32_t *cell_of, *t_cell;
    uint32_t N;
};

__global__ void k_b_gather(BPerm a, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.N) return;
    const uint32_t o = a.members[s];
    a.t_pos[s] = a.pos[o];
    a.t_vel[s] = a.vel[o];
    for (int d = 0; d < 3; ++d) {
        a.t_accel[3 * s + d] = a.accel[3 * o + d];
        a.t_image[3 * s + d] = a.image[3 * o + d];
    }
    a.t_tag[s] = a.tag[o];
    a.t_sys[s] = a.sys[o];
    a.t_cell[s] = a.cell_of[o];
}

__global__ void k_b_back(BPerm a, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= a.N) return;
    a.pos[s] = a.t_pos[s];
    a.vel[s] = a.t_vel[s];
    for (int d = 0; d < 3; ++d) {
        a.accel[3 * s + d] = a.t_accel[3 * s + d];
        a.image[3 * s + d] = a.t_image[3 * s + d];
    }
    a.tag[s] = a.t_tag[s];
    a.sys[s] = a.t_sys[s];
    a.cell_of[s] = a.t_cell[s];
}

__global__ void k_b_fixed(const double4_32a* __restrict__ pos, const uint16_t* __restrict__ sys, uint32_t N,
                          const SysInfo* __restrict__ info, uint4* __restrict__ fa, uint4* __restrict__ fb,
                          const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const SysInfo& si = info[sys[i]];
    const double4_32a p = pos[i];
    uint4 f;
    f.x = to_fixed(p.x, si.Linv[0]);
    f.y = to_fixed(p.y, si.Linv[1]);
    f.z = to_fixed(p.z, si.Linv[2]);
    f.w = sys[i];
    fa[i] = f;
    fb[i] = f;
}

// The list, a warp per B_CHUNK consecutive particles, those of one cell at a time. The
// stencil rows of the cell are laid end to end (nlist_chunk has the same walk) and taken 32
// candidates a step, each loaded once and tested against every particle of the chunk; a
// ballot ranks the hits, which go to the particles' rows side by side. Coordinates are
// floats relative to the chunk's first particle (an integer conversion per candidate, not
// per test); where an axis has fewer than 2 reach + 3 cells the difference is wrapped once
// more. |coordinate| <= L / 2 <= 2.5 r_list there, which the band around r_list
// (make_list_cuts, 5e-6) covers: both coordinates' roundings come to 2.1e-6 of r^2. Chunks
// with a particle that was clamped into its cell (word_in_cell) form the differences pair by
// pair.
// Bound by issue (14 or 23 instructions a test) at 22 % of the warps (114 registers). A
// build of 48 replicas (337,467 particles, 94 M entries), all kernels, takes 1,760 us so and
// took 3,115 with one thread per particle and a column of the list each, with 32 lanes on
// rows of 15 to 2,800 entries.
constexpr int B_CHUNK = 8;
// The list: entry k of particle i. Blocks of 16 entries, the particles' side by side: a
// pass of the step reads one block of each of its particles, and what is in use of the
// list is compact whatever the longest row. Whole rows one after the other, at 3,700
// entries each, spread 0.4 GB of entries over 5 GB and its pages: 390 us a step for 48
// replicas against 360 so (the list build, which writes a row in several places, takes 15 %
// longer; there are about 18 steps to a build).
constexpr uint32_t B_LIST_BLOCK = 16;
AZP_D size_t b_entry(uint32_t i, uint32_t k, uint32_t N)
{
    return ((size_t)(k / B_LIST_BLOCK) * N + i) * B_LIST_BLOCK + k % B_LIST_BLOCK;
}
constexpr int B_NL_WARPS = 4;
constexpr uint32_t B_RANGES = 2 * 3 * 3;  // stencil rows and their wrapped parts
constexpr int B_NEAR = 0, B_WRAP = 1, B_PAIR = 2;  // as they are, wrapped once more, or pair by pair
template<int FORM>
AZP_D uint32_t b_walk(const uint4* __restrict__ fixed, const double4_32a* __restrict__ pos, const SysInfo& si,
                      const uint2* range, uint32_t total, uint32_t first, uint32_t cnt, uint32_t* __restrict__ nbrs,
                      uint32_t N, uint32_t max_nn)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const float sx = si.sfix[0], sy = si.sfix[1], sz = si.sfix[2];
    const float Lx = sx * 4294967296.0f, Ly = sy * 4294967296.0f, Lz = sz * 4294967296.0f;
    const float ix = 1.0f / Lx, iy = 1.0f / Ly, iz = 1.0f / Lz;
    const float hi = si.list_hi, lo = si.list_lo;
    const uint4 ref = fixed[first];
    float px[B_CHUNK], py[B_CHUNK], pz[B_CHUNK];
    uint32_t n[B_CHUNK];
#pragma unroll
    for (int p = 0; p < B_CHUNK; ++p) {
        const uint4 f = fixed[first + min((uint32_t)p, cnt - 1u)];
        px[p] = (float)(int32_t)(f.x - ref.x) * sx;
        py[p] = (float)(int32_t)(f.y - ref.y) * sy;
        pz[p] = (float)(int32_t)(f.z - ref.z) * sz;
        n[p] = 0u;
    }
    uint32_t q = 0u;
    const auto slot_of = [&](uint32_t c) -> uint32_t {
        while (range[q + 1u].x <= c) ++q;
        const uint2 r = range[q];
        return r.y + (c - r.x);
    };
    uint32_t j = lane < total ? slot_of(lane) : 0u;
    uint4 w = fixed[j];
    for (uint32_t c0 = 0; c0 < total; c0 += 32u) {
        const bool on = c0 + lane < total;
        const uint4 wc = w;
        const uint32_t jc = j;
        if (c0 + 32u + lane < total) {
            j = slot_of(c0 + 32u + lane);
            w = fixed[j];
        }
        const float qx = (float)(int32_t)(wc.x - ref.x) * sx;
        const float qy = (float)(int32_t)(wc.y - ref.y) * sy;
        const float qz = (float)(int32_t)(wc.z - ref.z) * sz;
        // a lane without a candidate hits nothing
        const float hi_l = on ? hi : -1.0f;
#pragma unroll
        for (int p = 0; p < B_CHUNK; ++p) {
            if (p >= (int)cnt) break;
            float dx = px[p] - qx, dy = py[p] - qy, dz = pz[p] - qz;
            if constexpr (FORM == B_PAIR) {
                const uint4 f = fixed[first + (uint32_t)p];
                dx = (float)(int32_t)(f.x - wc.x) * sx;
                dy = (float)(int32_t)(f.y - wc.y) * sy;
                dz = (float)(int32_t)(f.z - wc.z) * sz;
            } else if constexpr (FORM == B_WRAP) {
                dx = fmaf(-Lx, rintf(dx * ix), dx);
                dy = fmaf(-Ly, rintf(dy * iy), dy);
                dz = fmaf(-Lz, rintf(dz * iz), dz);
            }
            const float rs = dx * dx + dy * dy + dz * dz;
            const uint32_t i = first + (uint32_t)p;
            bool hit = (rs < hi_l) & (jc != i);
            if (hit && !(rs < lo)) {
                // inside the band: the exact FP64 decision
                const double4_32a pi = pos[i];
                const double4_32a pj = pos[jc];
                const double vx = min_image1(pi.x - pj.x, si.L[0], si.Linv[0]);
                const double vy = min_image1(pi.y - pj.y, si.L[1], si.Linv[1]);
                const double vz = min_image1(pi.z - pj.z, si.L[2], si.Linv[2]);
                hit = rsq_exact(vx, vy, vz) < si.rlistsq;
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, hit);
            const uint32_t k = n[p] + __popc(hits & lt);
            if (hit && k < max_nn) nbrs[b_entry(i, k, N)] = jc;
            n[p] += __popc(hits);
        }
    }
    uint32_t mine = 0u;
#pragma unroll
    for (int p = 0; p < B_CHUNK; ++p)
        if (p == (int)lane) mine = n[p];
    return mine;
}

// out of line: its registers do not count against the others
static __device__ __noinline__ uint32_t b_walk_pairs(const uint4* fixed, const double4_32a* pos, const SysInfo& si,
                                                     const uint2* range, uint32_t total, uint32_t first, uint32_t cnt,
                                                     uint32_t* nbrs, uint32_t N, uint32_t max_nn)
{
    return b_walk<B_PAIR>(fixed, pos, si, range, total, first, cnt, nbrs, N, max_nn);
}

__global__ void __launch_bounds__(B_NL_WARPS * 32)
    k_b_nlist(const double4_32a* __restrict__ pos, const uint4* __restrict__ fixed, uint32_t N,
              const SysInfo* __restrict__ info, const uint32_t* __restrict__ cell_start,
              const uint32_t* __restrict__ cell_of, uint32_t* __restrict__ counts, uint32_t* __restrict__ nbrs,
              uint32_t max_nn, uint32_t* __restrict__ maxcount, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    __shared__ uint2 s_range[B_NL_WARPS][B_RANGES + 1];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint2* range = s_range[warp];
    const uint32_t s_begin = (blockIdx.x * B_NL_WARPS + warp) * B_CHUNK;
    if (s_begin >= N) return;
    const uint32_t s_end = min(s_begin + B_CHUNK, N);
    for (uint32_t sa = s_begin; sa < s_end;) {
        // the particles from sa on that share its cell (and with it the replica)
        const uint32_t my_cell = cell_of[min(sa + lane, s_end - 1u)];
        const uint32_t cc = __shfl_sync(0xffffffffu, my_cell, 0);
        const uint32_t same = __ballot_sync(0xffffffffu, my_cell == cc && sa + lane < s_end);
        const uint32_t cnt = (uint32_t)__ffs(~same) - 1u;  // B_CHUNK < 32: some lane is off
        const SysInfo& si = info[fixed[sa].w];
        const int ncx = si.dim[0], ncy = si.dim[1], ncz = si.dim[2];
        const int r0 = si.reach[0], r1 = si.reach[1], r2 = si.reach[2];
        const uint32_t c = cc - si.cell_off;
        const int cx = (int)(c % (uint32_t)ncx);
        const int cy = (int)((c / (uint32_t)ncx) % (uint32_t)ncy);
        const int cz = (int)(c / ((uint32_t)ncx * (uint32_t)ncy));
        // the x-cells of a stencil row in their order: one slot range, or two at a face
        const int x0 = cx - r0, x1 = cx + r0;
        const int b0 = x0 < 0 ? ncx + x0 : x0, e0 = x0 < 0 || x1 >= ncx ? ncx - 1 : x1;
        const int e1 = x1 >= ncx ? x1 - ncx : x1;  // the second range begins at cell 0
        const uint32_t parts = x0 < 0 || x1 >= ncx ? 2u : 1u;
        const uint32_t ny = 2u * r1 + 1u;
        const uint32_t nr = ny * (2u * r2 + 1u) * parts;
        uint32_t total = 0u;
        for (uint32_t q0 = 0; q0 < nr; q0 += 32u) {
            const uint32_t q = q0 + lane;
            uint32_t sb = 0u, len = 0u;
            if (q < nr) {
                const uint32_t row = q / parts, part = q - row * parts;
                int oz = cz - r2 + (int)(row / ny), oy = cy - r1 + (int)(row % ny);
                oz += (oz < 0) ? ncz : 0;
                oz -= (oz >= ncz) ? ncz : 0;
                oy += (oy < 0) ? ncy : 0;
                oy -= (oy >= ncy) ? ncy : 0;
                const uint32_t rb = si.cell_off + ((uint32_t)oz * ncy + oy) * ncx;
                sb = cell_start[rb + (part ? 0 : b0)];
                len = cell_start[rb + (part ? e1 : e0) + 1] - sb;
            }
            uint32_t sum = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
                if ((int)lane >= o) sum += v;
            }
            if (q < nr) range[q] = make_uint2(total + sum - len, sb);
            total += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0u) range[nr] = make_uint2(0xffffffffu, 0u);
        __syncwarp();
        const uint4 mine = fixed[min(sa + lane, s_end - 1u)];
        const bool in_cell = lane >= cnt || (word_in_cell(mine.x, cx, ncx) && word_in_cell(mine.y, cy, ncy) &&
                                             word_in_cell(mine.z, cz, ncz));
        const uint32_t n = !__all_sync(0xffffffffu, in_cell)
                               ? b_walk_pairs(fixed, pos, si, range, total, sa, cnt, nbrs, N, max_nn)
                           : si.far_cells ? b_walk<B_NEAR>(fixed, pos, si, range, total, sa, cnt, nbrs, N, max_nn)
                                          : b_walk<B_WRAP>(fixed, pos, si, range, total, sa, cnt, nbrs, N, max_nn);
        if (lane < cnt) {
            counts[sa + lane] = n;
            if (n > max_nn) atomicMax(maxcount, n);
        }
        __syncwarp();
        sa += cnt;
    }
}

// The list with a thread per particle: the same entries in the same order. For batches of
// many particles with rows of about one length (b_plan), where no lane waits for another
// and a warp's chunk of a few particles only leaves lanes without a candidate. Microseconds
// a step with its list builds, a warp per chunk and a thread per particle:
//   N = 400,000, rows of 7 (1,000,000) / 17 / 32 / 59 / 110: 226 and 155 / 111 and 93 /
//   125 and 112 / 190 and 166 / 313 and 268; N = 160,000, 7 / 32 / 59: 54 and 44 / 65 and 60 /
//   91 and 86; N = 40,000: 30 and 28 / 35 and 37 / 44 and 49; N = 4,000, 32: 22 and 26.
__global__ void __launch_bounds__(128)
    k_b_nlist_threads(const double4_32a* __restrict__ pos, const uint4* __restrict__ fixed, uint32_t N,
                      const SysInfo* __restrict__ info, const uint32_t* __restrict__ cell_start,
                      const uint32_t* __restrict__ cell_of, uint32_t* __restrict__ counts, uint32_t* __restrict__ nbrs,
                      uint32_t max_nn, uint32_t* __restrict__ maxcount, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const uint4 fi = fixed[i];
    const SysInfo& si = info[fi.w];
    const float sx = si.sfix[0], sy = si.sfix[1], sz = si.sfix[2], hi = si.list_hi, lo = si.list_lo;
    const int ncx = si.dim[0], ncy = si.dim[1], ncz = si.dim[2];
    const int r0 = si.reach[0], r1 = si.reach[1], r2 = si.reach[2];
    const uint32_t c = cell_of[i] - si.cell_off;
    const int cx = (int)(c % (uint32_t)ncx);
    const int cy = (int)((c / (uint32_t)ncx) % (uint32_t)ncy);
    const int cz = (int)(c / ((uint32_t)ncx * (uint32_t)ncy));
    // the x-cells of a stencil row in their order: one slot range, or two at a face
    const int x0 = cx - r0, x1 = cx + r0;
    const bool two = x0 < 0 || x1 >= ncx;
    const int b0 = x0 < 0 ? ncx + x0 : x0, e0 = two ? ncx - 1 : x1;
    const int e1 = x1 >= ncx ? x1 - ncx : x1;
    uint32_t n = 0u;
    for (int oz = cz - r2; oz <= cz + r2; ++oz) {
        const int nz = oz < 0 ? oz + ncz : (oz >= ncz ? oz - ncz : oz);
        for (int oy = cy - r1; oy <= cy + r1; ++oy) {
            const int ny = oy < 0 ? oy + ncy : (oy >= ncy ? oy - ncy : oy);
            const uint32_t rb = si.cell_off + ((uint32_t)nz * ncy + ny) * ncx;
            for (int part = 0; part < (two ? 2 : 1); ++part) {
                const uint32_t sb = cell_start[rb + (part ? 0 : b0)], se = cell_start[rb + (part ? e1 : e0) + 1];
                for (uint32_t j = sb; j < se; ++j) {
                    const uint4 fj = fixed[j];
                    const float dx = (float)(int32_t)(fi.x - fj.x) * sx;
                    const float dy = (float)(int32_t)(fi.y - fj.y) * sy;
                    const float dz = (float)(int32_t)(fi.z - fj.z) * sz;
                    const float rs = dx * dx + dy * dy + dz * dz;
                    if (!(rs < hi) || j == i) continue;
                    if (!(rs < lo)) {
                        // inside the band: the exact FP64 decision
                        const double4_32a pi = pos[i];
                        const double4_32a pj = pos[j];
                        const double vx = min_image1(pi.x - pj.x, si.L[0], si.Linv[0]);
                        const double vy = min_image1(pi.y - pj.y, si.L[1], si.Linv[1]);
                        const double vz = min_image1(pi.z - pj.z, si.L[2], si.Linv[2]);
                        if (!(rsq_exact(vx, vy, vz) < si.rlistsq)) continue;
                    }
                    if (n < max_nn) nbrs[b_entry(i, n, N)] = j;
                    ++n;
                }
            }
        }
    }
    counts[i] = n;
    if (n > max_nn) atomicMax(maxcount, n);
}

__global__ void k_b_finish(uint32_t* __restrict__ flags, const uint32_t* __restrict__ gate)
{
    if (gated_off(gate)) return;
    flags[0] = 0u;
    flags[2] += 1u;
}

__global__ void k_b_arm(const uint32_t* __restrict__ flags, cudaGraphConditionalHandle h)
{
    cudaGraphSetConditional(h, (flags[0] && !flags[1]) ? 1u : 0u);
}

// ---------------------------------------------------------------- fused step
struct BStep {
    const double4_32a* pos;
    double4_32a* pos_next;
    const uint4* fix;
    uint4* fix_next;
    const uint4* fix_build;
    double4_32a* vel;
    double* accel;
    int* image;
    const uint32_t* tag;
    const uint16_t* sys;
    const SysInfo* info;
    uint32_t N;
    const uint32_t* counts;
    const uint32_t* nbrs;
    uint32_t max_nn;
    double dt, kT, gamma, noise;
    int noiseless;
    FlowD flow;
    const unsigned long long* d_ts;
    unsigned long long* d_ts_rw;
    uint32_t* flags;
    float disp_thresh2;
    int next;
    const uint2* work;  // per block: (replica | log2 of the lanes per particle << 16, first particle)
    uint32_t blocks;    // 0: a thread per particle instead
    int block;  // threads per block of the launch
    cudaGraphConditionalHandle next_cond;
    int set_cond;
};

// neighbours gathered per batch in the FP32-force pair loop
#ifndef AZP_B_BATCH
#define AZP_B_BATCH 4
#endif
constexpr int B_BATCH = AZP_B_BATCH;
// blocks of BATCH_BLOCK_MAX threads an SM holds (64 registers a thread at 2): the FP32
// step of the light evaluators is faster at 2, a few spilled words and all, than at the 70 or
// so registers the compiler takes at 1 (20 steps of 48 replicas: 9.3 and 11.2 ms); the others
// would spill more
template<class PE, typename R>
constexpr int b_min_blocks()
{
    return std::is_same<R, float>::value && !std::is_same<PE, Colloid>::value ? 2 : 1;
}

// particles a block of `block` threads takes at 2^lt lanes each: all its threads at once,
// but at least a warp's worth, so that the integration runs on full warps
AZP_HD uint32_t b_block_particles(uint32_t block, uint32_t lt) { return block >> lt > 32u ? block >> lt : 32u; }

// force / r of a pair in the FP32 step
template<class PE> AZP_D float b_force(const float* rec, float rsq)
{
    float fdr, e;
    if constexpr (std::is_same<PE, ExpandedYukawa>::value) PE::force_f(rec, rsq, fdr);
    else PE::eval(rec, rsq, fdr, e);
    return fdr;
}

// Langevin step two of particle i with the force f, and step one of the next timestep; whether
// the particle asks for a list build
template<typename R>
AZP_D bool b_integrate(const BStep& a, const SysInfo* si, uint32_t i, R fx, R fy, R fz)
{
    const unsigned long long ts = *a.d_ts;
    double4_32a p = a.pos[i];
    double4_32a v = a.vel[i];
    const uint32_t tg = a.tag[i];
    bool want = false, moved = false;
    if constexpr (std::is_same<R, double>::value) {
        double ux, uy, uz;
        flow_at(a.flow, p.y, ux, uy, uz);
        const double c = a.noiseless ? 0.0 : a.noise;
        double r0, r1, r2;
        uniform3(AZP_RNG_LANGEVIN_FLOW, ts, si->seed, tg, -c, c - (-c), r0, r1, r2);
        const double minv = 1.0 / v.w;
        const double ax = (fx + (r0 - a.gamma * (v.x - ux))) * minv;
        const double ay = (fy + (r1 - a.gamma * (v.y - uy))) * minv;
        const double az = (fz + (r2 - a.gamma * (v.z - uz))) * minv;
        const double h = 0.5 * a.dt;
        v.x += h * ax;
        v.y += h * ay;
        v.z += h * az;
        if (a.next) {
            p.x += (v.x + h * ax) * a.dt;
            p.y += (v.y + h * ay) * a.dt;
            p.z += (v.z + h * az) * a.dt;
            v.x += h * ax;
            v.y += h * ay;
            v.z += h * az;
            moved = true;
        } else {
            a.accel[3 * i] = ax;
            a.accel[3 * i + 1] = ay;
            a.accel[3 * i + 2] = az;
        }
    } else {
        float ux, uy, uz;
        flow_at_f(a.flow, (float)p.y, ux, uy, uz);
        const float c = a.noiseless ? 0.0f : (float)a.noise;
        const float g = (float)a.gamma, dt = (float)a.dt;
        float r0, r1, r2;
        uniform3f(AZP_RNG_LANGEVIN_FLOW, ts, si->seed, tg, -c, 2.0f * c, r0, r1, r2);
        const float minv = __frcp_rn((float)v.w);
        const float ax = (fx + (r0 - g * ((float)v.x - ux))) * minv;
        const float ay = (fy + (r1 - g * ((float)v.y - uy))) * minv;
        const float az = (fz + (r2 - g * ((float)v.z - uz))) * minv;
        if (a.next) {
            const float kx = dt * ax, ky = dt * ay, kz = dt * az;
            p.x += (double)(((float)v.x + kx) * dt);
            p.y += (double)(((float)v.y + ky) * dt);
            p.z += (double)(((float)v.z + kz) * dt);
            v.x += (double)kx;
            v.y += (double)ky;
            v.z += (double)kz;
            moved = true;
        } else {
            const float h = 0.5f * dt;
            v.x += (double)(h * ax);
            v.y += (double)(h * ay);
            v.z += (double)(h * az);
            a.accel[3 * i] = ax;
            a.accel[3 * i + 1] = ay;
            a.accel[3 * i + 2] = az;
        }
    }
    a.vel[i] = v;
    if (moved) {
        int w[3] = {0, 0, 0};
        wrap1(p.x, w[0], si->L[0], si->lo[0], si->hi[0]);
        wrap1(p.y, w[1], si->L[1], si->lo[1], si->hi[1]);
        wrap1(p.z, w[2], si->L[2], si->lo[2], si->hi[2]);
        if (w[0] | w[1] | w[2])
            for (int d = 0; d < 3; ++d) a.image[3 * i + d] += w[d];
        a.pos_next[i] = p;
        uint4 f;
        f.x = to_fixed(p.x, si->Linv[0]);
        f.y = to_fixed(p.y, si->Linv[1]);
        f.z = to_fixed(p.z, si->Linv[2]);
        f.w = a.sys[i];
        a.fix_next[i] = f;
        const uint4 fb = a.fix_build[i];
        const float ddx = (float)(int32_t)(f.x - fb.x) * si->sfix[0];
        const float ddy = (float)(int32_t)(f.y - fb.y) * si->sfix[1];
        const float ddz = (float)(int32_t)(f.z - fb.z) * si->sfix[2];
        want = ddx * ddx + ddy * ddy + ddz * ddz > a.disp_thresh2;
        if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) atomicOr(&a.flags[1], AZP_EBIT_NONFINITE);
    }
    return want;
}

// the last block to finish advances the timestep and arms the next build
AZP_D void b_finish_step(const BStep& a, bool want)
{
    if (__any_sync(0xffffffffu, want) && (threadIdx.x & 31) == 0) atomicOr(&a.flags[0], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t t = atomicAdd(&a.flags[4], 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            const uint32_t req = atomicAdd(&a.flags[0], 0u) && !atomicAdd(&a.flags[1], 0u);
            if (a.set_cond) cudaGraphSetConditional(a.next_cond, req ? 1u : 0u);
            a.flags[4] = 0u;
            *a.d_ts_rw = *a.d_ts_rw + 1ull;
        }
    }
}

// FP32 step: 2^B_LT lanes evaluate the pairs of a particle, B_TERMS entries of its row a
// pass, and leave their terms in shared memory; one lane per particle and axis then adds
// them in list order. The compensated addition is not free of its order (its product is
// fused into the first sum only), so the split of the evaluation leaves the force, and with
// it the trajectory, as one lane walking the row has it.
constexpr uint32_t B_LT = 2;
constexpr uint32_t B_TERMS = B_BATCH << B_LT;
constexpr uint32_t B_WARP_P = 32u >> B_LT;             // particles of a warp
constexpr uint32_t B_TERM_ROW = B_TERMS * 4u + 4u;     // floats: (dx, dy, dz, f / r) and a pad against bank conflicts
constexpr size_t b_step_smem(uint32_t block) { return (size_t)(block / 32u) * B_WARP_P * B_TERM_ROW * sizeof(float); }
static_assert(3 * B_WARP_P <= 32, "a lane per particle and axis");
static_assert(B_TERM_ROW % 4 == 0, "rows of 16-byte terms");
static_assert(B_BATCH == 4 && B_LIST_BLOCK % 4 == 0, "a batch is a 16-byte word of the list");
static_assert(B_TERMS == B_LIST_BLOCK, "a pass takes a block of the list");

// The fused step. A block takes particles of one replica; 2^lt lanes of a warp walk the
// row of one particle, in passes over the block's particles, and its first threads
// integrate them. Replicas differ by two orders of magnitude in the entries of a row; in
// FP64 lt belongs to the replica (b_plan).
// One thread per particle took 1,200 us a step for 48 replicas (94 M entries in FP32; its
// last warps walked 2,800 entries each, one lane a row), this 360. Bound by issue
// (about 100 instructions an entry) and the latency of the gathers.
template<class PE, typename R>
__global__ void __launch_bounds__(BATCH_BLOCK_MAX, (b_min_blocks<PE, R>())) k_b_step(BStep a)
{
    __shared__ R s_force[3][BATCH_BLOCK_MAX];
    extern __shared__ __align__(16) float s_terms[];
    const uint2 work = a.work[blockIdx.x];
    const SysInfo* si = a.info + (work.x & 0xffffu);
    const uint32_t lt = work.x >> 16;
    const uint32_t tpp = 1u << lt;
    const uint32_t np = min(b_block_particles(blockDim.x, lt), si->off + si->n - work.y);
    const uint32_t sub = threadIdx.x & (tpp - 1u);
    R rec[PAIR_TBL];
#pragma unroll
    for (int k = 0; k < PAIR_TBL; ++k) {
        if constexpr (std::is_same<R, double>::value)
            rec[k] = si->rec[k];
        else
            rec[k] = si->recf[k];
    }
    const bool on = PE::enabled(rec);
    for (uint32_t first = 0; first < np; first += blockDim.x >> lt) {
        const uint32_t q = first + (threadIdx.x >> lt);
        const bool active = q < np;
        const uint32_t i = work.y + (active ? q : 0u);
        const uint32_t n = active && on ? min(a.counts[i], a.max_nn) : 0u;
        [[maybe_unused]] R fx = 0, fy = 0, fz = 0;
        if constexpr (std::is_same<R, double>::value) {
            const double4_32a pi = a.pos[i];
            for (uint32_t k = sub; k < n; k += tpp) {
                const uint32_t j = a.nbrs[b_entry(i, k, a.N)];
                const double4_32a pj = a.pos[j];
                const double dx = min_image1(pi.x - pj.x, si->L[0], si->Linv[0]);
                const double dy = min_image1(pi.y - pj.y, si->L[1], si->Linv[1]);
                const double dz = min_image1(pi.z - pj.z, si->L[2], si->Linv[2]);
                const double rsq = rsq_exact(dx, dy, dz);
                if (!(rsq < si->rcutsq)) continue;
                double fdr, e;
                PE::eval(rec, rsq, fdr, e);
                fx += dx * fdr;
                fy += dy * fdr;
                fz += dz * fdr;
            }
        } else {
            const uint4 fi = a.fix[i];
            const float rc2 = si->rcutf;
            const float rc_lo = rc2 * 0.999996f, rc_hi = rc2 * 1.000004f;
            const float sx = si->sfix[0], sy = si->sfix[1], sz = si->sfix[2];
            const uint32_t lane = threadIdx.x & 31u;
            float* rows = s_terms + (threadIdx.x >> 5) * (B_WARP_P * B_TERM_ROW);
            float4* put = reinterpret_cast<float4*>(rows + (lane >> B_LT) * B_TERM_ROW) + sub;
            const float* get = rows + lane / 3u * B_TERM_ROW;
            const uint32_t axis = lane % 3u;
            const uint32_t nmax = __reduce_max_sync(0xffffffffu, n);
            Comp sum{0.f, 0.f};
            // the words of a pass gathered together, the list entries of the next loaded
            // meanwhile; the evaluator runs on every lane, at r_cut where a pair does not
            // count, so that the pairs of a lane overlap
            const uint32_t* block = a.nbrs + (size_t)i * B_LIST_BLOCK + sub;
            uint32_t jn[B_BATCH];
#pragma unroll
            for (int u = 0; u < B_BATCH; ++u) {
                const uint32_t k = (uint32_t)u << B_LT;
                jn[u] = k + sub < n ? __ldg(block + k) : i;
            }
            for (uint32_t kb = 0; kb < nmax; kb += B_TERMS) {
                uint32_t jj[B_BATCH];
                uint4 fj[B_BATCH];
#pragma unroll
                for (int u = 0; u < B_BATCH; ++u) jj[u] = jn[u];
#pragma unroll
                for (int u = 0; u < B_BATCH; ++u) fj[u] = __ldg(a.fix + jj[u]);
                block += (size_t)a.N * B_LIST_BLOCK;
#pragma unroll
                for (int u = 0; u < B_BATCH; ++u) {
                    const uint32_t k = (uint32_t)u << B_LT;
                    jn[u] = kb + B_TERMS + sub + k < n ? __ldg(block + k) : i;
                }
#pragma unroll
                for (int u = 0; u < B_BATCH; ++u) {
                    const float dx = (float)(int32_t)(fi.x - fj[u].x) * sx;
                    const float dy = (float)(int32_t)(fi.y - fj[u].y) * sy;
                    const float dz = (float)(int32_t)(fi.z - fj[u].z) * sz;
                    const float rsq = dx * dx + dy * dy + dz * dz;
                    bool in = rsq < rc_hi && jj[u] != i;
                    if (in && rsq >= rc_lo) {
                        const double4_32a pi = a.pos[i];
                        const double4_32a pj = a.pos[jj[u]];
                        const double vx = min_image1(pi.x - pj.x, si->L[0], si->Linv[0]);
                        const double vy = min_image1(pi.y - pj.y, si->L[1], si->Linv[1]);
                        const double vz = min_image1(pi.z - pj.z, si->L[2], si->Linv[2]);
                        in = rsq_exact(vx, vy, vz) < si->rcutsq;
                    }
                    const float fdr = b_force<PE>(rec, in ? rsq : rc2);
                    put[u << B_LT] = make_float4(dx, dy, dz, in ? fdr : 0.0f);
                }
                __syncwarp();
                if (lane < 3u * B_WARP_P) {
#pragma unroll
                    for (uint32_t m = 0; m < B_TERMS; ++m) sum.add(get[4u * m + axis] * get[4u * m + 3u]);
                }
                __syncwarp();
            }
            const uint32_t qs = first + (threadIdx.x >> 5) * B_WARP_P + lane / 3u;
            if (lane < 3u * B_WARP_P && qs < np) s_force[axis][qs] = sum.value();
        }
        if constexpr (std::is_same<R, double>::value) {
            for (uint32_t m = tpp >> 1; m > 0; m >>= 1) {
                fx += __shfl_xor_sync(0xffffffffu, fx, m);
                fy += __shfl_xor_sync(0xffffffffu, fy, m);
                fz += __shfl_xor_sync(0xffffffffu, fz, m);
            }
            if (active && sub == 0) {
                s_force[0][q] = fx;
                s_force[1][q] = fy;
                s_force[2][q] = fz;
            }
        }
    }
    __syncthreads();
    bool want = false;
    if (threadIdx.x < np) {
        const uint32_t i = work.y + threadIdx.x;
        const R fx = s_force[0][threadIdx.x], fy = s_force[1][threadIdx.x], fz = s_force[2][threadIdx.x];
        want = b_integrate(a, si, i, fx, fy, fz);
    }
    b_finish_step(a, want);
}

// The same with a thread per particle, which walks its row in words of four entries, adds the
// terms in list order and integrates: full warps however small the replicas are, and no
// lanes without an entry. For batches of many particles with rows of about one length
// (b_plan); the states are those of k_b_step (FP32: bitwise).
template<class PE, typename R>
__global__ void __launch_bounds__(BATCH_BLOCK_MAX) k_b_step_threads(BStep a)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool want = false;
    if (i < a.N) {
        const SysInfo* si = a.info + a.sys[i];
        R rec[PAIR_TBL];
#pragma unroll
        for (int k = 0; k < PAIR_TBL; ++k) {
            if constexpr (std::is_same<R, double>::value)
                rec[k] = si->rec[k];
            else
                rec[k] = si->recf[k];
        }
        const uint32_t n = PE::enabled(rec) ? min(a.counts[i], a.max_nn) : 0u;
        if constexpr (std::is_same<R, double>::value) {
            double fx = 0, fy = 0, fz = 0;
            const double4_32a pi = a.pos[i];
            for (uint32_t k = 0; k < n; ++k) {
                const uint32_t j = a.nbrs[b_entry(i, k, a.N)];
                const double4_32a pj = a.pos[j];
                const double dx = min_image1(pi.x - pj.x, si->L[0], si->Linv[0]);
                const double dy = min_image1(pi.y - pj.y, si->L[1], si->Linv[1]);
                const double dz = min_image1(pi.z - pj.z, si->L[2], si->Linv[2]);
                const double rsq = rsq_exact(dx, dy, dz);
                if (!(rsq < si->rcutsq)) continue;
                double fdr, e;
                PE::eval(rec, rsq, fdr, e);
                fx += dx * fdr;
                fy += dy * fdr;
                fz += dz * fdr;
            }
            want = b_integrate(a, si, i, fx, fy, fz);
        } else {
            Comp cx{0.f, 0.f}, cy{0.f, 0.f}, cz{0.f, 0.f};
            const uint4 fi = a.fix[i];
            const float rc2 = si->rcutf;
            const float rc_lo = rc2 * 0.999996f, rc_hi = rc2 * 1.000004f;
            const float sx = si->sfix[0], sy = si->sfix[1], sz = si->sfix[2];
            for (uint32_t kb = 0; kb < n; kb += B_BATCH) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(a.nbrs + b_entry(i, kb, a.N)));
                const uint32_t jj[4] = {q.x, kb + 1u < n ? q.y : i, kb + 2u < n ? q.z : i, kb + 3u < n ? q.w : i};
                uint4 fj[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) fj[u] = __ldg(a.fix + jj[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float dx = (float)(int32_t)(fi.x - fj[u].x) * sx;
                    const float dy = (float)(int32_t)(fi.y - fj[u].y) * sy;
                    const float dz = (float)(int32_t)(fi.z - fj[u].z) * sz;
                    const float rsq = dx * dx + dy * dy + dz * dz;
                    bool in = rsq < rc_hi && jj[u] != i;
                    if (in && rsq >= rc_lo) {
                        const double4_32a pi = a.pos[i];
                        const double4_32a pj = a.pos[jj[u]];
                        const double vx = min_image1(pi.x - pj.x, si->L[0], si->Linv[0]);
                        const double vy = min_image1(pi.y - pj.y, si->L[1], si->Linv[1]);
                        const double vz = min_image1(pi.z - pj.z, si->L[2], si->Linv[2]);
                        in = rsq_exact(vx, vy, vz) < si->rcutsq;
                    }
                    if (!in) continue;
                    const float fdr = b_force<PE>(rec, rsq);
                    cx.add(dx * fdr);
                    cy.add(dy * fdr);
                    cz.add(dz * fdr);
                }
            }
            want = b_integrate(a, si, i, cx.value(), cy.value(), cz.value());
        }
    }
    b_finish_step(a, want);
}

// Langevin step one in place at the start of a run
__global__ void k_b_step1(double4_32a* __restrict__ pos, uint4* __restrict__ fix, const uint4* __restrict__ fix_build,
                          double4_32a* __restrict__ vel, const double* __restrict__ accel, int* __restrict__ image,
                          const uint16_t* __restrict__ sys, const SysInfo* __restrict__ info, uint32_t N, double dt,
                          float thresh2, uint32_t* __restrict__ flags)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool want = false;
    if (i < N) {
        const SysInfo& si = info[sys[i]];
        double4_32a p = pos[i];
        double4_32a v = vel[i];
        const double h = 0.5 * dt;
        const double ax = accel[3 * i], ay = accel[3 * i + 1], az = accel[3 * i + 2];
        p.x += (v.x + h * ax) * dt;
        p.y += (v.y + h * ay) * dt;
        p.z += (v.z + h * az) * dt;
        int w[3] = {0, 0, 0};
        wrap1(p.x, w[0], si.L[0], si.lo[0], si.hi[0]);
        wrap1(p.y, w[1], si.L[1], si.lo[1], si.hi[1]);
        wrap1(p.z, w[2], si.L[2], si.lo[2], si.hi[2]);
        if (w[0] | w[1] | w[2])
            for (int d = 0; d < 3; ++d) image[3 * i + d] += w[d];
        v.x += h * ax;
        v.y += h * ay;
        v.z += h * az;
        pos[i] = p;
        vel[i] = v;
        uint4 f;
        f.x = to_fixed(p.x, si.Linv[0]);
        f.y = to_fixed(p.y, si.Linv[1]);
        f.z = to_fixed(p.z, si.Linv[2]);
        f.w = sys[i];
        fix[i] = f;
        const uint4 fb = fix_build[i];
        const float dx = (float)(int32_t)(f.x - fb.x) * si.sfix[0];
        const float dy = (float)(int32_t)(f.y - fb.y) * si.sfix[1];
        const float dz = (float)(int32_t)(f.z - fb.z) * si.sfix[2];
        want = dx * dx + dy * dy + dz * dz > thresh2;
    }
    if (__any_sync(0xffffffffu, want) && (threadIdx.x & 31) == 0) atomicOr(&flags[0], 1u);
}

__global__ void k_b_load(const double* __restrict__ pos_in, const double* __restrict__ vel_in,
                         const double* __restrict__ acc_in, const int* __restrict__ img_in,
                         const uint32_t* __restrict__ sys_of, const uint32_t* __restrict__ tag_of, uint32_t N,
                         double4_32a* __restrict__ pos, double4_32a* __restrict__ vel, double* __restrict__ acc,
                         int* __restrict__ img, uint32_t* __restrict__ tag, uint16_t* __restrict__ sys,
                         uint32_t* __restrict__ rindex)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    pos[i] = make_double4_32a(pos_in[4 * i], pos_in[4 * i + 1], pos_in[4 * i + 2], type_as_double(0u));
    vel[i] = make_double4_32a(vel_in[4 * i], vel_in[4 * i + 1], vel_in[4 * i + 2], vel_in[4 * i + 3]);
    for (int d = 0; d < 3; ++d) {
        acc[3 * i + d] = acc_in ? acc_in[3 * i + d] : 0.0;
        img[3 * i + d] = img_in ? img_in[3 * i + d] : 0;
    }
    tag[i] = tag_of[i];
    sys[i] = (uint16_t)sys_of[i];
    rindex[i] = i;
}

// device state -> packed order (replica offsets + tag)
__global__ void k_b_store(const double4_32a* __restrict__ pos, const double4_32a* __restrict__ vel,
                          const double* __restrict__ acc, const int* __restrict__ img, const uint32_t* __restrict__ tag,
                          const uint16_t* __restrict__ sys, const uint32_t* __restrict__ sys_off, uint32_t N,
                          double* __restrict__ pos_out, double* __restrict__ vel_out, double* __restrict__ acc_out,
                          int* __restrict__ img_out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const uint32_t o = sys_off[sys[i]] + tag[i];
    const double4_32a p = pos[i];
    const double4_32a v = vel[i];
    pos_out[4 * o] = p.x;
    pos_out[4 * o + 1] = p.y;
    pos_out[4 * o + 2] = p.z;
    pos_out[4 * o + 3] = 0.0;
    vel_out[4 * o] = v.x;
    vel_out[4 * o + 1] = v.y;
    vel_out[4 * o + 2] = v.z;
    vel_out[4 * o + 3] = v.w;
    for (int d = 0; d < 3; ++d) {
        acc_out[3 * o + d] = acc[3 * i + d];
        img_out[3 * o + d] = img[3 * i + d];
    }
}

template<class PE>
int launch_b_step(int precision, const BStep& a, cudaStream_t s)
{
    if (a.blocks == 0) {  // a thread per particle
        const uint32_t blocks = (a.N + (uint32_t)a.block - 1u) / (uint32_t)a.block;
        if (blocks == 0) return AZP_OK;
        if (precision == AZP_FP32)
            k_b_step_threads<PE, float><<<blocks, a.block, 0, s>>>(a);
        else
            k_b_step_threads<PE, double><<<blocks, a.block, 0, s>>>(a);
        AZP_CHECK_LAUNCH("k_b_step_threads");
        return AZP_OK;
    }
    if (precision == AZP_FP32)
        k_b_step<PE, float><<<a.blocks, a.block, b_step_smem((uint32_t)a.block), s>>>(a);
    else
        k_b_step<PE, double><<<a.blocks, a.block, 0, s>>>(a);
    AZP_CHECK_LAUNCH("k_b_step");
    return AZP_OK;
}

int launch_b_step_kind(int kind, int precision, const BStep& a, cudaStream_t s)
{
    switch (kind) {
    case AZP_PAIR_PERTURBED_LJ: return launch_b_step<PerturbedLJ>(precision, a, s);
    case AZP_PAIR_EXPANDED_YUKAWA: return launch_b_step<ExpandedYukawa>(precision, a, s);
    case AZP_PAIR_HERTZ: return launch_b_step<Hertz>(precision, a, s);
    case AZP_PAIR_COLLOID: return launch_b_step<Colloid>(precision, a, s);
    default: return AZP_ERR_INVALID;
    }
}

}  // namespace azp

using namespace azp;

constexpr int B_TPPS = 6, B_BLOCKS = 4;  // 1 to 32 lanes per particle, blocks of 64 to 512 threads

struct azp_batch {
    uint32_t S = 0, N = 0;
    std::vector<uint32_t> n_of, off;
    int precision = AZP_FP64, kind = 0, tpp = 1, block = BATCH_BLOCK;
    std::vector<double> row_len;  // expected list entries per particle, by replica
    bool alike = false;           // rows of about one length (b_plan)
    uint2* work = nullptr;        // blocks of the fused step (b_plan)
    // first entry and number of entries of work, by log2(tpp) and log2(block / 64)
    std::pair<size_t, uint32_t> plan[B_TPPS][B_BLOCKS];
    double dt = 0.005, kT = 1.0, gamma = 1.0, r_buff = 0.4;
    int noiseless = 0;
    FlowD flow{};
    SysInfo* info = nullptr;
    uint32_t* sys_off = nullptr;
    // state
    double4_32a* pos[2] = {nullptr, nullptr};
    uint4* fix[2] = {nullptr, nullptr};
    uint4* fix_build = nullptr;
    int cur = 0;
    double4_32a* vel = nullptr;
    double* accel = nullptr;
    int* image = nullptr;
    uint32_t* tag = nullptr;
    uint16_t* sys = nullptr;
    // temps
    double4_32a *t_pos = nullptr, *t_vel = nullptr;
    double* t_accel = nullptr;
    int* t_image = nullptr;
    uint32_t* t_tag = nullptr;
    uint16_t* t_sys = nullptr;
    uint32_t* t_cell = nullptr;
    // packed state on its way to the host
    double *o_pos = nullptr, *o_vel = nullptr, *o_accel = nullptr;
    int* o_image = nullptr;
    // cells / list
    uint32_t ncell = 0;
    uint32_t *cell_of = nullptr, *slot = nullptr, *cell_count = nullptr, *cell_start = nullptr, *members = nullptr,
             *scan_tmp = nullptr, *rindex = nullptr;
    uint32_t max_nn = 32;
    uint32_t *counts = nullptr, *nbrs = nullptr;
    uint32_t* flags = nullptr;
    unsigned long long* d_ts = nullptr;
    uint64_t launches = 0;
    bool have_state = false, use_graphs = true;
    cudaGraphExec_t gexec[2] = {nullptr, nullptr};
    cudaStream_t gstream = nullptr;
};

namespace
{
template<typename T> int balloc(T** p, size_t n)
{
    *p = nullptr;
    const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * (n ? n : 1));
    return e == cudaSuccess ? AZP_OK : record_cuda_error(e, "cudaMalloc (batch)");
}

void b_free_graphs(azp_batch* b)
{
    for (auto& g : b->gexec)
        if (g) {
            cudaGraphExecDestroy(g);
            g = nullptr;
        }
}

void b_free(azp_batch* b)
{
    b_free_graphs(b);
    void* ptrs[] = {b->info, b->sys_off, b->pos[0], b->pos[1], b->fix[0], b->fix[1], b->fix_build, b->vel, b->accel,
                    b->image, b->tag, b->sys, b->t_pos, b->t_vel, b->t_accel, b->t_image, b->t_tag, b->t_sys,
                    b->t_cell, b->cell_of, b->slot, b->cell_count, b->cell_start, b->members, b->scan_tmp,
                    b->rindex, b->counts, b->nbrs, b->flags, b->d_ts, b->work, b->o_pos, b->o_vel, b->o_accel, b->o_image};
    for (void* p : ptrs) cudaFree(p);
    if (b->gstream) cudaStreamDestroy(b->gstream);
}

uint32_t nblk(uint32_t n) { return (n + 255) / 256; }

// words of a particle's list row
uint32_t b_width(uint32_t max_nn) { return (max_nn + B_LIST_BLOCK - 1u) / B_LIST_BLOCK * B_LIST_BLOCK; }

// The blocks of the fused step, for every block size and number of lanes per particle that
// can be asked for, laid out once: azp_batch_set_tpp and azp_batch_set_block choose among
// them on the host, beside runs in flight, allocations that are not to be made and captures.
// FP32: 2^B_LT lanes. FP64: a replica takes the smallest power of two at which a lane walks
// at most per_lane entries of a row, 4 or more (narrower reads waste the sectors of a block),
// tpp or more; per_lane is 128, where fewer sums are combined and the rows of a warp are
// read together, and less while the lanes would not fill a quarter of the chip. Replicas
// with the longest rows go first, so that the last blocks are short.
// Rows of about one length (alike): the longest is not longer, against the mean, than the
// particles are many against a quarter of the chip's threads, so that a thread per particle
// keeps them busy to the end, and no row has more than 1,000 entries; or all are short and
// the replicas too small to fill the blocks that they would have to themselves. Then the
// list and the FP32 step go a thread per particle (k_b_nlist_threads, k_b_step_threads; no
// entries here), and the FP64 step, which the pipe bounds whatever the split, where rows
// are short besides and no lanes are asked
// for. Microseconds a step without list builds, lanes and thread per particle, replicas of
// 1,000 particles with rows of 5 / 20 / 61 / 132 / 500:
//   FP32 N =   4,000: 18 and 20 / 20 and 24 / 22 and 36 / 26 and 51 / 46 and 137
//        N =  40,000: 25 and 24 / 28 and 28 / 35 and 41 / 47 and 59 / 106 and 157
//        N = 400,000: 96 and 56 / 122 and 72 / 175 and 124 / 254 and 205 / 720 and 641
//   FP64 N =  40,000: 61 and 70 / 154 and 219 / 398 and 620 / 758 and 1,204
//        N = 400,000: 349 and 297 / 1,154 and 1,133 / 3,192 and 3,335
//   4,000 replicas of 50: FP32 57 and 38 / 66 and 46; FP64 229 and 193 / 645 and 629
//   4,096 replicas of 10: FP32 48 and 23; FP64 89 and 57
//   with list builds, FP32, longest row / mean: N = 120,000 64 / 48: 63 and 55; 115 / 73: 73 and
//   70; 345 / 94: 99 and 159; N = 400,000 115 / 40: 162 and 109; 345 / 63: 212 and 193;
//   N = 1,200,000 345 / 63: 572 and 366; N = 680,095 2,232 / 223: 735 and 907;
//   N = 1,320,729 2,898 / 291: 1,753 and 1,836
// 48 replicas of 337,467 particles with rows of 15 to 2,800: 360 and 1,200.
int b_plan(azp_batch* b)
{
    int dev = 0, sms = 1;
    AZP_CUDA_TRY(cudaGetDevice(&dev));
    AZP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    std::vector<uint32_t> order(b->S);
    for (uint32_t r = 0; r < b->S; ++r) order[r] = r;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return b->row_len[x] > b->row_len[y]; });
    double longest = 0.0, entries = 0.0;
    for (uint32_t r = 0; r < b->S; ++r) {
        longest = std::max(longest, b->row_len[r]);
        entries += b->row_len[r] * b->n_of[r];
    }
    b->alike = (longest <= 1000.0 && longest * 512.0 * sms <= entries) || (longest <= 64.0 && b->N < 32u * b->S);
    const bool threads = b->alike && (b->precision == AZP_FP32 || longest <= 24.0);
    std::vector<uint2> work;
    for (int kt = 0; kt < B_TPPS; ++kt) {
        double per_lane = 128.0;
        const auto lanes_log2 = [&](uint32_t r) {
            uint32_t lt = B_LT;
            if (b->precision == AZP_FP32) return lt;
            while (lt < 5 && (b->row_len[r] > per_lane * (1u << lt) || (int)lt < kt)) ++lt;
            return lt;
        };
        for (; per_lane > 8.0; per_lane *= 0.5) {
            size_t lanes = 0;
            for (uint32_t r = 0; r < b->S; ++r) lanes += (size_t)b->n_of[r] << lanes_log2(r);
            if (lanes >= (size_t)sms * 512) break;
        }
        const bool one = threads && (b->precision == AZP_FP32 || kt == 0);
        for (int kb = 0; kb < B_BLOCKS; ++kb) {
            if (kt > 0 && b->precision == AZP_FP32) {
                b->plan[kt][kb] = b->plan[0][kb];
                continue;
            }
            b->plan[kt][kb].first = work.size();
            b->plan[kt][kb].second = 0u;
            if (one) continue;
            for (uint32_t r : order) {
                const uint32_t lt = lanes_log2(r);
                const uint32_t per = b_block_particles(64u << kb, lt);
                for (uint32_t k = 0; k < b->n_of[r]; k += per) work.push_back(make_uint2(r | lt << 16, b->off[r] + k));
            }
            b->plan[kt][kb].second = (uint32_t)(work.size() - b->plan[kt][kb].first);
        }
    }
    const int st = balloc(&b->work, work.size());
    if (st) return st;
    AZP_CUDA_TRY(cudaMemcpy(b->work, work.data(), sizeof(uint2) * work.size(), cudaMemcpyHostToDevice));
    return AZP_OK;
}

int b_rebuild(azp_batch* b, cudaStream_t s, const uint32_t* gate)
{
    const uint32_t N = b->N;
    k_b_zero<<<std::min<uint32_t>(nblk(b->ncell), 1024), 256, 0, s>>>(b->cell_count, b->ncell, gate);
    k_b_assign<<<nblk(N), 256, 0, s>>>(b->pos[b->cur], b->sys, N, b->info, b->cell_of, b->slot, b->cell_count, gate);
    int st = exclusive_scan(b->cell_count, b->cell_start, b->ncell, b->scan_tmp, s, gate);
    if (st) return st;
    k_b_scatter<<<nblk(N), 256, 0, s>>>(b->cell_of, b->slot, b->cell_start, b->members, N, gate);
    if (crowded_grid(N, b->ncell))
        k_b_cell_sort_crowded<<<(b->ncell + kSortWarps - 1) / kSortWarps, kSortWarps * 32, 0, s>>>(
            b->cell_start, b->members, b->ncell, gate);
    else
        k_b_cell_sort<<<(b->ncell + 32 * kSortWarps - 1) / (32 * kSortWarps), kSortWarps * 32, 0, s>>>(
            b->cell_start, b->members, b->ncell, gate);
    BPerm p;
    p.members = b->members;
    p.pos = b->pos[b->cur];
    p.t_pos = b->t_pos;
    p.vel = b->vel;
    p.t_vel = b->t_vel;
    p.accel = b->accel;
    p.t_accel = b->t_accel;
    p.image = b->image;
    p.t_image = b->t_image;
    p.tag = b->tag;
    p.t_tag = b->t_tag;
    p.sys = b->sys;
    p.t_sys = b->t_sys;
    p.cell_of = b->cell_of;
    p.t_cell = b->t_cell;
    p.N = N;
    k_b_gather<<<nblk(N), 256, 0, s>>>(p, gate);
    k_b_back<<<nblk(N), 256, 0, s>>>(p, gate);
    k_b_fixed<<<nblk(N), 256, 0, s>>>(b->pos[b->cur], b->sys, N, b->info, b->fix[b->cur], b->fix_build, gate);
    constexpr uint32_t per_block = B_NL_WARPS * B_CHUNK;
    if (b->alike)
        k_b_nlist_threads<<<(N + 127u) / 128u, 128, 0, s>>>(b->pos[b->cur], b->fix[b->cur], N, b->info, b->cell_start, b->cell_of,
                                                           b->counts, b->nbrs, b->max_nn, b->flags + 3, gate);
    else
        k_b_nlist<<<(N + per_block - 1) / per_block, B_NL_WARPS * 32, 0, s>>>(
            b->pos[b->cur], b->fix[b->cur], N, b->info, b->cell_start, b->cell_of, b->counts, b->nbrs, b->max_nn, b->flags + 3, gate);
    k_b_finish<<<1, 1, 0, s>>>(b->flags, gate);
    AZP_CHECK_LAUNCH("b_rebuild");
    b->launches += 12;
    return AZP_OK;
}

BStep b_args(azp_batch* b)
{
    BStep a{};
    a.pos = b->pos[b->cur];
    a.pos_next = b->pos[b->cur ^ 1];
    a.fix = b->fix[b->cur];
    a.fix_next = b->fix[b->cur ^ 1];
    a.fix_build = b->fix_build;
    a.vel = b->vel;
    a.accel = b->accel;
    a.image = b->image;
    a.tag = b->tag;
    a.sys = b->sys;
    a.info = b->info;
    a.N = b->N;
    a.counts = b->counts;
    a.nbrs = b->nbrs;
    a.max_nn = b->max_nn;
    a.dt = b->dt;
    a.kT = b->kT;
    a.gamma = b->gamma;
    a.noise = std::sqrt(6.0 * b->gamma * b->kT / b->dt);
    a.noiseless = b->noiseless;
    a.flow = b->flow;
    a.d_ts = b->d_ts;
    a.d_ts_rw = b->d_ts;
    a.flags = b->flags;
    const double half = 0.5 * b->r_buff;
    a.disp_thresh2 = (float)(half * half * (1.0 - 1e-5));
    int kt = 0, kb = 0;
    while ((1 << kt) < b->tpp) ++kt;
    while ((64 << kb) < b->block) ++kb;
    a.work = b->work + b->plan[kt][kb].first;
    a.blocks = b->plan[kt][kb].second;
    a.block = b->block;
    return a;
}

int b_step(azp_batch* b, int next, cudaStream_t s, int set_cond, cudaGraphConditionalHandle h)
{
    BStep a = b_args(b);
    a.next = next;
    a.set_cond = set_cond;
    a.next_cond = h;
    b->launches += 1;
    return launch_b_step_kind(b->kind, b->precision, a, s);
}

int b_build_graph(azp_batch* b, int cur0, cudaGraphExec_t* out)
{
    cudaGraph_t g = nullptr;
    AZP_CUDA_TRY(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h[2];
    for (int k = 0; k < 2; ++k) AZP_CUDA_TRY(cudaGraphConditionalHandleCreate(&h[k], g, 0, cudaGraphCondAssignDefault));
    const int saved = b->cur;
    const uint64_t saved_l = b->launches;
    b->cur = cur0;
    cudaStream_t s = b->gstream;
    int st = AZP_OK;
    cudaGraphNode_t prev = nullptr;
    AZP_CUDA_TRY(cudaStreamBeginCaptureToGraph(s, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    k_b_arm<<<1, 1, 0, s>>>(b->flags, h[0]);
    cudaGraph_t tmp = nullptr;
    AZP_CUDA_TRY(cudaStreamEndCapture(s, &tmp));
    {
        size_t n = 0;
        AZP_CUDA_TRY(cudaGraphGetNodes(g, nullptr, &n));
        std::vector<cudaGraphNode_t> nodes(n);
        AZP_CUDA_TRY(cudaGraphGetNodes(g, nodes.data(), &n));
        prev = nodes.back();
    }
    for (int k = 0; k < 2 && st == AZP_OK; ++k) {
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h[k];
        cp.conditional.type = cudaGraphCondTypeIf;
        cp.conditional.size = 1;
        cudaGraphNode_t cnode;
        AZP_CUDA_TRY(cudaGraphAddNode(&cnode, g, &prev, nullptr, 1, &cp));
        AZP_CUDA_TRY(cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                   cudaStreamCaptureModeThreadLocal));
        st = b_rebuild(b, s, nullptr);
        AZP_CUDA_TRY(cudaStreamEndCapture(s, &tmp));
        if (st) break;
        AZP_CUDA_TRY(cudaStreamBeginCaptureToGraph(s, g, &cnode, nullptr, 1, cudaStreamCaptureModeThreadLocal));
        st = b_step(b, 1, s, k == 0 ? 1 : 0, k == 0 ? h[1] : 0);
        AZP_CUDA_TRY(cudaStreamEndCapture(s, &tmp));
        if (st) break;
        size_t nd = 0;
        AZP_CUDA_TRY(cudaGraphNodeGetDependentNodes(cnode, nullptr, nullptr, &nd));
        std::vector<cudaGraphNode_t> deps(nd);
        AZP_CUDA_TRY(cudaGraphNodeGetDependentNodes(cnode, deps.data(), nullptr, &nd));
        if (nd != 1) {
            st = AZP_ERR_CUDA;
            break;
        }
        prev = deps[0];
        b->cur ^= 1;
    }
    b->cur = saved;
    b->launches = saved_l;
    if (st == AZP_OK) {
        const cudaError_t e = cudaGraphInstantiate(out, g, 0);
        if (e != cudaSuccess) st = record_cuda_error(e, "cudaGraphInstantiate (batch)");
    }
    cudaGraphDestroy(g);
    return st;
}

}  // namespace

extern "C" {

azp_batch* azp_batch_create(const azp_batch_config* c, int* status)
{
    auto fail = [&](int st, azp_batch* b) -> azp_batch* {
        if (status) *status = st;
        if (b) {
            b_free(b);
            delete b;
        }
        return nullptr;
    };
    if (!c || c->nsys == 0 || c->nsys > 65535 || !c->N || !c->L || !c->pair_params || !c->r_cut || !c->seeds)
        return fail(AZP_ERR_INVALID, nullptr);
    if (c->precision != AZP_FP64 && c->precision != AZP_FP32) return fail(AZP_ERR_INVALID, nullptr);
    if (c->pair_kind < 0 || c->pair_kind >= AZP_PAIR_NUM_KINDS || !(c->dt > 0.0)) return fail(AZP_ERR_INVALID, nullptr);
    azp_batch* b = new (std::nothrow) azp_batch();
    if (!b) return fail(AZP_ERR_INVALID, nullptr);
    b->S = c->nsys;
    b->precision = c->precision;
    b->kind = c->pair_kind;
    b->dt = c->dt;
    b->kT = c->kT;
    b->gamma = c->gamma;
    b->r_buff = c->r_buff;
    b->noiseless = c->noiseless;
    b->flow = make_flow(c->flow);
    const char* env_tpp = std::getenv("AZP_TPP");
    b->tpp = env_tpp ? std::atoi(env_tpp) : 1;
    if (!(b->tpp == 1 || b->tpp == 2 || b->tpp == 4 || b->tpp == 8 || b->tpp == 16 || b->tpp == 32)) b->tpp = 1;
    const char* env_graph = std::getenv("AZP_GRAPHS");
    b->use_graphs = !(env_graph && env_graph[0] == '0');
    b->n_of.assign(c->N, c->N + c->nsys);
    b->off.assign(c->nsys + 1, 0);
    for (uint32_t r = 0; r < c->nsys; ++r) b->off[r + 1] = b->off[r] + c->N[r];
    b->N = b->off[c->nsys];
    std::vector<SysInfo> info(c->nsys);
    uint32_t cell_off = 0;
    for (uint32_t r = 0; r < c->nsys; ++r) {
        SysInfo& si = info[r];
        azp_box box;
        for (int d = 0; d < 3; ++d) box.L[d] = c->L[3 * r + d];
        const double rc = c->r_cut[r];
        ListCut cut;
        double rmax = 0.0;
        make_list_cuts(&rc, 1, c->r_buff, box, &cut, &rmax);
        for (int d = 0; d < 3; ++d) {
            if (!(box.L[d] > 0.0)) return fail(AZP_ERR_INVALID, b);
            if (box.L[d] < 2.0 * rmax) return fail(AZP_ERR_BOX_TOO_SMALL, b);
            si.L[d] = box.L[d];
            si.Linv[d] = 1.0 / box.L[d];
            si.lo[d] = -0.5 * box.L[d];
            si.hi[d] = 0.5 * box.L[d];
            si.fscale[d] = si.Linv[d] * 4294967296.0;
            si.sfix[d] = (float)(box.L[d] * 2.3283064365386963e-10);
        }
        si.list_lo = cut.lo;
        si.list_hi = cut.hi;
        si.rlistsq = cut.rlistsq;
        const double volume = box.L[0] * box.L[1] * box.L[2];
        const CellGrid g = make_grid(box, rmax);
        b->row_len.push_back(std::min((double)c->N[r], c->N[r] / volume * 4.18879 * rmax * rmax * rmax));
        si.off = b->off[r];
        si.n = c->N[r];
        si.far_cells = 1u;
        for (int d = 0; d < 3; ++d)
            if (g.dim[d] < 2 * g.reach[d] + 3) si.far_cells = 0u;
        si.cell_off = cell_off;
        for (int d = 0; d < 3; ++d) {
            si.dim[d] = g.dim[d];
            si.reach[d] = g.reach[d];
            si.cscale[d] = g.scale[d];
        }
        cell_off += g.ncell;
        si.seed = c->seeds[r];
        const double zero = 0.0;
        int st = AZP_OK;
        double rec[PAIR_TBL];
        st = build_pair_table(c->pair_kind, c->pair_params + (size_t)pair_record_doubles(c->pair_kind) * r, &rc, &zero,
                              c->shift_mode, 1, rec);
        if (st) return fail(st, b);
        for (int k = 0; k < PAIR_TBL; ++k) si.rec[k] = rec[k];
        // the evaluator subtracts the shift itself in the single-system kernel; here fold it
        si.rcutsq = rec[PAIR_REC];
        for (int k = 0; k < PAIR_TBL; ++k) si.recf[k] = (float)rec[k];
        si.rcutf = (float)si.rcutsq;
    }
    b->ncell = cell_off;
    const uint32_t N = b->N;
    int st = AZP_OK;
#define BALLOC(p, n)             \
    do {                         \
        st = balloc(&(p), (n));  \
        if (st) return fail(st, b); \
    } while (0)
    BALLOC(b->info, c->nsys);
    BALLOC(b->sys_off, c->nsys + 1);
    BALLOC(b->pos[0], N);
    BALLOC(b->pos[1], N);
    BALLOC(b->fix[0], N);
    BALLOC(b->fix[1], N);
    BALLOC(b->fix_build, N);
    BALLOC(b->vel, N);
    BALLOC(b->accel, (size_t)3 * N);
    BALLOC(b->image, (size_t)3 * N);
    BALLOC(b->tag, N);
    BALLOC(b->sys, N);
    BALLOC(b->t_pos, N);
    BALLOC(b->t_vel, N);
    BALLOC(b->t_accel, (size_t)3 * N);
    BALLOC(b->t_image, (size_t)3 * N);
    BALLOC(b->t_tag, N);
    BALLOC(b->t_sys, N);
    BALLOC(b->t_cell, N);
    BALLOC(b->o_pos, (size_t)4 * N);
    BALLOC(b->o_vel, (size_t)4 * N);
    BALLOC(b->o_accel, (size_t)3 * N);
    BALLOC(b->o_image, (size_t)3 * N);
    BALLOC(b->cell_of, N);
    BALLOC(b->slot, N);
    BALLOC(b->members, N);
    BALLOC(b->rindex, N);
    BALLOC(b->cell_count, b->ncell);
    BALLOC(b->cell_start, (size_t)b->ncell + 1);
    BALLOC(b->scan_tmp, scan_tmp_words(b->ncell));
    BALLOC(b->counts, N);
    BALLOC(b->nbrs, (size_t)N * b_width(b->max_nn));
    BALLOC(b->flags, 8);
    BALLOC(b->d_ts, 1);
#undef BALLOC
    if (cudaMemcpy(b->info, info.data(), sizeof(SysInfo) * c->nsys, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->sys_off, b->off.data(), sizeof(uint32_t) * (c->nsys + 1), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(b->flags, 0, sizeof(uint32_t) * 8) != cudaSuccess ||
        cudaStreamCreateWithFlags(&b->gstream, cudaStreamNonBlocking) != cudaSuccess)
        return fail(record_cuda_error(cudaGetLastError(), "batch set-up"), b);
    st = b_plan(b);
    if (st) return fail(st, b);
    if (status) *status = AZP_OK;
    return b;
}

void azp_batch_destroy(azp_batch* b)
{
    if (!b) return;
    b_free(b);
    delete b;
}

int azp_batch_set_state(azp_batch* b, const double* pos, const double* vel, const double* accel, const int32_t* image,
                        uint64_t timestep, void* stream)
{
    if (!b || !pos || !vel) return AZP_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    const uint32_t N = b->N;
    std::vector<uint32_t> sys_of(N), tag_of(N);
    for (uint32_t r = 0; r < b->S; ++r)
        for (uint32_t k = 0; k < b->n_of[r]; ++k) {
            sys_of[b->off[r] + k] = r;
            tag_of[b->off[r] + k] = k;
        }
    double *dp, *dv, *da = nullptr;
    int* di = nullptr;
    uint32_t *ds, *dt;
    AZP_CUDA_TRY(cudaMalloc(&dp, sizeof(double) * 4 * N));
    AZP_CUDA_TRY(cudaMalloc(&dv, sizeof(double) * 4 * N));
    AZP_CUDA_TRY(cudaMalloc(&ds, sizeof(uint32_t) * N));
    AZP_CUDA_TRY(cudaMalloc(&dt, sizeof(uint32_t) * N));
    AZP_CUDA_TRY(cudaMemcpyAsync(dp, pos, sizeof(double) * 4 * N, cudaMemcpyHostToDevice, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(dv, vel, sizeof(double) * 4 * N, cudaMemcpyHostToDevice, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(ds, sys_of.data(), sizeof(uint32_t) * N, cudaMemcpyHostToDevice, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(dt, tag_of.data(), sizeof(uint32_t) * N, cudaMemcpyHostToDevice, s));
    if (accel) {
        AZP_CUDA_TRY(cudaMalloc(&da, sizeof(double) * 3 * N));
        AZP_CUDA_TRY(cudaMemcpyAsync(da, accel, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, s));
    }
    if (image) {
        AZP_CUDA_TRY(cudaMalloc(&di, sizeof(int) * 3 * N));
        AZP_CUDA_TRY(cudaMemcpyAsync(di, image, sizeof(int) * 3 * N, cudaMemcpyHostToDevice, s));
    }
    b->cur = 0;
    k_b_load<<<nblk(N), 256, 0, s>>>(dp, dv, da, di, ds, dt, N, b->pos[0], b->vel, b->accel, b->image, b->tag, b->sys,
                                     b->rindex);
    const unsigned long long ts = timestep;
    AZP_CUDA_TRY(cudaMemcpyAsync(b->d_ts, &ts, sizeof(ts), cudaMemcpyHostToDevice, s));
    AZP_CUDA_TRY(cudaMemsetAsync(b->flags, 0, sizeof(uint32_t) * 8, s));
    int st = AZP_OK;
    for (int attempt = 0; attempt < 4; ++attempt) {
        AZP_CUDA_TRY(cudaMemsetAsync(b->flags + 3, 0, sizeof(uint32_t), s));
        st = b_rebuild(b, s, nullptr);
        if (st) break;
        uint32_t need = 0;
        AZP_CUDA_TRY(cudaMemcpyAsync(&need, b->flags + 3, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        AZP_CUDA_TRY(cudaStreamSynchronize(s));
        if (need <= b->max_nn) break;
        cudaFree(b->nbrs);
        b->max_nn = (uint32_t)std::ceil(need * 1.3) + 8;
        st = balloc(&b->nbrs, (size_t)N * b_width(b->max_nn));
        if (st) break;
        b_free_graphs(b);
    }
    AZP_CUDA_TRY(cudaStreamSynchronize(s));
    cudaFree(dp);
    cudaFree(dv);
    cudaFree(ds);
    cudaFree(dt);
    cudaFree(da);
    cudaFree(di);
    b->have_state = (st == AZP_OK);
    return st;
}

int azp_batch_get_state(azp_batch* b, double* pos, double* vel, double* accel, int32_t* image, void* stream)
{
    if (!b || !b->have_state || !pos || !vel || !accel || !image) return AZP_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    const uint32_t N = b->N;
    // packed in buffers that nothing else writes: a call on another stream than the run's
    // may read a state that is changing, but changes none
    k_b_store<<<nblk(N), 256, 0, s>>>(b->pos[b->cur], b->vel, b->accel, b->image, b->tag, b->sys, b->sys_off, N, b->o_pos,
                                      b->o_vel, b->o_accel, b->o_image);
    AZP_CUDA_TRY(cudaMemcpyAsync(pos, b->o_pos, sizeof(double) * 4 * N, cudaMemcpyDeviceToHost, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(vel, b->o_vel, sizeof(double) * 4 * N, cudaMemcpyDeviceToHost, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(accel, b->o_accel, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, s));
    AZP_CUDA_TRY(cudaMemcpyAsync(image, b->o_image, sizeof(int) * 3 * N, cudaMemcpyDeviceToHost, s));
    AZP_CUDA_TRY(cudaStreamSynchronize(s));
    return AZP_OK;
}

int azp_batch_run(azp_batch* b, uint64_t steps, void* stream)
{
    if (!b || !b->have_state) return AZP_ERR_INVALID;
    b->launches = 0;
    if (steps == 0) return AZP_OK;
    cudaStream_t s = as_stream(stream);
    const uint32_t N = b->N;
    const double half = 0.5 * b->r_buff;
    k_b_step1<<<nblk(N), 256, 0, s>>>(b->pos[b->cur], b->fix[b->cur], b->fix_build, b->vel, b->accel, b->image, b->sys,
                                      b->info, N, b->dt, (float)(half * half * (1.0 - 1e-5)), b->flags);
    AZP_CHECK_LAUNCH("k_b_step1");
    b->launches += 1;
    uint64_t mid = steps - 1;
    int st = AZP_OK;
    if (b->use_graphs && mid >= 2) {
        for (int p = 0; p < 2; ++p)
            if (!b->gexec[p]) {
                st = b_build_graph(b, p, &b->gexec[p]);
                if (st) return st;
            }
        while (mid >= 2) {
            AZP_CUDA_TRY(cudaGraphLaunch(b->gexec[b->cur], s));
            b->launches += 3;
            mid -= 2;
        }
    }
    while (mid > 0) {
        st = b_rebuild(b, s, b->flags);
        if (st) return st;
        st = b_step(b, 1, s, 0, 0);
        if (st) return st;
        b->cur ^= 1;
        --mid;
    }
    st = b_rebuild(b, s, b->flags);
    if (st) return st;
    return b_step(b, 0, s, 0, 0);
}

int azp_batch_error(azp_batch* b, uint32_t* err_word, uint32_t* n_builds, void* stream)
{
    if (!b || !err_word) return AZP_ERR_INVALID;
    cudaStream_t s = as_stream(stream);
    uint32_t f[8];
    AZP_CUDA_TRY(cudaMemcpyAsync(f, b->flags, sizeof(f), cudaMemcpyDeviceToHost, s));
    AZP_CUDA_TRY(cudaStreamSynchronize(s));
    uint32_t e = f[1];
    if (f[3] > b->max_nn) e |= AZP_EBIT_NLIST_OVERFLOW;
    *err_word = e;
    if (n_builds) *n_builds = f[2];
    return AZP_OK;
}

int azp_batch_set_block(azp_batch* b, int block)
{
    if (!b || !(block == 64 || block == 128 || block == 256 || block == 512)) return AZP_ERR_INVALID;
    if (b->block != block) b_free_graphs(b);
    b->block = block;
    return AZP_OK;
}

int azp_batch_set_tpp(azp_batch* b, int tpp)
{
    if (!b || !(tpp == 1 || tpp == 2 || tpp == 4 || tpp == 8 || tpp == 16 || tpp == 32)) return AZP_ERR_INVALID;
    if (b->tpp != tpp && b->precision == AZP_FP64) b_free_graphs(b);  // (the FP32 step does not change)
    b->tpp = tpp;
    return AZP_OK;
}

uint64_t azp_batch_last_launches(const azp_batch* b) { return b ? b->launches : 0; }

}  // extern "C"
