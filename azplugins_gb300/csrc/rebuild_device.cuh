// rebuild_device.cuh -- the list rebuild of the resident engine inside one cooperative
// launch (the persistent run, engine_kernels.cuh): the phases of engine.cu's rebuild
// kernels as grid-stride loops with grid barriers between them.
#pragma once

#include "engine.cuh"
#include "nlist_device.cuh"

namespace azp
{
// The re-sort of the particles' arrays: temps[s] <- arrays[members[s]], then back.
struct PermArgs {
    const uint32_t* members;
    double4_32a *pos, *t_pos;   // pos NULL in FP32-force mode (the fixed words move instead)
    uint4 *fix, *t_fix;         // FP32-force mode: high and low fixed words, masses
    uint4 *lo, *t_lo;
    double *mass, *t_mass;
    uint4* fix_build;           // FP32-force mode: receives the new high words too
    double4_32a *vel, *t_vel;
    double *accel, *t_accel;
    int *image, *t_image;
    uint32_t *tag, *t_tag, *rtag;
    double *diam, *t_diam;
    uint32_t *cell_of, *t_cell;
    uint32_t N;
};

// One particle's records. All of them are loaded before any is stored: the arrays may
// alias as far as the compiler knows, and a load behind each store's operand would
// make the copy a chain of a dozen memory latencies.
struct PermRow {
    double4_32a pos, vel;
    uint4 fix, lo;
    double mass, diam, a0, a1, a2;
    int g0, g1, g2;
    uint32_t tag, cell;
};
// from the arrays (temps false) or the temporaries (temps true), particle o
template<bool TEMPS> AZP_D PermRow perm_load(const PermArgs& a, uint32_t o)
{
    PermRow r;
    if (a.pos) r.pos = (TEMPS ? a.t_pos : a.pos)[o];
    if (a.fix) {
        r.fix = (TEMPS ? a.t_fix : a.fix)[o];
        r.lo = (TEMPS ? a.t_lo : a.lo)[o];
        r.mass = (TEMPS ? a.t_mass : a.mass)[o];
    }
    r.vel = (TEMPS ? a.t_vel : a.vel)[o];
    const double* acc = (TEMPS ? a.t_accel : a.accel) + 3 * (size_t)o;
    const int* img = (TEMPS ? a.t_image : a.image) + 3 * (size_t)o;
    r.a0 = acc[0];
    r.a1 = acc[1];
    r.a2 = acc[2];
    r.g0 = img[0];
    r.g1 = img[1];
    r.g2 = img[2];
    r.tag = (TEMPS ? a.t_tag : a.tag)[o];
    if (a.diam) r.diam = (TEMPS ? a.t_diam : a.diam)[o];
    r.cell = (TEMPS ? a.t_cell : a.cell_of)[o];
    return r;
}
template<bool TEMPS> AZP_D void perm_store(const PermArgs& a, uint32_t s, const PermRow& r)
{
    if (a.pos) (TEMPS ? a.t_pos : a.pos)[s] = r.pos;
    if (a.fix) {
        (TEMPS ? a.t_fix : a.fix)[s] = r.fix;
        if (!TEMPS) a.fix_build[s] = r.fix;
        (TEMPS ? a.t_lo : a.lo)[s] = r.lo;
        (TEMPS ? a.t_mass : a.mass)[s] = r.mass;
    }
    (TEMPS ? a.t_vel : a.vel)[s] = r.vel;
    double* acc = (TEMPS ? a.t_accel : a.accel) + 3 * (size_t)s;
    int* img = (TEMPS ? a.t_image : a.image) + 3 * (size_t)s;
    acc[0] = r.a0;
    acc[1] = r.a1;
    acc[2] = r.a2;
    img[0] = r.g0;
    img[1] = r.g1;
    img[2] = r.g2;
    (TEMPS ? a.t_tag : a.tag)[s] = r.tag;
    if (a.diam) (TEMPS ? a.t_diam : a.diam)[s] = r.diam;
    (TEMPS ? a.t_cell : a.cell_of)[s] = r.cell;
}

// temps[s] <- arrays[members[s]]; the particle's tag
AZP_D uint32_t perm_gather(const PermArgs& a, uint32_t s)
{
    const PermRow r = perm_load<false>(a, a.members[s]);
    perm_store<true>(a, s, r);
    return r.tag;
}

// arrays[s] <- temps[s]; the tag of s
AZP_D uint32_t perm_back(const PermArgs& a, uint32_t s)
{
    const PermRow r = perm_load<true>(a, s);
    perm_store<false>(a, s, r);
    return r.tag;
}

struct BondTableArgs {
    const uint32_t *n_tag, *partner_tag, *type_tag;  // tag order [k * N + tag]; n_tag NULL: no bonds
    uint32_t* bt_n;
    uint2* bt;
    uint32_t *ex_n, *ex_idx;
    int exclude;
};

// per-particle bonds and exclusions of particle i (tag t) in index order
AZP_D void bond_row(const BondTableArgs& b, const uint32_t* rtag, uint32_t i, uint32_t t, uint32_t N)
{
    const uint32_t n = b.n_tag[t];
    for (uint32_t k = 0; k < n; ++k) {
        const uint32_t p = rtag[b.partner_tag[(size_t)k * N + t]];
        b.bt[(size_t)k * N + i] = make_uint2(p, b.type_tag[(size_t)k * N + t]);
        if (b.exclude) b.ex_idx[(size_t)k * N + i] = p;
    }
    b.bt_n[i] = n;
    if (b.ex_n) b.ex_n[i] = b.exclude ? n : 0u;
}

// ---------------------------------------------------------------- persistent run
struct RebuildArgs {
    PermArgs perm;
    BondTableArgs bonds;
    ListArgs list;              // members set (the cell member table)
    double Linv[3];
    uint32_t *slot, *cell_count, *scan_tmp, *cell_of, *members, *cell_start;
    uint32_t* sort_gate;        // [4]: order-keeping builds since the last re-sort
    uint32_t sort_every;
    uint4* words;               // fixed-point words in cell order (order-keeping builds): the next step's buffer
    int force_sort, crowded, by_reference, has_list;
};

constexpr uint32_t RUN_BLOCK = 256;
constexpr uint32_t RUN_TILE = 4 * RUN_BLOCK;          // cells a block scans at a time
constexpr uint32_t RUN_MAX_TILES = 2 * RUN_BLOCK;
constexpr uint32_t RUN_MAX_CELLS = RUN_TILE * RUN_MAX_TILES;

struct RunArgs {
    MDArgs step[2];             // by buffer parity
    RebuildArgs rebuild[2];
    uint32_t steps, blocks;     // timesteps, and thread blocks one step takes
    int cur;                    // parity of the first step
    uint32_t max_polls;         // of one wait at a barrier
    uint32_t* sync;             // grid barrier: arrivals, generation
    uint32_t* request;          // three rotating words: 1 a particle asked for a rebuild, 2 an error is set;
                                // then three rotating counters of the blocks taken beyond the launch's own
};

// All blocks of the (cooperative) launch. Thread 0 releases the block's writes with its
// arrival (an acquire-release add, which with the block barrier before it covers the
// whole block) and polls the generation with relaxed loads until the last arrival has
// raised it, then acquires. The wait is bounded: r.max_polls polls, after which the
// launch's error word gets AZP_EBIT_TIMEOUT and the block leaves. It has arrived, so the
// others pass this barrier at most, with all of the phase before it done, and give up at
// the next. AZP_RUN_POLLS sets another limit than about ten seconds.
// gen: the generation before the launch's first barrier, counted on by every thread.
constexpr uint32_t RUN_MAX_POLLS = 1u << 24;
AZP_D uint32_t load_relaxed(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
AZP_D bool grid_barrier(const RunArgs& r, uint32_t& gen, uint32_t* s_word)
{
    __syncthreads();
    if (gridDim.x == 1u) return true;
    if (threadIdx.x == 0u) {
        uint32_t ok = 1u, arrived;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(r.sync) : "memory");
        if (arrived == gridDim.x - 1u) {
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(r.sync), "r"(0u) : "memory");
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(r.sync + 1), "r"(gen + 1u) : "memory");
        } else {
            uint32_t polls = 0;
            while (load_relaxed(r.sync + 1) == gen)
                if (++polls >= r.max_polls) {
                    atomicOr(r.step[0].flags + 1, AZP_EBIT_TIMEOUT);
                    ok = 0u;
                    break;
                }
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
        }
        *s_word = ok;
    }
    ++gen;
    __syncthreads();
    return *s_word != 0u;
}

// inclusive sum over the block (RUN_BLOCK threads); s: RUN_BLOCK / 32 words
AZP_D uint32_t block_sum_scan(uint32_t v, uint32_t* s)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)lane >= o) v += t;
    }
    if (lane == 31u) s[warp] = v;
    __syncthreads();
    uint32_t before = 0u;
    for (uint32_t w = 0; w < warp; ++w) before += s[w];
    __syncthreads();
    return v + before;
}

// shared memory of the rebuild's phases
inline size_t rebuild_smem(uint32_t ntypes)
{
    const size_t sort = (size_t)(RUN_BLOCK / 32) * kMaxSortedCell * sizeof(uint32_t);
    const size_t scan = (RUN_BLOCK / 32 + RUN_MAX_TILES) * sizeof(uint32_t);
    const size_t list = nlw_shared_bytes<4>(ntypes, RUN_BLOCK / 32);
    size_t m = sort;
    if (scan > m) m = scan;
    if (list > m) m = list;
    return m;
}

// The rebuild at buffer parity par, by all blocks; six grid barriers. FX: FP32-force
// state. cell_count is zero on entry and on return. Returns false after a timed-out
// barrier.
template<bool FX>
static __device__ __noinline__ bool rebuild_cooperative(const RunArgs& r, int par, uint32_t& gen, unsigned char* pool,
                                                        uint32_t* s_word)
{
    const RebuildArgs& b = r.rebuild[par];
    const ListArgs& L = b.list;
    const CellGrid& g = L.g;
    // work in units of a warp goes round the blocks, so that a phase with fewer units than
    // warps keeps all SMs at it
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t gwarp = warp * gridDim.x + blockIdx.x, nwarps = gridDim.x * (RUN_BLOCK / 32u);
    const uint32_t N = L.N, tid = 32u * gwarp + lane, nth = 32u * nwarps;
    const uint32_t since = b.sort_gate[4];
    const bool sort = b.force_sort || since + 1u >= b.sort_every;
    // cells
    for (uint32_t i = tid; i < N; i += nth) {
        uint32_t c;
        if constexpr (FX) {
            c = cell_of_fixed(L.fixed[i], g);
        } else {
            c = cell_of_position(L.pos[i], g);
        }
        b.cell_of[i] = c;
        b.slot[i] = atomicAdd(&b.cell_count[c], 1u);
    }
    if (!grid_barrier(r, gen, s_word)) return false;
    // counts -> sums inside tiles (in place), tile totals
    uint32_t* s_scan = reinterpret_cast<uint32_t*>(pool);
    const uint32_t tiles = (g.ncell + RUN_TILE - 1u) / RUN_TILE;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t c0 = t * RUN_TILE + 4u * threadIdx.x;
        uint32_t v[4], sum = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = c0 + k < g.ncell ? b.cell_count[c0 + k] : 0u;
            sum += v[k];
        }
        const uint32_t inc = block_sum_scan(sum, s_scan);
        uint32_t e = inc - sum;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (c0 + k < g.ncell) b.cell_count[c0 + k] = e;
            e += v[k];
        }
        if (threadIdx.x == RUN_BLOCK - 1u) b.scan_tmp[t] = inc;
    }
    if (!grid_barrier(r, gen, s_word)) return false;
    // tile offsets, the members of each cell, the cell starts
    uint32_t* s_off = s_scan + RUN_BLOCK / 32;
    {
        const uint32_t t0 = 2u * threadIdx.x;
        const uint32_t a0 = t0 < tiles ? b.scan_tmp[t0] : 0u, a1 = t0 + 1u < tiles ? b.scan_tmp[t0 + 1u] : 0u;
        const uint32_t inc = block_sum_scan(a0 + a1, s_scan);
        s_off[t0] = inc - a0 - a1;
        s_off[t0 + 1u] = inc - a1;
        __syncthreads();
    }
    for (uint32_t i = tid; i < N; i += nth) {
        const uint32_t c = b.cell_of[i];
        b.members[b.cell_count[c] + s_off[c / RUN_TILE] + b.slot[i]] = i;
    }
    for (uint32_t c = tid; c <= g.ncell; c += nth)
        b.cell_start[c] = c < g.ncell ? b.cell_count[c] + s_off[c / RUN_TILE] : N;
    if (!grid_barrier(r, gen, s_word)) return false;
    // each cell's members in index order; a re-sort gathers them at once
    {
        uint32_t* s_row = reinterpret_cast<uint32_t*>(pool) + warp * kMaxSortedCell;
        const uint32_t per = b.crowded ? 1u : 32u;
        const uint32_t units = (g.ncell + per - 1u) / per;
        for (uint32_t u = gwarp; u < units; u += nwarps) {
            if (b.crowded) sort_cell_per_warp(b.cell_start, b.members, g.ncell, s_row, u);
            else sort_cells_warp(b.cell_start, b.members, g.ncell, s_row, u);
            __syncwarp();
            const uint32_t e = b.cell_start[min(u * per + per, g.ncell)];
            for (uint32_t s = b.cell_start[u * per] + lane; s < e; s += 32u) {
                if (sort) {
                    const uint32_t tag = perm_gather(b.perm, s);
                    b.perm.rtag[tag] = s;
                } else {
                    // (FP64: the shadow of the step that ended at these positions)
                    b.words[s] = L.fixed[b.members[s]];
                }
            }
            __syncwarp();
        }
    }
    if (!grid_barrier(r, gen, s_word)) return false;
    // back into place, with the bonds of the new order; the shadows of this build
    for (uint32_t i = tid; i < N; i += nth) {
        if (sort) {
            const uint32_t t = perm_back(b.perm, i);
            if (b.bonds.n_tag) bond_row(b.bonds, b.perm.rtag, i, t, N);
        }
        if constexpr (FX) {
            if (!sort) b.perm.fix_build[i] = b.perm.fix[i];
        } else {
            const double4_32a p = b.perm.pos[i];
            uint4 f;
            f.x = to_fixed(p.x, b.Linv[0]);
            f.y = to_fixed(p.y, b.Linv[1]);
            f.z = to_fixed(p.z, b.Linv[2]);
            f.w = type_of(p.w);
            const_cast<uint4*>(L.fixed)[i] = f;
            b.perm.fix_build[i] = f;
        }
    }
    for (uint32_t c = tid; c < g.ncell; c += nth) b.cell_count[c] = 0u;
    if (!grid_barrier(r, gen, s_word)) return false;
    if (b.has_list) {
        // a warp per chunk whatever the row: a launch of this size has warps to spare, and
        // a thread per particle would walk its stencil as a chain of memory latencies
        const NlwShared sh = nlw_shared<4>(pool, L.ntypes, RUN_BLOCK / 32);
        nlw_tables(sh, L.cuts, L.ntypes, g);
        __syncthreads();
        for (uint32_t c = gwarp; c * 4u < N; c += nwarps) {
            const auto chunk = [&](auto one, auto ref) {
                if (sort) nlist_chunk<false, one.value, true, ref.value, 4>(L, L.fixed, c, warp, sh);
                else nlist_chunk<false, one.value, false, ref.value, 4>(L, b.words, c, warp, sh);
            };
            if (L.ntypes == 1u) {
                if (b.by_reference) chunk(std::true_type{}, std::true_type{});
                else chunk(std::true_type{}, std::false_type{});
            } else {
                if (b.by_reference) chunk(std::false_type{}, std::true_type{});
                else chunk(std::false_type{}, std::false_type{});
            }
        }
    }
    if (tid == 0u) {
        r.step[0].flags[0] = 0u;
        r.step[0].flags[2] += 1u;
        b.sort_gate[4] = sort ? 0u : since + 1u;
    }
    return grid_barrier(r, gen, s_word);
}

}  // namespace azp
