// nlist_device.cuh -- the neighbour-list scans as device functions: a thread per
// particle and a warp per chunk of cell-ordered particles (nlist.cu launches them; the
// engine's persistent run calls them between its steps).
#pragma once

#include "celllist.cuh"
#include "fixed64.cuh"

#include <type_traits>

namespace azp
{
struct BoxArgs {
    double L[3], Linv[3];
    double l64[3];  // L * 2^-64 (64-bit fixed-point unit)
    float sfix[3];  // L * 2^-32 (fixed-point unit)
};

inline BoxArgs box_args(const azp_box& b)
{
    BoxArgs a;
    for (int d = 0; d < 3; ++d) {
        a.L[d] = b.L[d];
        a.Linv[d] = 1.0 / b.L[d];
        a.l64[d] = b.L[d] * 5.421010862427522e-20;
        a.sfix[d] = (float)(b.L[d] * 2.3283064365386963e-10);
    }
    return a;
}

// FP64 position of particle i from its 64-bit fixed-point words (fixed64.cuh)
__device__ __forceinline__ double4_32a fx_position(const uint4* hi, const uint4* lo, uint32_t i, const BoxArgs& bx)
{
    const uint4 h = hi[i], l = lo[i];
    return make_double4_32a(fx_to_double(fx_join(h.x, l.x), bx.l64[0]), fx_to_double(fx_join(h.y, l.y), bx.l64[1]),
                            fx_to_double(fx_join(h.z, l.z), bx.l64[2]), 0.0);
}

constexpr uint32_t MAX_LIST_TYPES = 16;  // ntypes^2 <= 256 thresholds in shared memory
constexpr int NLIST_BLOCK = 128;
static_assert(TILE_P % NLIST_BLOCK == 0, "a list-build block lies inside one tile block");
constexpr uint32_t NL_EX_REG = 4;  // exclusion keys of a particle held in registers
// Candidates in the FP32 band around r_list are appended with this mark and
// decided exactly in the compaction pass: the scan loop then holds no call and
// no FP64 state (measured at N = 1M: 40 registers instead of 64, the build 20 %
// faster, the same sets).
constexpr uint32_t NL_BAND = 0x80000000u;
constexpr uint32_t NL_MAX_N = NL_BAND - 1;  // particle indices stay below the mark

// The oracle's exact FP64 decision for a candidate inside the ambiguous band
// of the FP32 prefilter. Out of line: a candidate lands in the band about once
// per million.
static __device__ __noinline__ bool nl_exact_within(uint32_t i, uint32_t j, double rlistsq, const BoxArgs& bx,
                                                    const double4_32a* pos, const uint4* fixed, const uint4* lo)
{
    const double4_32a a = lo ? fx_position(fixed, lo, i, bx) : pos[i];
    const double4_32a b = lo ? fx_position(fixed, lo, j, bx) : pos[j];
    const double vx = min_image1(a.x - b.x, bx.L[0], bx.Linv[0]);
    const double vy = min_image1(a.y - b.y, bx.L[1], bx.Linv[1]);
    const double vz = min_image1(a.z - b.z, bx.L[2], bx.Linv[2]);
    return rsq_exact(vx, vy, vz) < rlistsq;
}

// exclusion keys of a particle beyond the NL_EX_REG held in registers
static __device__ __noinline__ bool nl_excluded_tail(uint32_t i, uint32_t kj, uint32_t nex, uint32_t N,
                                                     const uint32_t* ex_keys)
{
    for (uint32_t e = NL_EX_REG; e < nex; ++e)
        if (ex_keys[(size_t)e * N + i] == kj) return true;
    return false;
}

// What a list build reads and writes.
struct ListArgs {
    const double4_32a* pos;      // FP64 positions (null with lo)
    const uint4 *fixed, *lo;     // fixed-point words; lo: low words of 64-bit positions, or null
    uint32_t N, ntypes;
    BoxArgs bx;
    CellGrid g;
    const uint32_t *cell_start, *members, *cell_of;
    const ListCut* cuts;
    const uint32_t *ex_n, *ex_keys, *keys;
    uint32_t *counts, *nbrs;
    uint32_t max_nn;
    uint32_t* flags;             // [0]: largest count above max_nn
};

// a load through the read-only path (NC: what no thread of the launch writes), or a
// plain one (launches that rebuild and step in turn)
template<bool NC, class T> AZP_D T ld_ro(const T* p)
{
    if constexpr (NC) return __ldg(p);
    else return *p;
}

// Full list, one thread per particle. For every (y, z) offset row of the 3x3x3
// cell stencil, the x-neighbour cells cx-1, cx, cx+1 are consecutive cell
// indices, so their particles are one contiguous slot range (members[s], or s
// itself when the particles are stored in cell order); at the x faces the
// wrapped cell is a second range. The scan per candidate is one 16-byte gather,
// the integer minimum image and the FP32 prefilter; ONE_TYPE keeps the
// thresholds of a single-type system in registers.
// s_cut: the thresholds in shared memory; s_trec: the tile record of the block, or null
template<bool NC, bool ONE_TYPE, bool SORTED>
AZP_D void nlist_thread(const ListArgs& L, uint32_t i, const ListCut* s_cut, const uint32_t* s_trec)
{
    const double4_32a* pos = L.pos;
    const uint4 *fixed = L.fixed, *lo = L.lo;
    const uint32_t *cell_start = L.cell_start, *members = L.members, *cell_of = L.cell_of, *ex_n = L.ex_n,
                   *ex_keys = L.ex_keys, *keys = L.keys;
    uint32_t *counts = L.counts, *nbrs = L.nbrs, *flags = L.flags;
    const BoxArgs& bx = L.bx;
    const CellGrid& g = L.g;
    const uint32_t N = L.N, ntypes = L.ntypes, max_nn = L.max_nn;
    const bool tile = s_trec != nullptr;
    if (i >= N) return;
    const uint4 fi = ld_ro<NC>(fixed + i);
    const uint32_t row = fi.w * ntypes;
    const ListCut cut0 = s_cut[0];
    const uint32_t nex = ex_n ? ld_ro<NC>(ex_n + i) : 0u;
    const uint32_t cc = ld_ro<NC>(cell_of + i);
    const int dx = g.dim[0], dy = g.dim[1], dz = g.dim[2];
    const int cx = (int)(cc % (uint32_t)dx);
    const int cy = (int)((cc / (uint32_t)dx) % (uint32_t)dy);
    const int cz = (int)(cc / ((uint32_t)dx * (uint32_t)dy));
    // the x-cells cx - reach .. cx + reach: one contiguous range inside the row,
    // and the wrapped part at an x face, contiguous too ([wb, we]; empty: wb > we)
    int x0 = cx - g.reach[0], x1 = cx + g.reach[0], wb = 1, we = 0;
    if (x0 < 0) {
        wb = dx + x0;
        we = dx - 1;
        x0 = 0;
    }
    if (x1 >= dx) {
        wb = 0;
        we = x1 - dx;
        x1 = dx - 1;
    }
    uint32_t ex[NL_EX_REG];
#pragma unroll
    for (uint32_t e = 0; e < NL_EX_REG; ++e) ex[e] = e < nex ? ld_ro<NC>(ex_keys + (size_t)e * N + i) : 0xffffffffu;
    uint32_t n = 0;
    // one candidate: the integer minimum image, the FP32 prefilter, the append
    const auto test = [&](uint32_t j, const uint4& fj) {
        const float ddx = (float)(int32_t)(fi.x - fj.x) * bx.sfix[0];
        const float ddy = (float)(int32_t)(fi.y - fj.y) * bx.sfix[1];
        const float ddz = (float)(int32_t)(fi.z - fj.z) * bx.sfix[2];
        const float rs = ddx * ddx + ddy * ddy + ddz * ddz;
        const ListCut cut = ONE_TYPE ? cut0 : s_cut[row + fj.w];
        // within r_list or in the band around it: appended (i itself, its
        // excluded partners and the band candidates, marked, too; the pass
        // below takes out what does not belong)
        if (rs < cut.hi) {
            if (n < max_nn) nbrs[(size_t)n * N + i] = rs < cut.lo ? j : (j | NL_BAND);
            ++n;
        }
    };
    for (int oz = -g.reach[2]; oz <= g.reach[2]; ++oz) {
        int nz = cz + oz;
        nz += (nz < 0) ? dz : 0;
        nz -= (nz >= dz) ? dz : 0;
        for (int oy = -g.reach[1]; oy <= g.reach[1]; ++oy) {
            int ny = cy + oy;
            ny += (ny < 0) ? dy : 0;
            ny -= (ny >= dy) ? dy : 0;
            const uint32_t rb = ((uint32_t)nz * dy + ny) * dx;
            for (int part = 0; part < 2; ++part) {
                uint32_t sb, se;
                if (part == 0) {
                    sb = ld_ro<NC>(cell_start + rb + x0);
                    se = ld_ro<NC>(cell_start + rb + x1 + 1);
                } else {
                    if (wb > we) break;
                    sb = ld_ro<NC>(cell_start + rb + wb);
                    se = ld_ro<NC>(cell_start + rb + we + 1);
                }
#pragma unroll 4
                for (uint32_t sl = sb; sl < se; ++sl) {
                    const uint32_t j = SORTED ? sl : ld_ro<NC>(members + sl);
                    test(j, ld_ro<NC>(fixed + j));
                }
            }
        }
    }
    // Compact the row in place: drop i itself and the excluded partners, keeping
    // the order. The warp-wide scan above stays a load, a test and an append; the
    // exclusion compares run once per listed entry here instead of on every
    // candidate iteration. Overflow is judged on the raw count, which bounds the
    // true one, so a row that lost entries to the capacity is always reported.
    const uint32_t stored = min(n, max_nn);
    uint32_t m = 0;
    for (uint32_t k = 0; k < stored; ++k) {
        uint32_t j = nbrs[(size_t)k * N + i];
        const bool marked = (j & NL_BAND) != 0u;
        bool drop = false;
        if (marked) {
            // a candidate in the band around r_list: the oracle's exact FP64 decision
            j &= ~NL_BAND;
            const ListCut cut = ONE_TYPE ? cut0 : s_cut[row + ld_ro<NC>(fixed + j).w];
            drop = !nl_exact_within(i, j, cut.rlistsq, bx, pos, fixed, lo);
        }
        drop |= j == i;
        if (nex && !drop) {
            const uint32_t kj = keys ? ld_ro<NC>(keys + j) : j;
#pragma unroll
            for (uint32_t e = 0; e < NL_EX_REG; ++e) drop |= ex[e] == kj;
            if (nex > NL_EX_REG) drop |= nl_excluded_tail(i, kj, nex, N, ex_keys);
        }
        if (!drop) {
            if (tile) nbrs[(size_t)m * N + i] = tile_encode(s_trec, j);
            else if (m != k || marked) nbrs[(size_t)m * N + i] = j;  // a kept band entry loses its mark
            ++m;
        }
    }
    counts[i] = m;  // what is written, also past the capacity
    if (n > max_nn) atomicMax(&flags[0], n);
}

// The list with a warp per chunk of cell-ordered particles. A warp takes CH consecutive
// slots of the cell order, the particles of one cell at a time. The slot ranges of their
// stencil rows are laid end to end (bounds read and summed by the lanes together) and
// walked 32 candidates a step, each loaded once, a step ahead, and tested against every
// particle of the chunk: a ballot ranks the hits, which are appended to the particles' rows
// in shared memory. Rows with excluded partners or candidates of the band are then compacted
// there, and the rows written out with the chunk's particles side by side. Order and
// contents are those of k_nlist_build_threads.
// words: the candidates' fixed-point words in cell order (fixed itself when SORTED).
// Particles whose types have smaller list radii than the grid's walk fewer cells.
// REF: coordinates as floats relative to the chunk's first particle, so that a test
// costs no integer conversion (16 a clock and SM); grids with at least 2 reach + 3 cells on
// every axis, where the minimum image relative to that particle is the pair's for all
// pairs in range. A position far outside the box or not finite is clamped into some cell:
// the particles that share a chunk with it are tested pair by pair (word_in_cell); as a
// candidate it needs nothing, for a word outside the stencil is out of range either way.
constexpr int NLW_WARPS = 4;
constexpr uint32_t NLW_ROW = 192;   // entries of a row held in shared memory; the rest go to the list at once
constexpr uint32_t NLW_RANGES = 2 * 9 * 9;  // stencil rows (reach <= 4) and their wrapped parts
// whether every axis has the cells REF asks for
inline bool list_by_reference(const CellGrid& g)
{
    for (int d = 0; d < 3; ++d)
        if (g.dim[d] < 2 * g.reach[d] + 3) return false;
    return true;
}

// Shared memory of one block of the warp build: thresholds, reaches, and per warp the
// rows and the ranges.
struct NlwShared {
    ListCut* cut;
    float *hi, *lo;
    int* reach;       // [ntypes][3]
    uint32_t* rows;   // [warps][CH][NLW_ROW]
    uint2* range;     // [warps][NLW_RANGES + 1]: (first candidate, first slot) of each range
};
template<int CH> AZP_HD size_t nlw_shared_bytes(uint32_t ntypes, uint32_t warps)
{
    return (size_t)ntypes * ntypes * (sizeof(ListCut) + 8) + (size_t)ntypes * 12 + 8 +
           (size_t)warps * (CH * NLW_ROW * 4 + (NLW_RANGES + 1) * sizeof(uint2));
}
template<int CH> AZP_D NlwShared nlw_shared(unsigned char* p, uint32_t ntypes, uint32_t warps)
{
    NlwShared s;
    const uint32_t nt2 = ntypes * ntypes;
    s.cut = reinterpret_cast<ListCut*>(p);
    s.range = reinterpret_cast<uint2*>(s.cut + nt2);
    s.rows = reinterpret_cast<uint32_t*>(s.range + warps * (NLW_RANGES + 1u));
    s.hi = reinterpret_cast<float*>(s.rows + warps * CH * NLW_ROW);
    s.lo = s.hi + nt2;
    s.reach = reinterpret_cast<int*>(s.lo + nt2);
    return s;
}
// fills the tables (the caller synchronises)
AZP_D void nlw_tables(const NlwShared& s, const ListCut* cuts, uint32_t ntypes, const CellGrid& g)
{
    for (uint32_t t = threadIdx.x; t < ntypes * ntypes; t += blockDim.x) {
        s.cut[t] = cuts[t];
        s.hi[t] = cuts[t].hi;
        s.lo[t] = cuts[t].lo;
    }
    for (uint32_t t = threadIdx.x; t < ntypes; t += blockDim.x) {
        // cells beyond ceil(r / width) lie further than the type's largest list radius
        double r2 = 0.0;
        for (uint32_t u = 0; u < ntypes; ++u) r2 = fmax(r2, cuts[t * ntypes + u].rlistsq);
        const double r = sqrt(r2) * (1.0 + 1e-5);
        for (int d = 0; d < 3; ++d) s.reach[3 * t + d] = min(g.reach[d], (int)ceil(r * g.scale[d]));
    }
}

// chunk `chunk` (CH slots) by the calling warp, the warp-th of its block
template<bool NC, bool ONE_TYPE, bool SORTED, bool REF, int CH>
AZP_D void nlist_chunk(const ListArgs& L, const uint4* words, uint32_t chunk, uint32_t warp, const NlwShared& sh)
{
    const double4_32a* pos = L.pos;
    const uint4 *fixed = L.fixed, *lo = L.lo;
    const uint32_t *cell_start = L.cell_start, *members = L.members, *cell_of = L.cell_of, *ex_n = L.ex_n,
                   *ex_keys = L.ex_keys;
    uint32_t *counts = L.counts, *nbrs = L.nbrs, *flags = L.flags;
    const BoxArgs& bx = L.bx;
    const CellGrid& g = L.g;
    const uint32_t N = L.N, ntypes = L.ntypes, max_nn = L.max_nn;
    const ListCut* s_cut = sh.cut;
    const float *s_hi = sh.hi, *s_lo = sh.lo;
    const int* s_reach = sh.reach;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t(*rows)[NLW_ROW] = reinterpret_cast<uint32_t(*)[NLW_ROW]>(sh.rows + warp * CH * NLW_ROW);
    uint2* range = sh.range + warp * (NLW_RANGES + 1u);
    const ListCut cut0 = s_cut[0];
    const int dx = g.dim[0], dy = g.dim[1], dz = g.dim[2];
    const uint32_t s_begin = chunk * CH;
    const uint32_t s_end = min(s_begin + CH, N);
    for (uint32_t sa = s_begin; sa < s_end;) {
        // the slots from sa on that share its cell
        const uint32_t my_slot = min(sa + lane, s_end - 1u);
        const uint32_t my_i = SORTED ? my_slot : ld_ro<NC>(members + my_slot);
        const uint32_t my_cell = ld_ro<NC>(cell_of + my_i);
        const uint4 my_word = ld_ro<NC>(words + my_slot);
        const uint32_t cc = __shfl_sync(0xffffffffu, my_cell, 0);
        const uint32_t same = __ballot_sync(0xffffffffu, my_cell == cc && sa + lane < s_end);
        const uint32_t cnt = (uint32_t)__ffs(~same) - 1u;  // CH < 32: some lane is off
        uint32_t pi[CH], n[CH];
        uint4 pw[CH];
        float px[CH], py[CH], pz[CH];
        const uint4 ref = make_uint4(__shfl_sync(0xffffffffu, my_word.x, 0), __shfl_sync(0xffffffffu, my_word.y, 0),
                                     __shfl_sync(0xffffffffu, my_word.z, 0), 0u);
        int r0 = 0, r1 = 0, r2 = 0;
#pragma unroll
        for (int p = 0; p < CH; ++p) {
            pi[p] = __shfl_sync(0xffffffffu, my_i, p);
            pw[p].x = __shfl_sync(0xffffffffu, my_word.x, p);
            pw[p].y = __shfl_sync(0xffffffffu, my_word.y, p);
            pw[p].z = __shfl_sync(0xffffffffu, my_word.z, p);
            pw[p].w = ONE_TYPE ? 0u : __shfl_sync(0xffffffffu, my_word.w, p);
            n[p] = 0u;
            px[p] = (float)(int32_t)(pw[p].x - ref.x) * bx.sfix[0];
            py[p] = (float)(int32_t)(pw[p].y - ref.y) * bx.sfix[1];
            pz[p] = (float)(int32_t)(pw[p].z - ref.z) * bx.sfix[2];
            if (p < (int)cnt) {
                const int* r = s_reach + 3 * pw[p].w;
                r0 = max(r0, r[0]);
                r1 = max(r1, r[1]);
                r2 = max(r2, r[2]);
            }
            pw[p].w *= ntypes;
        }
        const int cx = (int)(cc % (uint32_t)dx);
        const int cy = (int)((cc / (uint32_t)dx) % (uint32_t)dy);
        const int cz = (int)(cc / ((uint32_t)dx * (uint32_t)dy));
        // the x-cells as in k_nlist_build_threads: one range, and the wrapped part
        int x0 = cx - r0, x1 = cx + r0, wb = 1, we = 0;
        if (x0 < 0) {
            wb = dx + x0;
            we = dx - 1;
            x0 = 0;
        }
        if (x1 >= dx) {
            wb = 0;
            we = x1 - dx;
            x1 = dx - 1;
        }
        const bool wrap = wb <= we;
        const uint32_t parts = wrap ? 2u : 1u;
        const uint32_t ny = 2u * r1 + 1u;
        const uint32_t nr = ny * (2u * r2 + 1u) * parts;
        uint32_t total = 0u;
        for (uint32_t q0 = 0; q0 < nr; q0 += 32u) {
            const uint32_t q = q0 + lane;
            uint32_t sb = 0u, len = 0u;
            if (q < nr) {
                const uint32_t row = q / parts, part = q - row * parts;
                int oz = cz - r2 + (int)(row / ny), oy = cy - r1 + (int)(row % ny);
                oz += (oz < 0) ? dz : 0;
                oz -= (oz >= dz) ? dz : 0;
                oy += (oy < 0) ? dy : 0;
                oy -= (oy >= dy) ? dy : 0;
                const uint32_t rb = ((uint32_t)oz * dy + oy) * dx;
                sb = ld_ro<NC>(cell_start + rb + (part ? wb : x0));
                len = ld_ro<NC>(cell_start + rb + (part ? we : x1) + 1) - sb;
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
        bool band = false;
        const auto scan = [&](auto by_ref) {
            uint32_t q = 0u;
            // slot of candidate c (rising by 32 a call)
            const auto slot_of = [&](uint32_t c) -> uint32_t {
                while (range[q + 1u].x <= c) ++q;
                const uint2 r = range[q];
                return r.y + (c - r.x);
            };
            uint32_t sl = lane < total ? slot_of(lane) : 0u;
            uint4 w = ld_ro<NC>(words + sl);
            uint32_t j = SORTED ? sl : ld_ro<NC>(members + sl);
            for (uint32_t c0 = 0; c0 < total; c0 += 32u) {
                const bool on = c0 + lane < total;
                const uint4 wc = w;
                const uint32_t jc = j;
                if (c0 + 32u + lane < total) {
                    sl = slot_of(c0 + 32u + lane);
                    w = ld_ro<NC>(words + sl);
                    j = SORTED ? sl : ld_ro<NC>(members + sl);
                }
                // a lane without a candidate stands outside every radius
                float qx = 0.0f, qy = 0.0f, qz = on ? 0.0f : INFINITY;
                if (by_ref.value && on) {
                    qx = (float)(int32_t)(wc.x - ref.x) * bx.sfix[0];
                    qy = (float)(int32_t)(wc.y - ref.y) * bx.sfix[1];
                    qz = (float)(int32_t)(wc.z - ref.z) * bx.sfix[2];
                }
                const float* hi = s_hi + (ONE_TYPE ? 0u : wc.w);
                const float* lo_ = s_lo + (ONE_TYPE ? 0u : wc.w);
#pragma unroll
                for (int p = 0; p < CH; ++p) {
                    if (p >= (int)cnt) break;
                    float ddx, ddy, ddz;
                    if constexpr (by_ref.value) {
                        ddx = px[p] - qx;
                        ddy = py[p] - qy;
                        ddz = pz[p] - qz;
                    } else {
                        ddx = (float)(int32_t)(pw[p].x - wc.x) * bx.sfix[0];
                        ddy = (float)(int32_t)(pw[p].y - wc.y) * bx.sfix[1];
                        ddz = (float)(int32_t)(pw[p].z - wc.z) * bx.sfix[2] - qz;
                    }
                    const float rs = ddx * ddx + ddy * ddy + ddz * ddz;
                    const bool hit = (rs < (ONE_TYPE ? cut0.hi : hi[pw[p].w])) & (jc != pi[p]);
                    const uint32_t hits = __ballot_sync(0xffffffffu, hit);
                    if (hit) {
                        const uint32_t k = n[p] + __popc(hits & lt);
                        const bool sure = rs < (ONE_TYPE ? cut0.lo : lo_[pw[p].w]);
                        const uint32_t e = sure ? jc : (jc | NL_BAND);
                        band = band || !sure;
                        if (k < NLW_ROW) rows[p][k] = e;
                        else if (k < max_nn) nbrs[(size_t)k * N + pi[p]] = e;
                    }
                    n[p] += __popc(hits);
                }
            }
        };
        if constexpr (REF) {
            // every particle of the chunk in its cell (with 64-bit fixed positions the cell
            // is the word's), or the differences are formed pair by pair
            const bool in_cell = lo || lane >= cnt || (word_in_cell(my_word.x, cx, dx) && word_in_cell(my_word.y, cy, dy) &&
                                                       word_in_cell(my_word.z, cz, dz));
            if (__all_sync(0xffffffffu, in_cell)) scan(std::true_type{});
            else scan(std::false_type{});
        } else {
            scan(std::false_type{});
        }
        band = __any_sync(0xffffffffu, band);
        __syncwarp();  // the rows' entries, before other lanes read them (a vote orders no memory)
        // compaction, in order, of the rows that may hold what does not belong
        uint32_t kept[CH], kept_max = 0u;
#pragma unroll
        for (int p = 0; p < CH; ++p) {
            kept[p] = 0u;
            if (p >= (int)cnt) continue;
            const uint32_t i = pi[p];
            // the particle itself counts as listed for the capacity, as in
            // k_nlist_build_threads, whose scan takes it in
            const uint32_t raw = n[p] + ((ONE_TYPE ? cut0.hi : s_hi[pw[p].w + pw[p].w / ntypes]) > 0.0f ? 1u : 0u);
            const uint32_t stored = min(n[p], max_nn);
            const uint32_t nex = ex_n ? ld_ro<NC>(ex_n + i) : 0u;
            uint32_t m = stored;
            if (band || nex) {
                m = 0u;
                for (uint32_t k0 = 0; k0 < stored; k0 += 32u) {
                    const uint32_t k = k0 + lane;
                    bool keep = k < stored;
                    uint32_t e = 0u;
                    if (keep) {
                        e = k < NLW_ROW ? rows[p][k] : nbrs[(size_t)k * N + i];
                        if (e & NL_BAND) {
                            // the oracle's exact FP64 decision
                            e &= ~NL_BAND;
                            const double r2l = ONE_TYPE ? cut0.rlistsq : s_cut[pw[p].w + ld_ro<NC>(fixed + e).w].rlistsq;
                            keep = nl_exact_within(i, e, r2l, bx, pos, fixed, lo);
                        }
                        for (uint32_t x = 0; x < nex; ++x) keep = keep && ld_ro<NC>(ex_keys + (size_t)x * N + i) != e;
                    }
                    __syncwarp();  // every lane has its entry before one is overwritten
                    const uint32_t mask = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const uint32_t d = m + __popc(mask & lt);
                        if (d < NLW_ROW) rows[p][d] = e;
                        else nbrs[(size_t)d * N + i] = e;
                    }
                    __syncwarp();
                    m += __popc(mask);
                }
            }
            kept[p] = min(m, NLW_ROW);
            kept_max = max(kept_max, kept[p]);
            if (lane == 0u) {
                counts[i] = m;  // what is written, also past the capacity
                if (raw > max_nn) atomicMax(&flags[0], raw);
            }
        }
        __syncwarp();
        // the chunk's rows side by side: lanes of consecutive particles
        {
            constexpr uint32_t STEP = 32u / CH;
            const uint32_t p = lane % CH, kk = lane / CH;
            uint32_t i = 0u, m = 0u;
#pragma unroll
            for (int u = 0; u < CH; ++u)
                if (u == (int)p && u < (int)cnt) {
                    i = pi[u];
                    m = kept[u];
                }
            for (uint32_t k = kk; k < kept_max; k += STEP)
                if (k < m) nbrs[(size_t)k * N + i] = rows[p][k];
        }
        __syncwarp();
        sa += cnt;
    }
}

}  // namespace azp
