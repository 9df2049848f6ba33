// walk64.cuh -- the neighbour walk of the FP64 drop-in drivers (pair forces, DPD
// forces, adjoints).
//
// The drivers are bound by the FP64 pipe (fp64.cuh). The walk therefore finds the
// partners inside r_cut without FP64 instructions: the tpp lanes of a particle scan
// its list in FP32 on the leading 24 bits of the caller's FP64 positions, taken from
// their bit patterns, with a margin above the scan's error, and queue the candidates
// together in shared memory; the queues of the warp are then drained together, the
// lanes of a particle taking its candidates in turn. The caller evaluates a drained
// partner in FP64 and decides r_cut exactly. No shadow of the positions is kept, so
// calls share nothing but the list.
#pragma once

#include "fp64.cuh"

namespace azp
{
constexpr uint32_t WALK_QUEUE = 16;  // queued candidates per lane of a particle
constexpr int WALK_SCAN = 4;         // list entries a lane scans per pass
// queue words of a block of `threads`: a row of 16 per lane and one of padding
// against bank conflicts
constexpr uint32_t walk_queue_words(uint32_t threads) { return threads * (WALK_QUEUE + 1u); }

// The box in FP32. margin: bound of the scan's error in r: the truncation of both
// coordinates (2^-23 of |x| each, |x| <= L) and the FP32 minimum image come to less
// than 2^-20 L per axis. Boxes whose squares leave the FP32 range are not screened.
struct WalkBox {
    float L[3], Linv[3], far, margin;
    bool usable;
};

AZP_D WalkBox walk_box(const double* L)
{
    WalkBox b;
    const double m = fmax(L[0], fmax(L[1], L[2]));
    b.usable = L[0] > 1e-12 && L[1] > 1e-12 && L[2] > 1e-12 && m < 1e12;
    for (int d = 0; d < 3; ++d) {
        b.L[d] = (float)L[d];
        b.Linv[d] = 1.0f / b.L[d];
    }
    b.far = (float)m;
    b.margin = b.far * 2.0e-6f;  // sqrt(3) 2^-20 L
    return b;
}

// FP32 threshold on the scan's r^2 for one type pair: -1 takes none (a pair that is
// off, rcutsq 0), NaN every candidate
AZP_D float walk_threshold(const WalkBox& b, double rcutsq, bool on)
{
    if (!on || !(rcutsq > 0.0)) return -1.0f;
    if (!b.usable || rcutsq < 1e-30 || rcutsq > 1e30) return __int_as_float(0x7fffffff);
    const float r = __double2float_ru(sqrt(rcutsq)) * 1.000002f + b.margin;
    return r * r * 1.000001f;
}

// x towards zero in 24 bits; below the FP32 range 0, above it (or not finite) NaN
AZP_D float leading_float(double x)
{
    const int hi = __double2hiint(x);
    const uint32_t e = (uint32_t)hi & 0x7fffffffu;
    float f = trunc_float(hi, __double2loint(x));
    if (e < 0x38100000u) f = 0.0f;
    if (e >= 0x47e00000u) f = __int_as_float(0x7fffffff);
    return f;
}

// Calls eval(j) for every listed neighbour j of particle i that may lie inside
// r_cut, spread over the particle's tpp lanes. All lanes of the warp call it
// (active false: no row). thr: thresholds by the neighbour's type (the row of
// the particle's own). queue: walk_queue_words(blockDim.x) words of shared memory.
template<class Eval>
AZP_D void walk_fp64(const double4_32a* __restrict__ pos, const uint32_t* __restrict__ nbrs, uint32_t N, uint32_t i,
                     bool active, uint32_t n, uint32_t tpp, const double4_32a& pi, const float* thr, const WalkBox& b,
                     uint32_t* queue, Eval&& eval)
{
    const uint32_t sub = threadIdx.x & (tpp - 1u);
    const uint32_t gshift = (threadIdx.x & 31u) & ~(tpp - 1u);
    const uint32_t gmask = tpp == 32u ? 0xffffffffu : (1u << tpp) - 1u;
    const uint32_t below_me = (1u << sub) - 1u;
    const uint32_t full = tpp * (WALK_QUEUE - WALK_SCAN);
    queue += (threadIdx.x & ~(tpp - 1u)) * (WALK_QUEUE + 1u);
    const float xi = leading_float(pi.x), yi = leading_float(pi.y), zi = leading_float(pi.z);
    // a particle further out than L (the caller may keep unwrapped positions) has a
    // larger error than the margin: every candidate is taken
    const bool out = fmaxf(fmaxf(fabsf(xi), fabsf(yi)), fabsf(zi)) > b.far;
    const uint32_t nmax = __reduce_max_sync(0xffffffffu, active ? n : 0u);
    if (!active) n = 0u;
    const uint32_t* col = nbrs + i;
    uint32_t nq = 0;
    for (uint32_t kb = 0; kb < nmax; kb += WALK_SCAN * tpp) {
        uint32_t jj[WALK_SCAN];
        double4_32a pj[WALK_SCAN];
#pragma unroll
        for (int u = 0; u < WALK_SCAN; ++u) {
            const uint32_t k = kb + sub + u * tpp;
            jj[u] = k < n ? col[(size_t)k * N] : 0xffffffffu;
        }
#pragma unroll
        for (int u = 0; u < WALK_SCAN; ++u) pj[u] = pos[jj[u] != 0xffffffffu ? jj[u] : 0u];
#pragma unroll
        for (int u = 0; u < WALK_SCAN; ++u) {
            const float xj = leading_float(pj[u].x), yj = leading_float(pj[u].y), zj = leading_float(pj[u].z);
            float dx = xi - xj, dy = yi - yj, dz = zi - zj;
            dx -= b.L[0] * rintf(dx * b.Linv[0]);
            dy -= b.L[1] * rintf(dy * b.Linv[1]);
            dz -= b.L[2] * rintf(dz * b.Linv[2]);
            const float rs = dx * dx + dy * dy + dz * dz;
            bool hit = false;
            if (jj[u] != 0xffffffffu) {
                const float t = thr[type_of(pj[u].w)];
                // (NaN on either side: taken)
                hit = t != -1.0f && (!(rs >= t) || out || fmaxf(fmaxf(fabsf(xj), fabsf(yj)), fabsf(zj)) > b.far);
            }
            const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> gshift) & gmask;
            if (hit) queue[nq + __popc(hits & below_me)] = jj[u];
            nq += __popc(hits);
        }
        const bool last = kb + WALK_SCAN * tpp >= nmax;
        if (!last && !__any_sync(0xffffffffu, nq > full)) continue;
        __syncwarp();
        for (uint32_t m = sub; m < nq; m += tpp) eval(queue[m]);
        __syncwarp();
        nq = 0;
    }
}

// L / 2 where v may skip min_image1 (min_image_if); 0, which skips it nowhere but at
// v = 0, for an edge that is not a positive number
AZP_D double half_edge(double L) { return L > 0.0 ? 0.5 * L : 0.0; }

}  // namespace azp
