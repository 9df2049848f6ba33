// engine_kernels.cuh -- the fused force-and-integrate step of the resident engine.
//
// One launch per timestep: pair forces over the column-major list + bond forces
// from the per-particle table (TPP threads per particle, warp-shuffle reduction),
// then, by the group's first lane, Langevin step two at timestep t followed by
// step one of timestep t + 1 (or the Brownian move at t), writing the next
// position buffer and its fixed-point shadow, and the list-rebuild request.
// Arithmetic of each phase follows the standalone kernels (pair.cu, bond.cu,
// integrate.cu) and through them the reference lines cited there.
#pragma once

#include <algorithm>

#include "barrier.cuh"
#include "celllist.cuh"
#include "engine.cuh"
#include "nlist_device.cuh"
#include "philox.cuh"
#include "evaluators.cuh"
#include "pair.cuh"
#include "rebuild_device.cuh"

namespace azp
{
static_assert(MD_PAIR_TBL == PAIR_TBL && MD_BOND_F == BOND_F, "record sizes of MDArgs");
constexpr int MD_BLOCK = 256;
// threads per block of the FP32-force step
#ifndef AZP_FX_BLOCK
#define AZP_FX_BLOCK 256
#endif
constexpr int FX_BLOCK = AZP_FX_BLOCK;
constexpr uint32_t MD_MAX_BOND_TYPES = 32;

struct NoPair {
    static constexpr int SHIFT_SLOT = 7;
    template<typename R> AZP_HD static bool enabled(const R*) { return false; }
    template<typename R> AZP_HD static void eval(const R*, R, R& f, R& e) { f = e = R(0); }
};
struct NoBond {
    template<typename R> AZP_HD static bool eval(const R*, R, R& f, R& e)
    {
        f = e = R(0);
        return true;
    }
    AZP_HD static void prepare_f(const double*, float*) {}
    AZP_D static bool eval_f(const float*, float, float& f, float& e)
    {
        f = e = 0.0f;
        return true;
    }
};

// accumulator with compensated force / energy in FP32
template<typename R> struct Acc;
// FP64 accumulator of the fused step; OUT: energy and virial too
template<bool OUT> struct Acc64 {
    double fx = 0, fy = 0, fz = 0, u = 0, w[6] = {0, 0, 0, 0, 0, 0};
    // force from fdr, virial from fvir (DPD: the conservative part only)
    AZP_D void add(double dx, double dy, double dz, double fdr, double fvir, double e)
    {
        fx += dx * fdr;
        fy += dy * fdr;
        fz += dz * fdr;
        if constexpr (OUT) {
            u += 0.5 * e;
            const double h = 0.5 * fvir;
            w[0] += h * dx * dx;
            w[1] += h * dx * dy;
            w[2] += h * dx * dz;
            w[3] += h * dy * dy;
            w[4] += h * dy * dz;
            w[5] += h * dz * dz;
        }
    }
    AZP_D void reduce(uint32_t tpp)
    {
        for (uint32_t m = tpp >> 1; m > 0; m >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, m);
            fy += __shfl_xor_sync(0xffffffffu, fy, m);
            fz += __shfl_xor_sync(0xffffffffu, fz, m);
            if constexpr (OUT) {
                u += __shfl_xor_sync(0xffffffffu, u, m);
                for (int c = 0; c < 6; ++c) w[c] += __shfl_xor_sync(0xffffffffu, w[c], m);
            }
        }
    }
    static constexpr int WORDS = OUT ? 10 : 3;
    // column p of a [WORDS][n] array of doubles
    AZP_D void put(double* s, uint32_t p, uint32_t n) const
    {
        s[p] = fx;
        s[n + p] = fy;
        s[2 * n + p] = fz;
        if constexpr (OUT) {
            s[3 * n + p] = u;
            for (int c = 0; c < 6; ++c) s[(4 + c) * n + p] = w[c];
        }
    }
    AZP_D void get(const double* s, uint32_t p, uint32_t n)
    {
        fx = s[p];
        fy = s[n + p];
        fz = s[2 * n + p];
        if constexpr (OUT) {
            u = s[3 * n + p];
            for (int c = 0; c < 6; ++c) w[c] = s[(4 + c) * n + p];
        }
    }
};
template<> struct Acc<float> {
    Comp fx{0.f, 0.f}, fy{0.f, 0.f}, fz{0.f, 0.f}, u{0.f, 0.f};
    float w[6] = {0, 0, 0, 0, 0, 0};
    AZP_D void add(float dx, float dy, float dz, float fdr, float e, bool vir)
    {
        fx.add(dx * fdr);
        fy.add(dy * fdr);
        fz.add(dz * fdr);
        u.add(0.5f * e);
        if (vir) {
            const float h = 0.5f * fdr;
            w[0] += h * dx * dx;
            w[1] += h * dx * dy;
            w[2] += h * dx * dz;
            w[3] += h * dy * dy;
            w[4] += h * dy * dz;
            w[5] += h * dz * dz;
        }
    }
    AZP_D static void comb(Comp& c, int m)
    {
        const float s2 = __shfl_xor_sync(0xffffffffu, c.s, m);
        const float c2 = __shfl_xor_sync(0xffffffffu, c.c, m);
        c.add(s2);
        c.c += c2;
    }
    AZP_D void reduce(int tpp, bool vir)
    {
        for (int m = tpp >> 1; m > 0; m >>= 1) {
            comb(fx, m);
            comb(fy, m);
            comb(fz, m);
            comb(u, m);
            if (vir)
                for (int c = 0; c < 6; ++c) w[c] += __shfl_xor_sync(0xffffffffu, w[c], m);
        }
    }
    // sum and carry converted separately: the FP64 result keeps the compensation
    AZP_D double Fx() const { return (double)fx.s + (double)fx.c; }
    AZP_D double Fy() const { return (double)fy.s + (double)fy.c; }
    AZP_D double Fz() const { return (double)fz.s + (double)fz.c; }
    AZP_D double U() const { return (double)u.s + (double)u.c; }
};

// Accumulator of the FP32-force step. The terms of one gather batch (at most
// FX_BATCH pairs, or the bonds) are summed in plain FP32, and each batch sum
// enters the per-particle force with two-sum compensation, so the rounding error
// does not grow with the neighbour count. Energy and virial are accumulated only
// when the step writes them (the integrator needs forces alone).
struct AccFx {
    Comp fx{0.f, 0.f}, fy{0.f, 0.f}, fz{0.f, 0.f}, u{0.f, 0.f};
    float w[6] = {0, 0, 0, 0, 0, 0};
    float bx = 0.f, by = 0.f, bz = 0.f, bu = 0.f;
    AZP_D void add(float dx, float dy, float dz, float fdr, float e, bool out)
    {
        bx += dx * fdr;
        by += dy * fdr;
        bz += dz * fdr;
        if (out) {
            bu += 0.5f * e;
            const float h = 0.5f * fdr;
            w[0] += h * dx * dx;
            w[1] += h * dx * dy;
            w[2] += h * dx * dz;
            w[3] += h * dy * dy;
            w[4] += h * dy * dz;
            w[5] += h * dz * dz;
        }
    }
    // force from fdr, virial from fvir (DPD: the conservative part only)
    AZP_D void add_split(float dx, float dy, float dz, float fdr, float fvir, float e, bool out)
    {
        bx += dx * fdr;
        by += dy * fdr;
        bz += dz * fdr;
        if (out) {
            bu += 0.5f * e;
            const float h = 0.5f * fvir;
            w[0] += h * dx * dx;
            w[1] += h * dx * dy;
            w[2] += h * dx * dz;
            w[3] += h * dy * dy;
            w[4] += h * dy * dz;
            w[5] += h * dz * dz;
        }
    }
    // close a batch: its sums enter the compensated totals
    AZP_D void commit(bool out)
    {
        fx.add(bx);
        fy.add(by);
        fz.add(bz);
        if (out) u.add(bu);
        bx = by = bz = bu = 0.f;
    }
    AZP_D void reduce(int tpp, bool out)
    {
        for (int m = tpp >> 1; m > 0; m >>= 1) {
            Acc<float>::comb(fx, m);
            Acc<float>::comb(fy, m);
            Acc<float>::comb(fz, m);
            if (out) {
                Acc<float>::comb(u, m);
                for (int c = 0; c < 6; ++c) w[c] += __shfl_xor_sync(0xffffffffu, w[c], m);
            }
        }
    }
    AZP_D double Fx() const { return (double)fx.s + (double)fx.c; }
    AZP_D double Fy() const { return (double)fy.s + (double)fy.c; }
    AZP_D double Fz() const { return (double)fz.s + (double)fz.c; }
    AZP_D double U() const { return (double)u.s + (double)u.c; }
};

// ---------------------------------------------------------------- harmonic barrier
// record offset of (timestep ts, type ti) in the barrier table (rows clamped)
AZP_D size_t barrier_slot(const MDArgs& a, unsigned long long ts, uint32_t ti)
{
    const unsigned long long t0 = a.bar_hdr[0], rows = a.bar_hdr[1];
    const unsigned long long r = ts <= t0 ? 0ull : min(ts - t0, rows - 1ull);
    return (size_t)r * a.ntypes + ti;
}

// FP64: the barrier force and energy of particle i (position p) at timestep ts
AZP_D void barrier_fp64(const MDArgs& a, const double4_32a& p, unsigned long long ts, double* f, double& e)
{
    const double2 ck = __ldg(reinterpret_cast<const double2*>(a.bar_tab) + barrier_slot(a, ts, type_of(p.w)));
    const double x[3] = {p.x, p.y, p.z};
    if (a.bar_geom == AZP_BARRIER_PLANAR)
        planar_barrier(x, ck.x, ck.y, f, e);
    else
        spherical_barrier(x, ck.x, ck.y, f, e);
}

// FP32: the same on the fixed-point shadow fi (hi words, type in w)
AZP_D void barrier_fx(const MDArgs& a, const uint4& fi, unsigned long long ts, float* f, float& e)
{
    const BarrierRecF* tab = reinterpret_cast<const BarrierRecF*>(a.bar_tab);
    const size_t k = barrier_slot(a, ts, fi.w);
    BarrierRecF r;
    const int4 raw = __ldg(reinterpret_cast<const int4*>(tab + k));
    r.q = (long long)(((unsigned long long)(uint32_t)raw.y << 32) | (uint32_t)raw.x);
    r.c = __int_as_float(raw.z);
    r.k = __int_as_float(raw.w);
    if (a.bar_geom == AZP_BARRIER_PLANAR)
        planar_barrier_fx(fi, r, a.sfix[1], f, e);
    else
        spherical_barrier_fx(fi, r, a.sfix, f, e);
}

// ---------------------------------------------------------------- walls
// wall_tab row of a type: record (4 doubles), r_cut^2, r_extrap, r_cut, -
constexpr int WALL_TAB = 8;

// FP64 force and energy of every wall on a particle at x (type t), added to
// F[0..2] and F[3]. Out of line: its registers and stack do not count against
// the step's neighbour loop.
static __device__ __noinline__ void engine_walls(int kind, const WallField* __restrict__ wf, const double* __restrict__ tab,
                                          double x0, double x1, double x2, uint32_t t, double* F)
{
    const double* row = tab + (size_t)t * WALL_TAB;
    const double p[4] = {row[0], row[1], row[2], row[3]};
    const double x[3] = {x0, x1, x2};
    double f[3] = {0.0, 0.0, 0.0}, u = 0.0;
    if (kind == AZP_WALL_LJ93)
        walls_force<WallLJ93>(*wf, p, row[4], row[5], x, f, u);
    else
        walls_force<WallColloid>(*wf, p, row[4], row[5], x, f, u);
    F[0] += f[0];
    F[1] += f[1];
    F[2] += f[2];
    F[3] += u;
}

// FP32 screen of the FP32-force step: could any wall act on a particle at
// (x, y, z) (positions good to about L 2^-24, covered by tol)? A wall acts within
// r_cut on its active side, and anywhere on its inactive side with r_extrap > 0.
AZP_D bool walls_near_f(const WallField* __restrict__ wf, const double* __restrict__ tab, uint32_t t, float x,
                        float y, float z, float tol)
{
    const double* row = tab + (size_t)t * WALL_TAB;
    return walls_near(*wf, (float)row[6] + tol, row[5] > 0.0, x, y, z, tol);
}

// |fixed - fixed at the last build|^2 > threshold, in FP32 on exact integer differences
AZP_D bool displaced(const uint4& f, const uint4& fb, const float* sfix, float thresh2)
{
    const float dx = (float)(int32_t)(f.x - fb.x) * sfix[0];
    const float dy = (float)(int32_t)(f.y - fb.y) * sfix[1];
    const float dz = (float)(int32_t)(f.z - fb.z) * sfix[2];
    return dx * dx + dy * dy + dz * dz > thresh2;
}

// ---------------------------------------------------------------- DPD in the step
// The timestep whose forces a step at ts evaluates (the DPD draw's timestep): a
// Langevin step evaluates ts + 1 (HOOMD computes the net force of ts + 1 between the
// halves), a forces-only launch its own timestep.
// alpha in (-1, 1) of the pair (tags ti, tj): the first 64-bit word of the
// pair's Philox block, stream (AZP_RNG_DPD_GENERAL_WEIGHT, timestep, seed),
// counter {0, min tag, max tag, 0}, as azp_dpd_forces draws it
AZP_D void dpd_key(const MDArgs& a, unsigned long long ts, uint32_t& k0, uint32_t& k1)
{
    stream_key(AZP_RNG_DPD_GENERAL_WEIGHT, ts, a.seed, k0, k1);
}

// (the first root is shared by the lanes of h = 1/2 and 1/4; pow out of line)
static __device__ __noinline__ double dpd_weight_pow(double x, double h) { return pow(x, h); }
AZP_D double dpd_weight_engine(double x, double h)
{
    const bool half = h == 0.5, quarter = h == 0.25;
    if (!half && !quarter && h != 1.0) return dpd_weight_pow(x, h);
    if (half || quarter) x = d_sqrt(x);
    if (quarter) x = d_sqrt(x);
    return x;
}

AZP_D float dpd_weight_engine_f(float x, float h)
{
    if (h == 0.5f) return sqrtf(x);
    if (h == 0.25f) return sqrtf(sqrtf(x));
    if (h == 1.0f) return x;
    return powf(x, h);
}

// the last block to finish advances the timestep and arms the next rebuild
AZP_D void finish_step(const MDArgs& a, bool want_rebuild)
{
    if (__any_sync(0xffffffffu, want_rebuild) && (threadIdx.x & 31) == 0) atomicOr(&a.flags[0], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t t = atomicAdd(&a.flags[4], 1u);
        if (t == gridDim.x - 1) {
            __threadfence();
            const uint32_t req = atomicAdd(&a.flags[0], 0u) && !atomicAdd(&a.flags[1], 0u);
            if (a.set_cond) cudaGraphSetConditional(a.next_cond, req ? 1u : 0u);
            a.flags[4] = 0u;
            *a.d_timestep_rw = *a.d_timestep_rw + 1ull;
        }
    }
}

// one pair in FP64: dx = x_i - x_j, dv = v_i - v_j; rec as in DpdEngine.
// Returns false outside r_cut (rsq >= rcutsq).
AZP_D bool dpd_term_fp64(const double* rec, double rcutsq, double dx, double dy, double dz, double dvx, double dvy,
                         double dvz, uint32_t k0, uint32_t k1, uint32_t tgi, uint32_t tgj, double& fdr, double& fc,
                         double& e)
{
    const double rs = rsq_exact(dx, dy, dz);
    if (!less_nonneg(rs, rcutsq)) return false;
    const double rcinv = rec[0], rc = rec[1], A = rec[2], gamma = rec[3];
    double rinv;
    const double r = d_sqrt(rs, rinv);
    const double dot = dx * dvx + dy * dvy + dz * dvz;
    fc = A * (rinv - rcinv);
    const double wR = dpd_weight_engine(nonneg(1.0 - r * rcinv), rec[4]) * rinv;
    const Philox4 ph = philox4x32_10(0u, min(tgi, tgj), max(tgi, tgj), 0u, k0, k1);
    const double alpha = -1.0 + 2.0 * open01(ph.v[0], ph.v[1]);
    fdr = fc - gamma * wR * wR * dot + rec[5] * wR * alpha;
    e = A * (rc - r) - 0.5 * A * rcinv * (rcutsq - rs);
    return true;
}

// a pair's force with the rare modifications: the smoothing of mode xplor (and the
// energy shift it needs) and the cap of the overlap relaxation. Out of line, with an
// evaluation of its own, so that the plain step computes no energy for it.
template<class PE>
static __device__ __noinline__ double2 adjusted_fp64(const MDArgs& a, const double* rec, double rsq)
{
    double fdr, e;
    PE::eval(rec, rsq, fdr, e);
    e -= rec[PE::SHIFT_SLOT];
    xplor(rec + PAIR_REC, rsq, fdr, e);
    if (a.capped && fdr * fdr * rsq > a.fcap * a.fcap) fdr = copysign(a.fcap / sqrt(rsq), fdr);
    return make_double2(fdr, e);
}

// FP64 step: FP64 positions, forces and integration, the oracle's rounding for
// every decision. Bound by the FP64 pipe (fp64.cuh), so FP64 instructions are kept
// to the pairs inside r_cut and run on full warps. The tpp lanes of a particle scan
// its list on the 16-byte fixed-point shadow in FP32, with a margin above the
// scan's error (a.screen), and queue the candidates together in shared memory;
// the queues of the warp are then drained together, the lanes of a particle taking
// its candidates in turn. A drained pair takes its FP64 displacement (the minimum
// image where the bits say that it changes anything), the oracle's exact r^2 and the
// r_cut decision. The particles' sums then move to the block's first threads, so
// that bonds and integration run on full warps too.
// Measured (ncu, LJ fluid of N = 54,872, 131 listed and 90 in range a particle):
// 950 us with one thread per particle evaluating as it walked, 250 us so; melt of
// N = 131,300: 274 -> 118 us.
constexpr uint32_t MD_QUEUE = 16;  // queued candidates per lane of a particle
constexpr int MD_SCAN = 4;         // list entries a lane scans per pass

// The body for the block-th MD_BLOCK / tpp particles at timestep ts; whether the calling
// thread's particle asks for a list rebuild. smem_raw: md_step_smem bytes. NC: loads of
// the particle arrays through the read-only path (nothing in the launch writes them).
template<class PE, class BE, int INTEG, bool OUT, bool NC>
AZP_D bool md_step_body(const MDArgs& a, uint32_t block, unsigned long long ts, unsigned char* smem_raw)
{
    constexpr bool PAIR = !std::is_same<PE, NoPair>::value;
    constexpr bool DPD = std::is_same<PE, DpdEngine>::value;
    const uint32_t nt2 = a.ntypes * a.ntypes;
    double* s_gamma = reinterpret_cast<double*>(smem_raw);
    double* s_noise = s_gamma + a.ntypes;
    double* s_rec = s_noise + a.ntypes;
    double* s_bond = s_rec + nt2 * REC64;
    double* s_sum = s_bond + a.nbondtypes * BOND_REC;
    const uint32_t tpp = (uint32_t)a.tpp;
    const uint32_t P = MD_BLOCK >> a.tpp_shift;  // particles of the block
    float* s_screen = reinterpret_cast<float*>(s_sum + (tpp > 1u ? Acc64<OUT>::WORDS * P : 0u));
    if constexpr (PAIR) {
        for (uint32_t t = threadIdx.x; t < nt2; t += blockDim.x) {
            const double* rec = a.pair_table + (size_t)t * PAIR_TBL;
            const bool on = PE::enabled(rec);
            prepare64<PE>(rec, on, s_rec + (size_t)t * REC64);
            s_screen[t] = on ? __double2float_ru(rec[PAIR_REC] * (1.0 + (double)a.screen)) : -1.0f;
        }
    }
    if constexpr (!std::is_same<BE, NoBond>::value)
        for (uint32_t t = threadIdx.x; t < a.nbondtypes; t += blockDim.x)
            BE::prepare(a.bond_params + (size_t)t * AZP_BOND_PARAM_DOUBLES, s_bond + (size_t)t * BOND_REC);
    if (INTEG != MD_FORCES_ONLY && !a.use_lambda)
        for (uint32_t t = threadIdx.x; t < a.ntypes; t += blockDim.x) {
            s_gamma[t] = a.gamma[t];
            s_noise[t] = a.noise[t];
        }
    __syncthreads();

    const double half0 = 0.5 * a.L[0], half1 = 0.5 * a.L[1], half2 = 0.5 * a.L[2];
    Acc64<OUT> acc;
    uint32_t i = block * P + (threadIdx.x >> a.tpp_shift);
    bool active = i < a.N;
    double4_32a pi = make_double4_32a(0.0, 0.0, 0.0, 0.0);
    if (active) pi = a.pos[i];
    // ---------------------------------------------------------------- pair
    if constexpr (PAIR) {
        const uint32_t sub = threadIdx.x & (tpp - 1u);
        const uint32_t gshift = (threadIdx.x & 31u) & ~(tpp - 1u);
        const uint32_t gmask = tpp == 32u ? 0xffffffffu : (1u << tpp) - 1u;
        const uint32_t below_me = (1u << sub) - 1u;
        // a row of 16 entries per lane and one of padding, against bank conflicts
        uint32_t* queue = reinterpret_cast<uint32_t*>(s_screen + nt2) + (threadIdx.x & ~(tpp - 1u)) * (MD_QUEUE + 1u);
        const uint32_t full = tpp * (MD_QUEUE - MD_SCAN);
        const uint32_t n = active ? min(ld_ro<NC>(a.counts + i), a.max_nn) : 0u;
        const uint32_t nmax = __reduce_max_sync(0xffffffffu, n);
        const uint32_t row = type_of(pi.w) * a.ntypes;
        uint4 fi = make_uint4(0u, 0u, 0u, 0u);
        uint32_t k0 = 0, k1 = 0, tgi = 0;
        double4_32a vi{};
        if (active) {
            fi = ld_ro<NC>(a.fix + i);
            if constexpr (DPD) {
                dpd_key(a, ts + (INTEG == MD_INTEG_LANGEVIN ? 1ull : 0ull), k0, k1);
                tgi = a.tag[i];
                vi = reinterpret_cast<const double4_32a*>(a.dvel)[i];
            }
        }
        const uint32_t* col = a.nbrs + i;
        uint32_t nq = 0;
        for (uint32_t kb = 0; kb < nmax; kb += MD_SCAN * tpp) {
            uint32_t jj[MD_SCAN];
            uint4 fj[MD_SCAN];
#pragma unroll
            for (int u = 0; u < MD_SCAN; ++u) {
                const uint32_t k = kb + sub + u * tpp;
                jj[u] = k < n ? ld_ro<NC>(col + (size_t)k * a.N) : 0xffffffffu;
            }
#pragma unroll
            for (int u = 0; u < MD_SCAN; ++u) fj[u] = ld_ro<NC>(a.fix + (jj[u] != 0xffffffffu ? jj[u] : 0u));
#pragma unroll
            for (int u = 0; u < MD_SCAN; ++u) {
                const float dx = (float)(int32_t)(fi.x - fj[u].x) * a.sfix[0];
                const float dy = (float)(int32_t)(fi.y - fj[u].y) * a.sfix[1];
                const float dz = (float)(int32_t)(fi.z - fj[u].z) * a.sfix[2];
                const float rs = dx * dx + dy * dy + dz * dz;
                const bool hit = jj[u] != 0xffffffffu && rs < s_screen[row + fj[u].w];
                const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> gshift) & gmask;
                if (hit) queue[nq + __popc(hits & below_me)] = jj[u];
                nq += __popc(hits);
            }
            const bool last = kb + MD_SCAN * tpp >= nmax;
            if (!last && !__any_sync(0xffffffffu, nq > full)) continue;
            __syncwarp();
            for (uint32_t m = sub; m < nq; m += tpp) {
                const uint32_t j = queue[m];
                const double4_32a pj = a.pos[j];
                const double dx = min_image_if(pi.x - pj.x, half0, a.L[0], a.Linv[0]);
                const double dy = min_image_if(pi.y - pj.y, half1, a.L[1], a.Linv[1]);
                const double dz = min_image_if(pi.z - pj.z, half2, a.L[2], a.Linv[2]);
                const uint32_t tp = row + type_of(pj.w);
                const double* rec = s_rec + (size_t)tp * REC64;
                double fdr, e;
                if constexpr (DPD) {
                    const double4_32a vj = reinterpret_cast<const double4_32a*>(a.dvel)[j];
                    double fc;
                    if (dpd_term_fp64(rec, rec[CUT64], dx, dy, dz, vi.x - vj.x, vi.y - vj.y, vi.z - vj.z, k0, k1, tgi,
                                      a.tag[j], fdr, fc, e))
                        acc.add(dx, dy, dz, fdr, fc, e);
                } else {
                    double rsq;
                    if (!pair_inside(dx, dy, dz, rec + CUT64, rsq)) continue;
                    if (a.xplor | a.capped) {
                        const double2 fe = adjusted_fp64<PE>(a, a.pair_table + (size_t)tp * PAIR_TBL, rsq);
                        fdr = fe.x;
                        e = fe.y;
                    } else {
                        Pair64<PE>::template force64<OUT>(rec, rsq, fdr, e);
                    }
                    acc.add(dx, dy, dz, fdr, fdr, e);
                }
            }
            __syncwarp();
            nq = 0;
        }
        if (tpp > 1u) {
            acc.reduce(tpp);
            if (sub == 0u) acc.put(s_sum, threadIdx.x >> a.tpp_shift, P);
        }
    }
    if (tpp > 1u) {
        // one thread per particle from here on: the block's first P
        i = block * P + threadIdx.x;
        active = threadIdx.x < P && i < a.N;
        if constexpr (PAIR) {
            __syncthreads();
            if (active) acc.get(s_sum, threadIdx.x, P);
        }
        if (active) pi = a.pos[i];
    }
    if (active) {
        // ---------------------------------------------------------------- bonds
        if constexpr (!std::is_same<BE, NoBond>::value) {
            const uint32_t nb = ld_ro<NC>(a.bt_n + i);
            for (uint32_t k = 0; k < nb; ++k) {
                const uint2 e2 = ld_ro<NC>(a.bt + (size_t)k * a.N + i);
                const double4_32a pj = a.pos[e2.x];
                double dx, dy, dz;
                if constexpr (bond_uses_image<BE>::value) {
                    // (x_i - x_j) + (img_i - img_j) L (src/ImagePotentialBond.h:144-152)
                    const int* gi = a.img0 + 3 * (size_t)i;
                    const int* gj = a.img0 + 3 * (size_t)e2.x;
                    dx = __dadd_rn(pi.x - pj.x, __dmul_rn((double)(gi[0] - gj[0]), a.L[0]));
                    dy = __dadd_rn(pi.y - pj.y, __dmul_rn((double)(gi[1] - gj[1]), a.L[1]));
                    dz = __dadd_rn(pi.z - pj.z, __dmul_rn((double)(gi[2] - gj[2]), a.L[2]));
                } else {
                    dx = min_image_if(pi.x - pj.x, half0, a.L[0], a.Linv[0]);
                    dy = min_image_if(pi.y - pj.y, half1, a.L[1], a.Linv[1]);
                    dz = min_image_if(pi.z - pj.z, half2, a.L[2], a.Linv[2]);
                }
                const double rsq = rsq_exact(dx, dy, dz);
                double fdr, en;
                if (!BE::eval_prepared(s_bond + (size_t)e2.y * BOND_REC, rsq, fdr, en)) {
                    atomicOr(&a.flags[1], AZP_EBIT_BOND);
                    continue;
                }
                acc.add(dx, dy, dz, fdr, fdr, en);
            }
        }
    }

    bool want_rebuild = false;
    if (active) {
        double Fx = acc.fx, Fy = acc.fy, Fz = acc.fz;
        double Ub = 0.0;
        if (a.bar_geom >= 0) {
            // the barrier's force joins the net force (src/HarmonicBarrier.h:149-180)
            double fb[3] = {0.0, 0.0, 0.0};
            barrier_fp64(a, pi, ts + (INTEG == MD_INTEG_LANGEVIN ? 1ull : 0ull), fb, Ub);
            Fx += fb[0];
            Fy += fb[1];
            Fz += fb[2];
        }
        double fw[4] = {0.0, 0.0, 0.0, 0.0};
        if (a.wall_kind >= 0) {
            // the wall potential's force joins the net force (HOOMD adds the
            // external wall compute into net_force)
            engine_walls(a.wall_kind, a.walls, a.wall_tab, pi.x, pi.y, pi.z, type_of(pi.w), fw);
            Fx += fw[0];
            Fy += fw[1];
            Fz += fw[2];
            Ub += fw[3];
        }
        if constexpr (OUT) {
            a.out_force[i] = make_double4_32a(Fx, Fy, Fz, acc.u + Ub);
            double wv[6] = {acc.w[0], acc.w[1], acc.w[2], acc.w[3], acc.w[4], acc.w[5]};
            if (a.wall_kind >= 0) {
                wv[0] += fw[0] * pi.x;
                wv[1] += fw[0] * pi.y;
                wv[2] += fw[0] * pi.z;
                wv[3] += fw[1] * pi.y;
                wv[4] += fw[1] * pi.z;
                wv[5] += fw[2] * pi.z;
            }
            for (int c = 0; c < 6; ++c) a.out_virial[(size_t)c * a.N + i] = wv[c];
        }
        if constexpr (INTEG != MD_FORCES_ONLY) {
            double4_32a p = pi;
            const uint32_t ti = type_of(p.w);
            const uint32_t tg = a.tag[i];
            bool moved = false;
            // The reference arithmetic; the per-type noise amplitude
            // sqrt(6 gamma kT / dt) comes from a host table built with the same
            // double operations, so the draws stay bit-exact
            const double gam = a.use_lambda ? a.lambda * a.diameter[i] : s_gamma[ti];
            // the method's temperature at this timestep (a table when it varies)
            double kTv = a.kT, nz = a.use_lambda ? 0.0 : s_noise[ti];
            if (a.kT_hdr) {
                const size_t r = kT_row(a, ts);
                kTv = a.kT_tab[r];
                nz = a.noise_tab[r * a.ntypes + ti];
            }
            const double c = a.noiseless ? 0.0 : (a.use_lambda ? sqrt(6.0 * gam * kTv / a.dt) : nz);
            const bool mover = in_group(a, ti);
            double ux, uy, uz;
            flow_at(a.flow, p.y, ux, uy, uz);
            double r0 = 0.0, r1 = 0.0, r2 = 0.0;
            if constexpr (INTEG == MD_INTEG_LANGEVIN) {
                uniform3(AZP_RNG_LANGEVIN_FLOW, ts, a.seed, tg, -c, c - (-c), r0, r1, r2);
                double4_32a v = a.vel[i];
                const double minv = rcp(v.w);
                const double ax = (Fx + (r0 - gam * (v.x - ux))) * minv;
                const double ay = (Fy + (r1 - gam * (v.y - uy))) * minv;
                const double az = (Fz + (r2 - gam * (v.z - uz))) * minv;
                const double h = 0.5 * a.dt;
                if (mover) {
                    v.x += h * ax;
                    v.y += h * ay;
                    v.z += h * az;
                }
                if (a.next) {
                    // step one of the next timestep with the acceleration just computed
                    if (mover) {
                        p.x += (v.x + h * ax) * a.dt;
                        p.y += (v.y + h * ay) * a.dt;
                        p.z += (v.z + h * az) * a.dt;
                        v.x += h * ax;
                        v.y += h * ay;
                        v.z += h * az;
                    }
                    moved = true;
                } else if (mover) {
                    a.accel[3 * i] = ax;
                    a.accel[3 * i + 1] = ay;
                    a.accel[3 * i + 2] = az;
                }
                a.vel[i] = v;
            } else {
                uniform3(AZP_RNG_BROWNIAN_FLOW, ts, a.seed, tg, -c, c - (-c), r0, r1, r2);
                double dx = (ux + (Fx + r0) / gam) * a.dt;
                double dy = (uy + (Fy + r1) / gam) * a.dt;
                double dz = (uz + (Fz + r2) / gam) * a.dt;
                if (a.max_disp > 0.0) {
                    dx = fmin(fmax(dx, -a.max_disp), a.max_disp);
                    dy = fmin(fmax(dy, -a.max_disp), a.max_disp);
                    dz = fmin(fmax(dz, -a.max_disp), a.max_disp);
                }
                if (mover) {
                    p.x += dx;
                    p.y += dy;
                    p.z += dz;
                }
                moved = true;
            }
            if (moved) {
                int wx = 0, wy = 0, wz = 0;
                wrap_if(p.x, wx, a.L[0], a.lo[0], a.hi[0]);
                wrap_if(p.y, wy, a.L[1], a.lo[1], a.hi[1]);
                wrap_if(p.z, wz, a.L[2], a.lo[2], a.hi[2]);
                if (wx | wy | wz) {
                    a.image[3 * i] += wx;
                    a.image[3 * i + 1] += wy;
                    a.image[3 * i + 2] += wz;
                }
                a.pos_next[i] = p;
                uint4 f;
                f.x = to_fixed(p.x, a.Linv[0]);
                f.y = to_fixed(p.y, a.Linv[1]);
                f.z = to_fixed(p.z, a.Linv[2]);
                f.w = ti;
                a.fix_next[i] = f;
                want_rebuild = displaced(f, a.fix_build[i], a.sfix, a.disp_thresh2);
                if (!(finite_bits(p.x) && finite_bits(p.y) && finite_bits(p.z)))
                    atomicOr(&a.flags[1], AZP_EBIT_NONFINITE);
            }
        }
    }
    return want_rebuild;
}

template<class PE, class BE, int INTEG, bool OUT>
__global__ void __launch_bounds__(MD_BLOCK) k_md_step(const __grid_constant__ MDArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const bool want = md_step_body<PE, BE, INTEG, OUT, true>(a, blockIdx.x, *a.d_timestep, smem_raw);
    if constexpr (INTEG != MD_FORCES_ONLY) finish_step(a, want);
}

// dynamic shared memory of k_md_step
template<class PE> inline size_t md_step_smem(const MDArgs& a)
{
    const size_t nt2 = (size_t)a.ntypes * a.ntypes;
    return 2 * a.ntypes * sizeof(double) + nt2 * REC64 * sizeof(double) +
           (size_t)a.nbondtypes * BOND_REC * sizeof(double) + nt2 * sizeof(float) +
           (a.tpp > 1 ? (size_t)(MD_BLOCK / a.tpp) * (a.out ? 10 : 3) * sizeof(double) : 0) +
           (std::is_same<PE, NoPair>::value ? 0 : MD_BLOCK * (MD_QUEUE + 1) * sizeof(uint32_t));
}

// ---------------------------------------------------------------- FP32-force step
// State: 64-bit fixed positions (fix = high words, lo = low words) and
// float-float velocities (fixed64.cuh). Pair and bond arithmetic in FP32 on the
// exact integer displacement of the high words, compensated force / energy sums;
// the r_cut decision is the oracle's FP64 one within 4e-6 of r_cut^2, on the
// full 64-bit positions. Integration with FP32 increments accumulated exactly
// (positions) or in float-float (velocities): no FP64 instruction per particle.

// |x_i - x_j|^2 < rc2 exactly as the FP64 oracle decides it, on the 64-bit positions
AZP_D bool inside_exact(const MDArgs& a, uint32_t i, uint32_t j, double rc2)
{
    const uint4 hi = a.fix[i], hj = a.fix[j];
    const uint4 li = a.flo[i], lj = a.flo[j];
    const double vx = min_image1(fx_to_double(fx_join(hi.x, li.x), a.l64[0]) - fx_to_double(fx_join(hj.x, lj.x), a.l64[0]),
                                 a.L[0], a.Linv[0]);
    const double vy = min_image1(fx_to_double(fx_join(hi.y, li.y), a.l64[1]) - fx_to_double(fx_join(hj.y, lj.y), a.l64[1]),
                                 a.L[1], a.Linv[1]);
    const double vz = min_image1(fx_to_double(fx_join(hi.z, li.z), a.l64[2]) - fx_to_double(fx_join(hj.z, lj.z), a.l64[2]),
                                 a.L[2], a.Linv[2]);
    return rsq_exact(vx, vy, vz) < rc2;
}

// exact minimum-image displacement of one axis from the 64-bit fixed positions
// (the wrapping 64-bit difference), in FP64 (one rounding)
AZP_D double fx_disp(uint32_t hi_i, uint32_t lo_i, uint32_t hi_j, uint32_t lo_j, double l64)
{
    const long long d = (long long)((unsigned long long)fx_join(hi_i, lo_i) - (unsigned long long)fx_join(hi_j, lo_j));
    return (double)d * l64;
}

// r^2 of the displacement between two fixed-point positions (high words): in a
// cubic box (AZP_FX_IRSQ=1, the default) the exact integer sum of squares of the
// int32 differences (each below 2^62, the sum below 2^64) rounded once to FP32
// and scaled by (L / 2^32)^2 held as a float pair; otherwise the sum of squares of
// the FP32 components. The integer form's r^2 is about three times closer (1.2e-7
// against 3.4e-7 relative), which r^-14 and the bond polynomial amplify: on the
// melt at N = 1M the force error against the FP64 oracle was 8.2e-6 to 1.07e-5
// over the end states of the bench runs with the FP32 components (over the 1e-5
// budget once) and 5.8-6.1e-6 with the integer form, for a step kernel about
// 9 % longer (0.090 -> 0.098 ms).
#ifndef AZP_FX_IRSQ
#define AZP_FX_IRSQ 1
#endif
AZP_D float fx_rsq(const MDArgs& a, const uint4& fi, const uint4& fj, float dx, float dy, float dz)
{
#if AZP_FX_IRSQ
    if (a.cubic) {
        const long long ix = (int32_t)(fi.x - fj.x), iy = (int32_t)(fi.y - fj.y), iz = (int32_t)(fi.z - fj.z);
        const unsigned long long q = (unsigned long long)(ix * ix) + (unsigned long long)(iy * iy) +
                                     (unsigned long long)(iz * iz);
        // (the conversion runs on the FP64 pipe, 32 % busy; a shifted 32-bit
        // conversion on other pipes measured slower, 0.102 against 0.098 ms)
        const float qf = __ull2float_rn(q);
        return fmaf(qf, a.s2h, qf * a.s2l);
    }
#endif
    return dx * dx + dy * dy + dz * dz;
}

// r^2 and the contact difference dq = c^2 - r^2 of a colloid point-sphere or
// sphere-sphere pair, each rounded once to FP32, for PE::eval_gap.
// AZP_COLLOID_GAP 2 (default; cubic boxes): from the 64-bit displacement rounded
// to 2^-32 L, whose integer sum of squares q (below 2^62 for a pair inside the
// half box) is exact, with c^2 held in the same units as the 64-bit integer
// contact_q (c^2 2^64 / L^2): dq = contact_q - q is an exact integer difference,
// so the cancellation costs nothing and no FP64 instruction runs. Other boxes, and
// AZP_COLLOID_GAP 1: in FP64 from the exact 64-bit displacement. Measured on the
// colloid mixture (N = 262,144, 5000 Brownian steps): FP64 841 timesteps/s, force
// error 6.7e-6; integer 968, 7.2e-6; the FP32 forms on the FP32 r^2 (0) 1,399 but
// 1.1e-5, over the 1e-5 budget; the exact difference only for r^2 < 2 c^2 1,015,
// 8.2e-6.
#ifndef AZP_COLLOID_GAP
#define AZP_COLLOID_GAP 2
#endif
// the integer r^2, in units of (L / 2^32)^2, of the 64-bit fixed-point
// displacement rounded to 2^-32 L per axis; exact, and below 2^62 for a pair
// inside the half box
AZP_D long long fx_rsq_rounded(const uint4& fi, const uint4& li, const uint4& fj, const uint4& lj)
{
    const auto axis = [](uint32_t hi_i, uint32_t lo_i, uint32_t hi_j, uint32_t lo_j) -> long long {
        const unsigned long long d = (unsigned long long)fx_join(hi_i, lo_i) - (unsigned long long)fx_join(hi_j, lo_j);
        return (long long)(d + 0x80000000ull) >> 32;
    };
    const long long ix = axis(fi.x, li.x, fj.x, lj.x), iy = axis(fi.y, li.y, fj.y, lj.y),
                    iz = axis(fi.z, li.z, fj.z, lj.z);
    return ix * ix + iy * iy + iz * iz;
}
template<class PE, bool NC>
AZP_D void gap_args(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t i, uint32_t j, uint32_t tp,
                    float& rsq, float& dq)
{
    const uint4 li = ld_ro<NC>(a.flo + i), lj = ld_ro<NC>(a.flo + j);
#if AZP_COLLOID_GAP == 2
    if (a.contact_q) {
        const long long q = fx_rsq_rounded(fi, li, fj, lj);
        const long long dqi = __ldg(a.contact_q + tp) - q;
        const float qf = __ll2float_rn(q), df = __ll2float_rn(dqi);
        rsq = fmaf(qf, a.s2h, qf * a.s2l);
        dq = fmaf(df, a.s2h, df * a.s2l);
        return;
    }
#endif
    const double vx = fx_disp(fi.x, li.x, fj.x, lj.x, a.l64[0]);
    const double vy = fx_disp(fi.y, li.y, fj.y, lj.y, a.l64[1]);
    const double vz = fx_disp(fi.z, li.z, fj.z, lj.z, a.l64[2]);
    const double rsq_d = vx * vx + vy * vy + vz * vz;
    rsq = (float)rsq_d;
    dq = (float)(PE::contact2(a.pair_table + (size_t)tp * PAIR_TBL) - rsq_d);
}

// ONE: a single-type system; the type pair is 0 at compile time, so the record
// lookups resolve to the caller's registers
template<class PE, bool ONE, bool NC>
AZP_D void pair_term_fx(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t i, uint32_t j,
                        const float* s_rec, const double* s_rc2, AccFx& acc, bool vir)
{
    const float dx = (float)(int32_t)(fi.x - fj.x) * a.sfix[0];
    const float dy = (float)(int32_t)(fi.y - fj.y) * a.sfix[1];
    const float dz = (float)(int32_t)(fi.z - fj.z) * a.sfix[2];
    const float rsq = fx_rsq(a, fi, fj, dx, dy, dz);
    const uint32_t tp = ONE ? 0u : fi.w * a.ntypes + fj.w;
    const float* rec = s_rec + (size_t)tp * PAIR_TBL;
    const float* cut = rec + PAIR_REC;
    const float rc2 = cut[0];
    if (rsq >= rc2 * 1.000004f || !PE::enabled(rec)) return;
    if (rsq >= rc2 * 0.999996f && !inside_exact(a, i, j, s_rc2[tp])) return;
    float fdr, e;
    if constexpr (has_gap_form<PE>::value) {
        if (AZP_COLLOID_GAP && PE::gap_form(rec)) {
            // the cancelling contact difference (colloid point-sphere and
            // sphere-sphere forms) formed exactly
            float rg, dq;
            gap_args<PE, NC>(a, fi, fj, i, j, tp, rg, dq);
            PE::eval_gap(rec, rg, dq, fdr, e);
        } else {
            PE::eval(rec, rsq, fdr, e);
        }
    } else {
        PE::eval(rec, rsq, fdr, e);
    }
    e -= rec[PE::SHIFT_SLOT];
    xplor(cut, rsq, fdr, e);
    if (a.fcapf > 0.0f && fdr * fdr * rsq > a.fcapf * a.fcapf) fdr = copysignf(a.fcapf * rsqrtf(rsq), fdr);
    acc.add(dx, dy, dz, fdr, e, vir);
}

// pair_term_fx for a candidate that may be a padding slot (ok false) or lie
// outside r_cut: the evaluator runs on every lane (at r_cut where the pair does
// not count) and the pair's terms are masked, so a batch has no per-lane exits;
// only the rare candidate in the band around r_cut takes the exact FP64 branch
template<class PE, bool TILE, bool ONE, bool NC>
AZP_D void pair_term_fx_masked(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t i, uint32_t ent, bool ok,
                               const float* s_rec, const double* s_rc2, AccFx& acc, bool vir,
                               const uint32_t* trec = nullptr)
{
    // the particle index of the entry, needed only on the rare exact paths
    const auto jof = [&]() -> uint32_t {
        if constexpr (TILE) return tile_decode(trec, ent);
        return ent;
    };
    const float dx = (float)(int32_t)(fi.x - fj.x) * a.sfix[0];
    const float dy = (float)(int32_t)(fi.y - fj.y) * a.sfix[1];
    const float dz = (float)(int32_t)(fi.z - fj.z) * a.sfix[2];
    const float rsq = fx_rsq(a, fi, fj, dx, dy, dz);
    const uint32_t tp = ONE ? 0u : fi.w * a.ntypes + fj.w;
    const float* rec = s_rec + (size_t)tp * PAIR_TBL;
    const float* cut = rec + PAIR_REC;
    const float rc2 = cut[0];
    const bool on = ok && PE::enabled(rec);
    bool in = on && rsq < rc2 * 0.999996f;
    if (on && !in && rsq < rc2 * 1.000004f) in = inside_exact(a, i, jof(), s_rc2[tp]);
    const float rs = in ? rsq : rc2;
    float fdr, e;
    if constexpr (has_gap_form<PE>::value && AZP_COLLOID_GAP != 0) {
        // the cancelling contact difference of the colloid point-sphere and
        // sphere-sphere forms formed exactly for a pair inside r_cut (a masked
        // slot takes any finite gap); every lane then runs one evaluation of its
        // own form, so a warp never runs a gap form twice
        float rg = rs, dq = 0.0f;
        if (PE::gap_form(rec)) {
            dq = PE::contact2_f(rec) - rs;
            if (in) gap_args<PE, NC>(a, fi, fj, i, jof(), tp, rg, dq);
        }
        PE::eval_any(rec, rg, dq, fdr, e);
    } else {
        PE::eval(rec, rs, fdr, e);
    }
    e -= rec[PE::SHIFT_SLOT];
    xplor(cut, rs, fdr, e);
    if (a.fcapf > 0.0f && fdr * fdr * rs > a.fcapf * a.fcapf) fdr = copysignf(a.fcapf * rsqrtf(rs), fdr);
    acc.add(dx, dy, dz, in ? fdr : 0.0f, in ? e : 0.0f, vir);
}

// A DPD pair near r_cut in a box that is not cubic, in FP64 from the 64-bit
// positions. Out of line: its registers do not count against the pair loop.
static __device__ __noinline__ bool dpd_near_cutoff_fp64(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t i,
                                                         uint32_t j, uint32_t tp, double rc2, const float4& vi,
                                                         const float4& vj, uint32_t tgi, uint32_t tgj, uint32_t k0,
                                                         uint32_t k1, float& dx, float& dy, float& dz, float& fdr,
                                                         float& fc, float& e)
{
    const uint4 li = a.flo[i], lj = a.flo[j];
    const double ddx = min_image1(fx_to_double(fx_join(fi.x, li.x), a.l64[0]) - fx_to_double(fx_join(fj.x, lj.x), a.l64[0]),
                                  a.L[0], a.Linv[0]);
    const double ddy = min_image1(fx_to_double(fx_join(fi.y, li.y), a.l64[1]) - fx_to_double(fx_join(fj.y, lj.y), a.l64[1]),
                                  a.L[1], a.Linv[1]);
    const double ddz = min_image1(fx_to_double(fx_join(fi.z, li.z), a.l64[2]) - fx_to_double(fx_join(fj.z, lj.z), a.l64[2]),
                                  a.L[2], a.Linv[2]);
    double f, c, u;
    if (!dpd_term_fp64(a.pair_table + (size_t)tp * PAIR_TBL, rc2, ddx, ddy, ddz, (double)(vi.x - vj.x),
                       (double)(vi.y - vj.y), (double)(vi.z - vj.z), k0, k1, tgi, tgj, f, c, u))
        return false;
    dx = (float)ddx;
    dy = (float)ddy;
    dz = (float)ddz;
    fdr = (float)f;
    fc = (float)c;
    e = (float)u;
    return true;
}

// DPD pair in the FP32-force step: FP32 on the exact fixed-point displacement,
// FP64 from the full 64-bit positions within 0.2 % of r_cut^2 (the weight
// (1 - r / r_cut)^(s/2) is steep there, and the cutoff decision is the oracle's);
// velocities and tag from the step's snapshot (float4: v, tag bits)
template<bool ONE, bool NC>
AZP_D void pair_term_dpd_fx(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t i, uint32_t j,
                            const float* s_rec, const double* s_rc2, AccFx& acc, bool vir, const float4& vi,
                            uint32_t tgi, uint32_t k0, uint32_t k1)
{
    const float dx = (float)(int32_t)(fi.x - fj.x) * a.sfix[0];
    const float dy = (float)(int32_t)(fi.y - fj.y) * a.sfix[1];
    const float dz = (float)(int32_t)(fi.z - fj.z) * a.sfix[2];
    const float rs = fx_rsq(a, fi, fj, dx, dy, dz);
    const uint32_t tp = ONE ? 0u : fi.w * a.ntypes + fj.w;
    const float* rec = s_rec + (size_t)tp * PAIR_TBL;
    const float rc2 = rec[PAIR_REC];
    if (!(rc2 > 0.0f) || rs >= rc2 * 1.000004f) return;
    const float4 vj = ld_ro<NC>(reinterpret_cast<const float4*>(a.dvel) + j);
    const uint32_t tgj = __float_as_uint(vj.w);
    if (rs >= rc2 * 0.998f && a.contact_q) {
        // within 0.2 % of r_cut^2 in a cubic box: the cutoff decided and 1 - r / r_cut
        // formed from the exact integer difference r_cut^2 - r^2, the rest in FP32
        const long long q = fx_rsq_rounded(fi, a.flo[i], fj, a.flo[j]);
        const long long dqi = __ldg(a.contact_q + tp) - q;
        if (dqi <= 0) return;
        const float qf = __ll2float_rn(q), df = __ll2float_rn(dqi);
        const float r2 = fmaf(qf, a.s2h, qf * a.s2l), dq = fmaf(df, a.s2h, df * a.s2l);
        const float rcinv = rec[0], rc = rec[1], A = rec[2];
        const float rinv = rsqrtf(r2);
        const float x = dq * rcinv / (rc + r2 * rinv);  // 1 - r / r_cut = (r_cut^2 - r^2) / (r_cut (r_cut + r))
        const float dot = dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z);
        const float fc = A * x * rinv;
        const float wR = dpd_weight_engine_f(x, rec[4]) * rinv;
        const Philox4 ph = philox4x32_10(0u, min(tgi, tgj), max(tgi, tgj), 0u, k0, k1);
        const float alpha = -1.0f + 2.0f * open01f(ph.v[0]);
        const float fdr = fc - rec[3] * wR * wR * dot + rec[5] * wR * alpha;
        const float e = A * rc * x - 0.5f * A * rcinv * dq;
        acc.add_split(dx, dy, dz, fdr, fc, e, vir);
        return;
    }
    if (rs >= rc2 * 0.998f) {
        float ddx, ddy, ddz, fdr, fc, e;
        if (dpd_near_cutoff_fp64(a, fi, fj, i, j, tp, s_rc2[tp], vi, vj, tgi, tgj, k0, k1, ddx, ddy, ddz, fdr, fc, e))
            acc.add_split(ddx, ddy, ddz, fdr, fc, e, vir);
        return;
    }
    const float rcinv = rec[0], A = rec[2];
    const float rinv = rsqrtf(rs);
    const float r = rs * rinv;
    const float dot = dx * (vi.x - vj.x) + dy * (vi.y - vj.y) + dz * (vi.z - vj.z);
    const float fc = A * (rinv - rcinv);
    const float wR = dpd_weight_engine_f(fmaxf(1.0f - r * rcinv, 0.0f), rec[4]) * rinv;
    const Philox4 ph = philox4x32_10(0u, min(tgi, tgj), max(tgi, tgj), 0u, k0, k1);
    const float alpha = -1.0f + 2.0f * open01f(ph.v[0]);
    const float fdr = fc - rec[3] * wR * wR * dot + rec[5] * wR * alpha;
    const float e = A * (rec[1] - r) - 0.5f * A * rcinv * (rc2 - rs);
    acc.add_split(dx, dy, dz, fdr, fc, e, vir);
}

template<class BE, bool ONE = false>
AZP_D void bond_term_fx(const MDArgs& a, const uint4& fi, const uint4& fj, uint32_t btype, const float* s_bond,
                        AccFx& acc, bool vir)
{
    const float dx = (float)(int32_t)(fi.x - fj.x) * a.sfix[0];
    const float dy = (float)(int32_t)(fi.y - fj.y) * a.sfix[1];
    const float dz = (float)(int32_t)(fi.z - fj.z) * a.sfix[2];
    const float rsq = fx_rsq(a, fi, fj, dx, dy, dz);
    float fdr, en;
    if (!BE::eval_f(s_bond + (ONE ? 0u : btype) * BOND_F, rsq, fdr, en)) {
        atomicOr(&a.flags[1], AZP_EBIT_BOND);
        return;
    }
    acc.add(dx, dy, dz, fdr, en, vir);
}

// image-unwrapped displacement of one axis from the 64-bit fixed positions
// (hi, lo words) and the image difference: the wrapping 64-bit difference is
// the minimum image; w = +-1 where the exact difference overflowed it; the
// result is (minimum image) + (img_i - img_j + w) L, in FP32
AZP_D float unwrapped_fx(uint32_t hi_i, uint32_t lo_i, uint32_t hi_j, uint32_t lo_j, int dimg, float sfix)
{
    const long long qi = fx_join(hi_i, lo_i), qj = fx_join(hi_j, lo_j);
    const long long dq = (long long)((unsigned long long)qi - (unsigned long long)qj);
    const int w = (qi >= 0 && qj < 0 && dq < 0) ? 1 : ((qi < 0 && qj >= 0 && dq >= 0) ? -1 : 0);
    const float dmin =
        ((float)(int)(dq >> 32) + (float)(unsigned)((unsigned long long)dq & 0xffffffffull) * 2.3283064365386963e-10f) *
        sfix;
    // sfix = L 2^-32 rounded to float, so sfix 2^32 is L rounded to float
    return dmin + (float)(dimg + w) * (sfix * 4294967296.0f);
}

// one ImageHarmonic bond of particle i (fixed words fi / li, images g[3] of the
// step's start) with partner j in the FP32-force step
template<class BE, bool ONE, bool NC>
AZP_D void bond_term_fx_image(const MDArgs& a, const uint4& fi, const uint4& li, const int* g, uint32_t j,
                              uint32_t btype, const float* s_bond, AccFx& acc, bool vir)
{
    const uint4 fj = ld_ro<NC>(a.fix + j);
    const uint4 lj = ld_ro<NC>(a.flo + j);
    const int* gj = a.img0 + 3 * (size_t)j;
    const float dx = unwrapped_fx(fi.x, li.x, fj.x, lj.x, g[0] - ld_ro<NC>(gj), a.sfix[0]);
    const float dy = unwrapped_fx(fi.y, li.y, fj.y, lj.y, g[1] - ld_ro<NC>(gj + 1), a.sfix[1]);
    const float dz = unwrapped_fx(fi.z, li.z, fj.z, lj.z, g[2] - ld_ro<NC>(gj + 2), a.sfix[2]);
    const float rsq = dx * dx + dy * dy + dz * dz;
    float fdr, en;
    if (!BE::eval_f(s_bond + (ONE ? 0u : btype) * BOND_F, rsq, fdr, en)) {
        atomicOr(&a.flags[1], AZP_EBIT_BOND);
        return;
    }
    acc.add(dx, dy, dz, fdr, en, vir);
}


// DPD: queued partners per lane, and the margin of the scan's r_cut^2: above the
// 4e-6 at which pair_term_dpd_fx itself stops, by the difference of the two FP32
// forms of r^2 (each within 1e-6)
constexpr uint32_t DPD_QUEUE_FX = 16;
constexpr float DPD_SCREEN = 1.00001f;

// neighbours gathered per batch: the list indices of a batch are loaded first,
// then their positions, so each thread keeps this many gathers in flight
#ifndef AZP_FX_BATCH
#define AZP_FX_BATCH 4
#endif
constexpr int FX_BATCH = AZP_FX_BATCH;
// Resident blocks per SM the FP32-force step is compiled for (the register cap):
// with the FP32-component r^2, 5 (48 registers) for the plain single-type step of
// the light evaluators, whose few spilled bytes cost less than the extra resident
// warps gain (measured on the melt at N = 1M: 0.0946 -> 0.0897 ms); 4 (64
// registers) for the rest, which would spill hundreds of bytes at 48 (Colloid,
// DPD, energy-writing launches), and for every step with the integer r^2.
// AZP_FX_MIN_BLOCKS overrides both.
template<class PE> struct fx_light : std::false_type {};
template<> struct fx_light<PerturbedLJ> : std::true_type {};
template<> struct fx_light<ExpandedYukawa> : std::true_type {};
template<> struct fx_light<Hertz> : std::true_type {};
template<> struct fx_light<NoPair> : std::true_type {};
template<class PE, bool OUT, bool ONE>
constexpr int fx_min_blocks()
{
#ifdef AZP_FX_MIN_BLOCKS
    return AZP_FX_MIN_BLOCKS;
#else
    // with the integer r^2 (more registers live) 4 blocks measured faster
    return (ONE && !OUT && fx_light<PE>::value && FX_BLOCK == 256 && !AZP_FX_IRSQ) ? 5 : 4;
#endif
}

// neighbour list entries of the next batch loaded while the current batch is
// evaluated (1), or at the top of each batch (0)
#ifndef AZP_FX_PIPE
#define AZP_FX_PIPE 0
#endif

// prefetch of the DRAM rows a warp's particles read (0 off, 1 into L1, 2 into L2)
#ifndef AZP_FX_PREFETCH
#define AZP_FX_PREFETCH 1
#endif
// neighbour batches walked to the warp's longest row with masked lanes instead of
// per-lane loop exits and early returns
#ifndef AZP_FX_UNIFORM
#define AZP_FX_UNIFORM 1
#endif

// the per-particle rows of step two / step one (velocity record, low position
// words, build shadow, tag) copied into shared memory by cp.async at the start of
// the step, so that their DRAM latency passes while the neighbour loop runs (1),
// or loaded where they are used (0)
#ifndef AZP_FX_STAGE
#define AZP_FX_STAGE 1
#endif

// per-thread asynchronous global -> shared copies (completed by cp_async_wait_all
// in the issuing thread, which alone reads what it copied)
AZP_D void cp_async16(void* smem, const void* g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}
AZP_D void cp_async4(void* smem, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g)
                 : "memory");
}
AZP_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
AZP_D void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

AZP_D void prefetch_line(const void* p)
{
#if AZP_FX_PREFETCH == 1
    asm volatile("prefetch.L1 [%0];" ::"l"(p));
#elif AZP_FX_PREFETCH == 2
    asm volatile("prefetch.L2 [%0];" ::"l"(p));
#else
    (void)p;
#endif
}

// Prefetch, by one instruction per lane, the lines of the warp's particles
// [i0, i_last] that the step reads from DRAM (velocities, low position words,
// build shadow, tags, bond counts, the first two bond-table columns) and the
// first nmax columns of their list rows, so that those latencies overlap at
// the start instead of chaining behind the neighbour loop. Addresses stay
// inside the arrays: every one is clamped to the warp's last particle.
AZP_D void prefetch_warp_rows(const MDArgs& a, uint32_t i0, uint32_t i_last, uint32_t nmax, bool bonds, bool rows)
{
    const uint32_t lane = threadIdx.x & 31u;
    if (lane < nmax) {
        prefetch_line(a.nbrs + (size_t)lane * a.N + i0);
        prefetch_line(a.nbrs + (size_t)lane * a.N + i_last);
    }
    const void* p = nullptr;
    if (!rows && lane < 18u) {
        // the integration rows are staged in shared memory instead
    } else if (lane < 8u) {
        p = a.velf + min(i0 + lane * 4u, i_last);
    } else if (lane < 12u) {
        p = a.flo + min(i0 + (lane - 8u) * 8u, i_last);
    } else if (lane < 16u) {
        p = a.fix_build + min(i0 + (lane - 12u) * 8u, i_last);
    } else if (lane < 18u) {
        p = a.tag + (lane == 16u ? i0 : i_last);
    } else if (bonds && lane < 20u) {
        p = a.bt_n + (lane == 18u ? i0 : i_last);
    } else if (bonds && lane < 26u) {
        const uint32_t c = (lane - 20u) / 3u, part = (lane - 20u) % 3u;
        p = a.bt + (size_t)c * a.N + min(i0 + part * 16u, i_last);
    }
    if (p) prefetch_line(p);
}

// ONE: single-type system, records from the kernel arguments (no shared-memory
// tables, no block barrier before the work)
// TILE (single-type systems, TILE_P particles per block, one thread each): the
// block's neighbour ranges are staged in shared memory first and the list
// entries address them there (celllist.cuh, TILE_GLOBAL entries are gathered)
// The body for the block-th FX_BLOCK / tpp particles at timestep ts; whether the calling
// thread's particle asks for a list rebuild (NC as in md_step_body)
template<class PE, class BE, int INTEG, bool OUT, bool ONE, bool TILE, bool NC>
AZP_D bool md_step_fx_body(const MDArgs& a, uint32_t block, unsigned long long ts, unsigned char* smem_raw)
{
    const uint32_t nt2 = a.ntypes * a.ntypes;
    double* s_rc2 = reinterpret_cast<double*>(smem_raw);
    float* s_rec = reinterpret_cast<float*>(s_rc2 + nt2);
    float* s_bond = s_rec + nt2 * PAIR_TBL;
    float* s_gamma = s_bond + a.nbondtypes * BOND_F;
    float* s_noise = s_gamma + a.ntypes;
    const uint4* s_tile = reinterpret_cast<const uint4*>(smem_raw);
    const uint32_t* trec = nullptr;
    // single-type systems: the records copied from the kernel arguments into
    // registers (every lookup below has a compile-time index; no address of the
    // kernel argument is taken, so it is not copied to local memory)
    float one_rec[ONE ? PAIR_TBL : 1], one_bond[ONE ? BOND_F : 1], one_gamma = 0.0f, one_noise = 0.0f;
    double one_rc2 = 0.0;
    if constexpr (ONE) {
#pragma unroll
        for (int k = 0; k < PAIR_TBL; ++k) one_rec[k] = a.rec0[k];
#pragma unroll
        for (int k = 0; k < BOND_F; ++k) one_bond[k] = a.bond0[k];
        one_rc2 = a.rc2_0;
        one_gamma = a.gamma0;
        one_noise = a.noise0;
        s_rc2 = &one_rc2;
        s_rec = one_rec;
        s_bond = one_bond;
        s_gamma = &one_gamma;
        s_noise = &one_noise;
        if constexpr (TILE) {
            // stage the block's neighbour ranges: coalesced 16-byte copies
            trec = a.tile + (size_t)block * TILE_REC;
            const uint32_t nr = ld_ro<NC>(trec);
            uint4* st = reinterpret_cast<uint4*>(smem_raw);
            for (uint32_t k = 0; k < nr; ++k) {
                const uint32_t b = ld_ro<NC>(trec + 2 + 3 * k), e = ld_ro<NC>(trec + 3 + 3 * k), off = ld_ro<NC>(trec + 4 + 3 * k);
                for (uint32_t q = threadIdx.x; q < e - b; q += blockDim.x) st[off + q] = ld_ro<NC>(a.fix + b + q);
            }
            __syncthreads();
        }
    } else {
        if (!std::is_same<PE, NoPair>::value)
            for (uint32_t t = threadIdx.x; t < nt2 * PAIR_TBL; t += blockDim.x) {
                s_rec[t] = (float)a.pair_table[t];
                if (t % PAIR_TBL == PAIR_REC) s_rc2[t / PAIR_TBL] = a.pair_table[t];
            }
        if (!std::is_same<BE, NoBond>::value)
            for (uint32_t t = threadIdx.x; t < a.nbondtypes; t += blockDim.x)
                BE::prepare_f(a.bond_params + (size_t)t * AZP_BOND_PARAM_DOUBLES, s_bond + (size_t)t * BOND_F);
        if (INTEG != MD_FORCES_ONLY && !a.use_lambda)
            for (uint32_t t = threadIdx.x; t < a.ntypes; t += blockDim.x) {
                s_gamma[t] = (float)a.gamma[t];
                s_noise[t] = (float)a.noise[t];
            }
        __syncthreads();
    }

    const uint32_t tpp = (uint32_t)a.tpp;
    const uint32_t gid = block * blockDim.x + threadIdx.x;
    const uint32_t i = gid >> a.tpp_shift;
    const uint32_t sub = gid & (tpp - 1u);
    const bool active = i < a.N;
    constexpr bool vir = OUT;
#if AZP_FX_STAGE
    constexpr bool STAGE = INTEG != MD_FORCES_ONLY;
    constexpr bool STAGE_V = INTEG == MD_INTEG_LANGEVIN;
#else
    constexpr bool STAGE = false, STAGE_V = false;
#endif
    __shared__ __align__(32) VelFF st_vel[STAGE_V ? FX_BLOCK : 1];
    __shared__ __align__(16) uint4 st_lo[STAGE ? FX_BLOCK : 1];
    __shared__ __align__(16) uint4 st_fb[STAGE ? FX_BLOCK : 1];
    __shared__ uint32_t st_tag[STAGE ? FX_BLOCK : 1];
    __shared__ uint32_t s_queue[std::is_same<PE, DpdEngine>::value ? DPD_QUEUE_FX * FX_BLOCK : 1];
    if constexpr (STAGE) {
        if (active && sub == 0) {
            if constexpr (STAGE_V) {
                cp_async16(&st_vel[threadIdx.x].h, &a.velf[i].h);
                cp_async16(&st_vel[threadIdx.x].l, &a.velf[i].l);
            }
            cp_async16(&st_lo[threadIdx.x], a.flo + i);
            cp_async16(&st_fb[threadIdx.x], a.fix_build + i);
            if constexpr (NC) cp_async4(&st_tag[threadIdx.x], a.tag + i);
            else st_tag[threadIdx.x] = a.tag[i];  // (a 4-byte cp.async goes through L1 lines of earlier steps)
            cp_async_commit();
        }
    }
    AccFx acc;
    uint4 fi = make_uint4(0u, 0u, 0u, 0u);
    uint32_t n = 0u;
    if constexpr (!std::is_same<PE, NoPair>::value) n = active ? min(ld_ro<NC>(a.counts + i), a.max_nn) : 0u;
    // the warp's longest list row
    const uint32_t nmax = __reduce_max_sync(0xffffffffu, n);
#if AZP_FX_PREFETCH
    {
        const uint32_t i0 = (block * blockDim.x + (threadIdx.x & ~31u)) >> a.tpp_shift;
        if (i0 < a.N) {
            const uint32_t i_last = min(i0 + (32u >> a.tpp_shift) - 1u, a.N - 1u);
            prefetch_warp_rows(a, i0, i_last, std::is_same<PE, NoPair>::value ? 0u : nmax,
                               !std::is_same<BE, NoBond>::value, !AZP_FX_STAGE || INTEG == MD_FORCES_ONLY);
        }
    }
#endif
    if (active) fi = ld_ro<NC>(a.fix + i);
    // -------------------------------------------------------------------- DPD pairs
    if constexpr (std::is_same<PE, DpdEngine>::value) {
        // Two phases, as the FP64 step: the scan queues the partners inside
        // r_cut, the warp then evaluates its queues together (a Philox draw
        // and the weight a pair cost far more than the scan). Bit 31 marks
        // the first partner of a batch, so that the batch sums are the ones
        // of a walk that evaluates as it goes.
        uint32_t* queue = s_queue + threadIdx.x;
        const uint32_t* col = a.nbrs + i;
        uint32_t k0 = 0, k1 = 0, tgi = 0;
        float4 vi = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        dpd_key(a, ts + (INTEG == MD_INTEG_LANGEVIN ? 1ull : 0ull), k0, k1);
        if (active) {
            vi = ld_ro<NC>(reinterpret_cast<const float4*>(a.dvel) + i);
            tgi = __float_as_uint(vi.w);
        }
        uint32_t nq = 0;
        for (uint32_t kb = 0; kb < nmax; kb += FX_BATCH * tpp) {
            uint32_t jj[FX_BATCH];
            uint4 fj[FX_BATCH];
            const uint32_t k = kb + sub * FX_BATCH;
#pragma unroll
            for (int u = 0; u < FX_BATCH; ++u) jj[u] = k + u < n ? ld_ro<NC>(col + (size_t)(k + u) * a.N) : 0u;
#pragma unroll
            for (int u = 0; u < FX_BATCH; ++u) fj[u] = ld_ro<NC>(a.fix + jj[u]);
            uint32_t mark = 0x80000000u;
#pragma unroll
            for (int u = 0; u < FX_BATCH; ++u) {
                const float dx = (float)(int32_t)(fi.x - fj[u].x) * a.sfix[0];
                const float dy = (float)(int32_t)(fi.y - fj[u].y) * a.sfix[1];
                const float dz = (float)(int32_t)(fi.z - fj[u].z) * a.sfix[2];
                const float rc2 = s_rec[(size_t)(ONE ? 0u : fi.w * a.ntypes + fj[u].w) * PAIR_TBL + PAIR_REC];
                if (k + u < n && rc2 > 0.0f && dx * dx + dy * dy + dz * dz < rc2 * DPD_SCREEN) {
                    queue[FX_BLOCK * nq++] = jj[u] | mark;
                    mark = 0u;
                }
            }
            if (kb + FX_BATCH * tpp < nmax && !__any_sync(0xffffffffu, nq > DPD_QUEUE_FX - FX_BATCH)) continue;
            for (uint32_t m = 0; m < nq; ++m) {
                const uint32_t e = queue[FX_BLOCK * m];
                if (e & 0x80000000u) acc.commit(vir);
                const uint32_t j = e & 0x7fffffffu;
                pair_term_dpd_fx<ONE, NC>(a, fi, ld_ro<NC>(a.fix + j), i, j, s_rec, s_rc2, acc, vir, vi, tgi, k0, k1);
            }
            nq = 0;
        }
        acc.commit(vir);
    }
    if (active) {
        // ---------------------------------------------------------------- pair
        if constexpr (!std::is_same<PE, NoPair>::value && !std::is_same<PE, DpdEngine>::value) {
            const uint32_t* col = a.nbrs + i;
#if AZP_FX_UNIFORM
            // every lane walks to the warp's longest row; slots past a lane's own
            // row are masked (no per-lane loop exit)
            const uint32_t kend = nmax;
#else
            const uint32_t kend = n;
#endif
#if AZP_FX_PIPE
            // the list entries of the first batch; each later batch's entries are
            // loaded while the current batch is evaluated
            uint32_t jn[FX_BATCH];
#pragma unroll
            for (int u = 0; u < FX_BATCH; ++u) {
                const uint32_t k = sub * FX_BATCH + u;
                jn[u] = k < n ? ld_ro<NC>(col + (size_t)k * a.N) : (TILE ? (TILE_GLOBAL | i) : i);
            }
#endif
            // a lane's batch is FX_BATCH consecutive entries, so that the batch sums do not
            // depend on the threads per particle (the total does in its last bits: each
            // lane compensates its own batches, and reduce() joins the lanes)
            for (uint32_t kb = sub * FX_BATCH; kb < kend; kb += FX_BATCH * tpp) {
                uint32_t jj[FX_BATCH];
                uint4 fj[FX_BATCH];
#if AZP_FX_PIPE
#pragma unroll
                for (int u = 0; u < FX_BATCH; ++u) jj[u] = jn[u];
#else
#pragma unroll
                for (int u = 0; u < FX_BATCH; ++u) {
                    const uint32_t k = kb + u;
                    jj[u] = k < n ? ld_ro<NC>(col + (size_t)k * a.N) : (TILE ? (TILE_GLOBAL | i) : i);
                }
#endif
                if constexpr (TILE) {
#pragma unroll
                    for (int u = 0; u < FX_BATCH; ++u)
                        fj[u] = (jj[u] & TILE_GLOBAL) ? ld_ro<NC>(a.fix + (jj[u] & ~TILE_GLOBAL)) : s_tile[jj[u]];
                } else {
#pragma unroll
                    for (int u = 0; u < FX_BATCH; ++u) fj[u] = ld_ro<NC>(a.fix + jj[u]);
                }
#if AZP_FX_PIPE
#pragma unroll
                for (int u = 0; u < FX_BATCH; ++u) {
                    const uint32_t k = kb + FX_BATCH * tpp + u;
                    jn[u] = k < n ? ld_ro<NC>(col + (size_t)k * a.N) : (TILE ? (TILE_GLOBAL | i) : i);
                }
#endif
#pragma unroll
                for (int u = 0; u < FX_BATCH; ++u) {
                    {
#if AZP_FX_UNIFORM
                        pair_term_fx_masked<PE, TILE, ONE, NC>(a, fi, fj[u], i, jj[u], kb + u < n, s_rec, s_rc2,
                                                           acc, vir, trec);
#else
                        if (kb + u < n) pair_term_fx<PE, ONE, NC>(a, fi, fj[u], i, jj[u], s_rec, s_rc2, acc, vir);
#endif
                    }
                }
                acc.commit(vir);
            }
        }
        // ---------------------------------------------------------------- bonds
        if constexpr (bond_uses_image<BE>::value) {
            const uint32_t nb = ld_ro<NC>(a.bt_n + i);
            const uint4 li = ld_ro<NC>(a.flo + i);
            const int g[3] = {ld_ro<NC>(a.img0 + 3 * (size_t)i), ld_ro<NC>(a.img0 + 3 * (size_t)i + 1),
                              ld_ro<NC>(a.img0 + 3 * (size_t)i + 2)};
            for (uint32_t k = sub; k < nb; k += tpp) {
                const uint2 e = ld_ro<NC>(a.bt + (size_t)k * a.N + i);
                bond_term_fx_image<BE, ONE, NC>(a, fi, li, g, e.x, e.y, s_bond, acc, vir);
                acc.commit(vir);
            }
        } else if constexpr (!std::is_same<BE, NoBond>::value) {
            const uint32_t nb = ld_ro<NC>(a.bt_n + i);
            for (uint32_t k0 = 2u * sub; k0 < nb; k0 += 2u * tpp) {
                const uint32_t k1 = k0 + 1u;
                const uint2 e0 = ld_ro<NC>(a.bt + (size_t)k0 * a.N + i);
                const uint2 e1 = k1 < nb ? ld_ro<NC>(a.bt + (size_t)k1 * a.N + i) : make_uint2(i, 0u);
                const uint4 f0 = ld_ro<NC>(a.fix + e0.x);
                const uint4 f1 = ld_ro<NC>(a.fix + e1.x);
                bond_term_fx<BE, ONE>(a, fi, f0, e0.y, s_bond, acc, vir);
                if (k1 < nb) bond_term_fx<BE, ONE>(a, fi, f1, e1.y, s_bond, acc, vir);
                acc.commit(vir);
            }
        }
    }
    if (tpp > 1) acc.reduce((int)tpp, vir);

    bool want_rebuild = false;
    if (active && sub == 0) {
        float fb[3] = {0.0f, 0.0f, 0.0f}, ub = 0.0f;
        if (a.bar_geom >= 0)
            // the barrier's force joins the net force (src/HarmonicBarrier.h:149-180)
            barrier_fx(a, fi, ts + (INTEG == MD_INTEG_LANGEVIN ? 1ull : 0ull), fb, ub);
        // the walls' force and energy (k_walls_fx, launched right before the step)
        const float4 fw = a.wall_kind >= 0 ? a.wall_f[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if constexpr (OUT) {
            a.out_force[i] = make_double4_32a(acc.Fx() + fb[0] + fw.x, acc.Fy() + fb[1] + fw.y,
                                              acc.Fz() + fb[2] + fw.z, acc.U() + ub + fw.w);
            double wv[6];
            for (int c = 0; c < 6; ++c) wv[c] = (double)acc.w[c];
            if (a.wall_kind >= 0) {
                // the wall virial F_a x_b (FP32 position: 2^-24 relative)
                const float x = (float)(int32_t)fi.x * a.sfix[0], y = (float)(int32_t)fi.y * a.sfix[1],
                            z = (float)(int32_t)fi.z * a.sfix[2];
                wv[0] += fw.x * x;
                wv[1] += fw.x * y;
                wv[2] += fw.x * z;
                wv[3] += fw.y * y;
                wv[4] += fw.y * z;
                wv[5] += fw.z * z;
            }
            for (int c = 0; c < 6; ++c) a.out_virial[(size_t)c * a.N + i] = wv[c];
        }
        if constexpr (INTEG != MD_FORCES_ONLY) {
            if constexpr (STAGE) cp_async_wait_all();
            const uint32_t ti = fi.w;
            const uint32_t tg = STAGE ? st_tag[threadIdx.x] : ld_ro<NC>(a.tag + i);
            const float fx = acc.fx.s + (acc.fx.c + (fb[0] + fw.x));
            const float fy = acc.fy.s + (acc.fy.c + (fb[1] + fw.y));
            const float fz = acc.fz.s + (acc.fz.c + (fb[2] + fw.z));
            const uint32_t tix = ONE ? 0u : ti;
            const float gam = a.use_lambda ? a.lambdaf * (float)a.diameter[i] : s_gamma[tix];
            // the method's temperature at this timestep (a table when it varies)
            float kTv = a.kTf, nz = a.use_lambda ? 0.0f : s_noise[tix];
            if (a.kT_hdr) {
                const size_t r = kT_row(a, ts);
                kTv = (float)a.kT_tab[r];
                nz = (float)a.noise_tab[r * a.ntypes + ti];
            }
            const float c = a.noiseless ? 0.0f : (a.use_lambda ? sqrtf(6.0f * gam * kTv / a.dtf) : nz);
            const bool mover = in_group(a, ti);
            float ux, uy, uz;
            flow_at_ff(a.flowf, (float)(int32_t)fi.y * a.sfix[1], ux, uy, uz);
            const float dt = a.dtf;
            float r0, r1, r2, ddx = 0.0f, ddy = 0.0f, ddz = 0.0f;
            bool moved = false;
            if constexpr (INTEG == MD_INTEG_LANGEVIN) {
                uniform3f(AZP_RNG_LANGEVIN_FLOW, ts, a.seed, tg, -c, 2.0f * c, r0, r1, r2);
                VelFF v = STAGE_V ? st_vel[threadIdx.x] : a.velf[i];
                const float minv = mover ? v.h.w : 0.0f;  // a particle outside the group keeps its velocity
                const float ax = (fx + (r0 - gam * (v.h.x - ux))) * minv;
                const float ay = (fy + (r1 - gam * (v.h.y - uy))) * minv;
                const float az = (fz + (r2 - gam * (v.h.z - uz))) * minv;
                if (a.next) {
                    // v(t + dt/2) = v(t - dt/2) + dt a: the half kick of step two and of
                    // step one; then x += v(t + dt/2) dt
                    const float kx = dt * ax, ky = dt * ay, kz = dt * az;
                    const float mdt = mover ? dt : 0.0f;
                    ddx = (v.h.x + kx) * mdt;
                    ddy = (v.h.y + ky) * mdt;
                    ddz = (v.h.z + kz) * mdt;
                    ff_add(v.h.x, v.l.x, kx);
                    ff_add(v.h.y, v.l.y, ky);
                    ff_add(v.h.z, v.l.z, kz);
                    moved = true;
                } else {
                    const float h = 0.5f * dt;
                    ff_add(v.h.x, v.l.x, h * ax);
                    ff_add(v.h.y, v.l.y, h * ay);
                    ff_add(v.h.z, v.l.z, h * az);
                    a.accel[3 * i] = ax;
                    a.accel[3 * i + 1] = ay;
                    a.accel[3 * i + 2] = az;
                }
                a.velf[i] = v;
            } else {
                uniform3f(AZP_RNG_BROWNIAN_FLOW, ts, a.seed, tg, -c, 2.0f * c, r0, r1, r2);
                const float gi = 1.0f / gam;
                const float mdt = mover ? dt : 0.0f;
                ddx = (ux + (fx + r0) * gi) * mdt;
                ddy = (uy + (fy + r1) * gi) * mdt;
                ddz = (uz + (fz + r2) * gi) * mdt;
                if (a.max_dispf > 0.0f) {
                    const float m = a.max_dispf;
                    ddx = fminf(fmaxf(ddx, -m), m);
                    ddy = fminf(fmaxf(ddy, -m), m);
                    ddz = fminf(fmaxf(ddz, -m), m);
                }
                moved = true;
            }
            if (moved) {
                uint4 lo = STAGE ? st_lo[threadIdx.x] : a.flo[i];
                bool bad = false;
                const int wx = fx_advance(fi.x, lo.x, ddx, a.s64h[0], a.s64l[0], bad);
                const int wy = fx_advance(fi.y, lo.y, ddy, a.s64h[1], a.s64l[1], bad);
                const int wz = fx_advance(fi.z, lo.z, ddz, a.s64h[2], a.s64l[2], bad);
                if (wx | wy | wz) {
                    a.image[3 * i] += wx;
                    a.image[3 * i + 1] += wy;
                    a.image[3 * i + 2] += wz;
                }
                a.fix_next[i] = fi;
                a.flo_next[i] = lo;
                want_rebuild = displaced(fi, STAGE ? st_fb[threadIdx.x] : a.fix_build[i], a.sfix, a.disp_thresh2);
                if (bad) atomicOr(&a.flags[1], AZP_EBIT_NONFINITE);
            }
        }
    }
    return want_rebuild;
}

template<class PE, class BE, int INTEG, bool OUT, bool ONE, bool TILE = false>
__global__ void __launch_bounds__(FX_BLOCK, (fx_min_blocks<PE, OUT, ONE>())) k_md_step_fx(const __grid_constant__ MDArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const bool want = md_step_fx_body<PE, BE, INTEG, OUT, ONE, TILE, true>(a, blockIdx.x, *a.d_timestep, smem_raw);
    if constexpr (INTEG != MD_FORCES_ONLY) finish_step(a, want);
}

// dynamic shared memory of k_md_step_fx (without tiles)
inline size_t md_step_fx_smem(const MDArgs& a)
{
    const size_t nt2 = (size_t)a.ntypes * a.ntypes;
    return nt2 * sizeof(double) + nt2 * PAIR_TBL * sizeof(float) + (size_t)a.nbondtypes * BOND_F * sizeof(float) +
           2 * a.ntypes * sizeof(float);
}

// ---------------------------------------------------------------- persistent run
// r.steps timesteps in one cooperative launch: each step is the body of the step kernels
// over the launch's blocks, then a grid barrier, then the rebuild when a particle asked
// for one. Launched kernel by kernel, a step of a small system waits longer for the graph's
// conditional node and launches (8 to 10 us) than it computes; here it waits for one
// barrier. The particle arrays change within the launch, so the bodies load them with
// plain loads (NC false), which the barriers' fences order.
// Bound: in a step, as the step kernels, until the step is shorter than the barrier and
// the load latencies of its chain (6.4 us at 216 particles); in a rebuild, the seven
// barriers and the chain list -> cell -> particles of each phase. Microseconds per step with
// the rebuilds, graph and this kernel: FP32 LJ fluid 28.5 and 18.6 at 1,000 particles,
// 30.5 and 21.6 at 4,096, 72.0 and 63.7 at 54,872; FP32 melt 31.3 and 16.9 at 10,000;
// FP64 fluid 52.8 and 42.3 at 4,096. Three FP32 blocks per SM: with two, steps past 304
// blocks go in two turns; with four, 64 registers spill and the 54,872 take 75.2.
// The request of step s goes to word s mod 3, so that a block that is already in the next
// step cannot change what a slower one still reads; the word after next is cleared.
template<class PE, class BE, int INTEG, bool FX, bool ONE>
__global__ void __launch_bounds__(RUN_BLOCK, FX ? 3 : 2) k_md_run(const __grid_constant__ RunArgs r)
{
    static_assert(FX_BLOCK == RUN_BLOCK && MD_BLOCK == RUN_BLOCK, "one block size");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_word;
    const uint32_t tid = blockIdx.x * RUN_BLOCK + threadIdx.x, nth = gridDim.x * RUN_BLOCK;
    uint32_t* flags = r.step[0].flags;
    const unsigned long long ts0 = *r.step[0].d_timestep;
    uint32_t gen = load_relaxed(r.sync + 1);
    bool wanted = *(volatile uint32_t*)(flags) != 0u, failed = *(volatile uint32_t*)(flags + 1) != 0u;
    if (*(volatile uint32_t*)(flags + 1) & AZP_EBIT_TIMEOUT) return;  // the barrier's words are unsound
    for (uint32_t c = tid; c < r.rebuild[0].list.g.ncell; c += nth) r.rebuild[0].cell_count[c] = 0u;
    if (tid < 6u) r.request[tid] = 0u;
    if (!grid_barrier(r, gen, &s_word)) return;
    int par = r.cur;
    for (uint32_t s = 0; s < r.steps; ++s) {
        if (wanted && !failed && !rebuild_cooperative<FX>(r, par, gen, smem_raw, &s_word)) return;
        const MDArgs& a = r.step[par];
        bool want = false;
        // blocks beyond the launch's own are taken as they become free
        uint32_t* next = r.request + 3u + s % 3u;
        for (uint32_t b = blockIdx.x; b < r.blocks;) {
            if constexpr (FX)
                want |= md_step_fx_body<PE, BE, INTEG, false, ONE, false, false>(a, b, ts0 + s, smem_raw);
            else
                want |= md_step_body<PE, BE, INTEG, false, false>(a, b, ts0 + s, smem_raw);
            if (r.blocks <= gridDim.x) break;
            if (threadIdx.x == 0u) s_word = atomicAdd(next, 1u);
            __syncthreads();
            b = gridDim.x + s_word;
            __syncthreads();  // s_word, and the body's shared memory
        }
        uint32_t* word = r.request + s % 3u;
        if (__any_sync(0xffffffffu, want) && (threadIdx.x & 31u) == 0u) atomicOr(word, 1u);
        // (every warp of the block has raised its errors: a step that fails is followed by no
        // rebuild, as where the steps are launches)
        __syncthreads();
        if (threadIdx.x == 0u && *(volatile uint32_t*)(flags + 1) != 0u) atomicOr(word, 2u);
        if (!grid_barrier(r, gen, &s_word)) return;
        const uint32_t got = *(volatile uint32_t*)word;
        if (tid == 0u) {
            r.request[(s + 2u) % 3u] = 0u;
            r.request[3u + (s + 2u) % 3u] = 0u;
        }
        wanted = (got & 1u) != 0u;
        failed = failed || (got & 2u) != 0u;
        par ^= 1;
    }
    // a rebuild asked for by the last step, for the launch that follows
    if (wanted && !failed && !rebuild_cooperative<FX>(r, par, gen, smem_raw, &s_word)) return;
    if (tid == 0u) {
        if (wanted && failed) flags[0] = 1u;
        *r.step[0].d_timestep_rw = ts0 + r.steps;
    }
}

template<class PE, class BE, int INTEG, bool FX, bool ONE>
int launch_run_k(const RunArgs& r, cudaStream_t s)
{
    auto k = k_md_run<PE, BE, INTEG, FX, ONE>;
    const size_t step = FX ? md_step_fx_smem(r.step[0]) : md_step_smem<PE>(r.step[0]);
    const size_t smem = std::max(step, rebuild_smem(r.step[0].ntypes));
    int dev = 0, sms = 0, per_sm = 0;
    AZP_CUDA_TRY(cudaGetDevice(&dev));
    AZP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    AZP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    AZP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)RUN_BLOCK, smem));
    const uint32_t most = (uint32_t)(per_sm * sms);
    // The line against the step-by-step run (the launch is refused before anything is
    // enqueued). FP32: a step must fit the resident blocks at once, for in this kernel the
    // body has 80 registers and the rebuild's phases share the residency: graph and this
    // kernel 113.9 and 111.7 us per step at 432 blocks (fluid 110,592), but 54.5 and 63.4
    // at 500 (colloid 8,000), 42.9 and 46.6 at 513 (melt 131,300), 173 and 271 at 4,097.
    // Colloid mixtures below the line: 38.9 and 32.2 at 63 blocks (1,000 particles), 45.7 and
    // 38.7 at 313, 48.1 and 39.5 at 456.
    // FP64, whose longer steps refill the SMs block by block: a thread per particle must
    // fit, for the rebuild; 73.9 and 61.9 (melt 40,000), 580 and 573 (colloid 65,537),
    // but 122.6 and 122.1 at 131,300 and 319 and 348 at 400,000.
    if (most == 0 || (FX ? r.blocks > most : r.step[0].N > most * RUN_BLOCK)) return AZP_ERR_UNSUPPORTED;
    // at least a few blocks, for the rebuild
    const uint32_t grid = std::min(std::max(r.blocks, 16u), most);
    RunArgs args = r;
    void* params[] = {&args};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k, dim3(grid), dim3(RUN_BLOCK), params, smem, s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        // a stream with part of the device's SMs (a green context): step by step there
        cudaGetLastError();
        return AZP_ERR_TOO_LARGE;
    }
    AZP_CUDA_TRY(e);
    return AZP_OK;
}

template<class PE, class BE>
int launch_run_be(int precision, int integ, const RunArgs& r, cudaStream_t s)
{
    // the forms that need a kernel of their own before each step (DPD and ImageHarmonic
    // snapshots, FP32 walls) run step by step
    if constexpr (!std::is_same<PE, DpdEngine>::value && !bond_uses_image<BE>::value) {
        const bool one = r.step[0].one_type != 0;
        if (integ == MD_INTEG_LANGEVIN) {
            if (precision == AZP_FP64) return launch_run_k<PE, BE, MD_INTEG_LANGEVIN, false, false>(r, s);
            return one ? launch_run_k<PE, BE, MD_INTEG_LANGEVIN, true, true>(r, s)
                       : launch_run_k<PE, BE, MD_INTEG_LANGEVIN, true, false>(r, s);
        }
        if (integ == MD_INTEG_BROWNIAN) {
            if (precision == AZP_FP64) return launch_run_k<PE, BE, MD_INTEG_BROWNIAN, false, false>(r, s);
            return one ? launch_run_k<PE, BE, MD_INTEG_BROWNIAN, true, true>(r, s)
                       : launch_run_k<PE, BE, MD_INTEG_BROWNIAN, true, false>(r, s);
        }
    }
    return AZP_ERR_UNSUPPORTED;
}

template<class PE>
int launch_run_pe(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s)
{
    switch (bond_kind) {
    case -1: return launch_run_be<PE, NoBond>(precision, integ, r, s);
    case AZP_BOND_QUARTIC: return launch_run_be<PE, QuarticBond>(precision, integ, r, s);
    case AZP_BOND_DOUBLE_WELL: return launch_run_be<PE, DoubleWellBond>(precision, integ, r, s);
    default: return AZP_ERR_UNSUPPORTED;
    }
}

template<class PE, class BE, typename R, int INTEG>
int launch_md_t(const MDArgs& a, cudaStream_t s)
{
    const size_t threads = (size_t)a.N * a.tpp;
    const int bs = std::is_same<R, float>::value ? FX_BLOCK : MD_BLOCK;
    const uint32_t blocks = (uint32_t)((threads + bs - 1) / bs);
    if (blocks == 0) return AZP_OK;
    if constexpr (std::is_same<R, float>::value) {
        const size_t smem = md_step_fx_smem(a);
        constexpr bool can_tile = !std::is_same<PE, NoPair>::value && !std::is_same<PE, DpdEngine>::value &&
                                  !bond_uses_image<BE>::value;
        auto k = a.out ? (a.one_type ? k_md_step_fx<PE, BE, INTEG, true, true> : k_md_step_fx<PE, BE, INTEG, true, false>)
                       : (a.one_type ? k_md_step_fx<PE, BE, INTEG, false, true>
                                     : k_md_step_fx<PE, BE, INTEG, false, false>);
        size_t smem_k = smem;
        if (a.tile && (FX_BLOCK != (int)TILE_P || a.tpp != 1 || !a.one_type || !can_tile))
            return record_error(AZP_ERR_UNSUPPORTED, "k_md_step_fx: tiles need one type, 256-thread blocks, tpp 1");
        if constexpr (can_tile) {
            if (a.tile) {
                k = a.out ? k_md_step_fx<PE, BE, INTEG, true, true, true> : k_md_step_fx<PE, BE, INTEG, false, true, true>;
                smem_k = (size_t)TILE_CAP * sizeof(uint4);
            }
        }
        if (smem_k > 8 * 1024)  // beside up to 33 KB of static shared memory
            AZP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_k));
        k<<<blocks, FX_BLOCK, smem_k, s>>>(a);
        AZP_CHECK_LAUNCH("k_md_step_fx");
    } else {
        const size_t smem = md_step_smem<PE>(a);
        // a Brownian step writes no forces, a forces-only launch nothing else
        auto k = k_md_step<PE, BE, INTEG, INTEG == MD_FORCES_ONLY>;
        if constexpr (INTEG == MD_INTEG_LANGEVIN) {
            if (a.out) k = k_md_step<PE, BE, INTEG, true>;
        } else if ((a.out != 0) != (INTEG == MD_FORCES_ONLY)) {
            return record_error(AZP_ERR_UNSUPPORTED, "k_md_step: output mode not built");
        }
        if (smem > 48 * 1024) AZP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<blocks, MD_BLOCK, smem, s>>>(a);
        AZP_CHECK_LAUNCH("k_md_step");
    }
    return AZP_OK;
}

template<class PE, class BE, typename R>
int launch_md_integ(int integ, const MDArgs& a, cudaStream_t s)
{
    switch (integ) {
    case MD_INTEG_LANGEVIN: return launch_md_t<PE, BE, R, MD_INTEG_LANGEVIN>(a, s);
    case MD_INTEG_BROWNIAN: return launch_md_t<PE, BE, R, MD_INTEG_BROWNIAN>(a, s);
    case MD_FORCES_ONLY: return launch_md_t<PE, BE, R, MD_FORCES_ONLY>(a, s);
    default: return AZP_ERR_INVALID;
    }
}

template<class PE>
int launch_md_pe(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s)
{
    if (precision == AZP_FP32) {
        switch (bond_kind) {
        case -1: return launch_md_integ<PE, NoBond, float>(integ, a, s);
        case AZP_BOND_QUARTIC: return launch_md_integ<PE, QuarticBond, float>(integ, a, s);
        case AZP_BOND_DOUBLE_WELL: return launch_md_integ<PE, DoubleWellBond, float>(integ, a, s);
        case AZP_BOND_IMAGE_HARMONIC: return launch_md_integ<PE, HarmonicBond, float>(integ, a, s);
        default: return AZP_ERR_INVALID;
        }
    }
    switch (bond_kind) {
    case -1: return launch_md_integ<PE, NoBond, double>(integ, a, s);
    case AZP_BOND_QUARTIC: return launch_md_integ<PE, QuarticBond, double>(integ, a, s);
    case AZP_BOND_DOUBLE_WELL: return launch_md_integ<PE, DoubleWellBond, double>(integ, a, s);
    case AZP_BOND_IMAGE_HARMONIC: return launch_md_integ<PE, HarmonicBond, double>(integ, a, s);
    default: return AZP_ERR_INVALID;
    }
}

// per-evaluator entry points, one per translation unit
int launch_md_nopair(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
int launch_md_plj(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
int launch_md_eyuk(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
int launch_md_hertz(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
int launch_md_colloid(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
int launch_md_dpd(int bond_kind, int precision, int integ, const MDArgs& a, cudaStream_t s);
// the persistent run of the same (DPD: none)
int launch_run_nopair(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s);
int launch_run_plj(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s);
int launch_run_eyuk(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s);
int launch_run_hertz(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s);
int launch_run_colloid(int bond_kind, int precision, int integ, const RunArgs& r, cudaStream_t s);

}  // namespace azp
