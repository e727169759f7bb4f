// Reverse-mode adjoint of the cloth substep (no reference counterpart: the
// reference calibrates with external finite-difference sensitivities,
// docs/CLOTH_SPECIMEN_CALIBRATION.md:52-82).
//
// The forward records a tape: the positions at the start of every substep
// and after every phase barrier, the velocities at the start of every
// substep, and the grips of every substep.  This kernel walks the taped substeps and each substep's phases in
// reverse and applies the vector-Jacobian product of every projection.  Branch decisions are
// recomputed in FP32 from the tape exactly as the forward made them; the
// derivatives are evaluated in FP64 at the FP32 state, and adjoints and
// parameter gradients are accumulated in FP64.
//
// Differentiated: predict with gravity and damping, the swept ground clamp,
// XPBD distance / shear / knot / bend projections (one iteration, so lambda
// starts at zero), the bend's ground active set, step fraction and ground
// clamp, compliant grips, the ground clamp, unilateral strain limits,
// finalize with cloth/ground Coulomb friction (sticking and sliding).  Each
// is piecewise smooth: the pieces the forward took are recomputed in FP32
// and differentiated exactly.  Fruit/yarn contact and its friction move
// the cloth through the fruits' rigid-body state, which the adjoint does not
// carry; where they change the cloth the event is counted in `nonsmooth` and
// passed through as the identity.
#pragma once

#include "cloth_kernels.cuh"

enum AdjointPhase : uint32_t {
    ADJ_KNOT = 10,
    ADJ_BEGIN = 0,
    ADJ_DIST = 1,
    ADJ_BEND = 2,
    ADJ_GRIP = 3,
    ADJ_YARN = 4,
    ADJ_GROUND = 5,
    ADJ_STRAIN = 6,
    ADJ_FINAL = 7,
    ADJ_TAIL = 9,
};

// Gradients: d loss / d log-scale of each compliance group (the distinct
// compliance values of each constraint family, numbered by the host), then
// d loss / d damping.
#define ADJ_MAX_GROUPS 16u

struct AdjointArgs {
    const DeviceCloth* cloth;        // device copy of the handle's descriptor
    const NumiClothConfig* cfg;      // the segment's Configs
    const float4* tape;              // [substeps][slots][n]
    const float4* tape_v;            // [substeps][n]
    const NumiClothGrip* tape_grip;  // [substeps][grips], where the grip is active
    const uint4* phases;             // [slots - 1] (type, first record, records, 0) per barrier
    uint32_t slots;
    uint32_t shift;                  // log2 of the particles each CTA of the cluster owns
    uint32_t substeps;               // substeps of the segment
    uint32_t first_substep;          // rollout index of the segment's first substep
    uint32_t interval;               // substeps whose gradients are summed before they join the totals
    float damping;                   // the schedule's (or the cloth's) damping
    uint32_t frictions;              // the schedule's frictions switch
    const uint32_t* tracked;         // [n_tracked]
    uint32_t n_tracked;
    const double* targets;           // [losses][n_tracked][3]
    uint32_t loss_every;             // loss after substeps s with (s + 1) % loss_every == 0
    double4* gx;                     // [n] adjoint of positions (xyz; w unused)
    double4* gv;                     // [n] adjoint of velocities
    double4* gprev;                  // [n] scratch: adjoint of the substep's start positions via finalize
    const uint8_t* d_group;          // [distances] compliance group
    const uint8_t* k_group;          // [knots]
    const uint8_t* b_group;          // [bends]
    const uint8_t* g_group;          // [grips]
    uint32_t groups;
    double* grads;                   // [groups + 1] accumulated (groups, then damping)
    double* grip_grads;              // [rollout substeps][6] or null
    double* loss;                    // [1] accumulated
    unsigned int* nonsmooth;         // [1] count of non-smooth events met
};

namespace adj {

struct D3v {
    double x, y, z;
};
__device__ __forceinline__ D3v d3(const double4& a) { return D3v{a.x, a.y, a.z}; }
__device__ __forceinline__ D3v d3f(const V3& a) { return D3v{a.x, a.y, a.z}; }
__device__ __forceinline__ D3v d4f(const float4& a) { return D3v{a.x, a.y, a.z}; }
__device__ __forceinline__ double dotd(D3v a, D3v b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3v addd(D3v a, D3v b) { return D3v{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3v subd(D3v a, D3v b) { return D3v{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3v muld(D3v a, double s) { return D3v{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ D3v crossd(D3v a, D3v b) {
    return D3v{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ void put(double4* g, uint32_t i, D3v v) { g[i] = make_double4(v.x, v.y, v.z, 0.0); }

// Adjoint of the positions during a segment.  kShared: CTA r of the cloth's
// cluster holds particles [r << shift, (r + 1) << shift) in its shared
// memory (three doubles each: an odd stride, so neighbouring particles fall
// in different banks), the others' through distributed shared memory.
// Otherwise (clouds too large for that) the global array, past L1.
template <bool kShared>
struct AdjointX {
    double* own;
    double4* all;
    uint32_t rank, shift;

    __device__ __forceinline__ double* at(uint32_t i) const {
        const uint32_t r = i >> shift;
        double* p = own + 3u * (i & ((1u << shift) - 1u));
        return r == rank ? p : static_cast<double*>(__cluster_map_shared_rank(p, r));
    }
    __device__ __forceinline__ D3v get(uint32_t i) const {
        if constexpr (kShared) {
            const double* p = at(i);
            return D3v{p[0], p[1], p[2]};
        } else {
            const double2* p = reinterpret_cast<const double2*>(all + i);
            const double2 xy = __ldcg(p);
            return D3v{xy.x, xy.y, __ldcg(&p[1].x)};
        }
    }
    __device__ __forceinline__ void put(uint32_t i, D3v v) const {
        if constexpr (kShared) {
            double* p = at(i);
            p[0] = v.x;
            p[1] = v.y;
            p[2] = v.z;
        } else {
            all[i] = make_double4(v.x, v.y, v.z, 0.0);
        }
    }
};

// VJP of x_a' = x_a - w_a dl n, x_b' = x_b + w_b dl n with
// dl = -(L - rest) / (w_a + w_b + alpha) (lambda from zero), n = (x_b - x_a)/L,
// at the FP32 state a, b (derivatives in FP64).  Returns d loss / d alpha.
template <class X>
__device__ __forceinline__ double distance_vjp(const X& gx, uint32_t ia, uint32_t ib, const float4& a, const float4& b,
                                               double rest, double alpha) {
    const D3v dd = subd(d4f(b), d4f(a));
    const double L = sqrt(dotd(dd, dd));
    const D3v n = muld(dd, 1.0 / L);
    const double den = (static_cast<double>(a.w) + b.w) + alpha;
    const double dl = -(L - rest) / den;
    const D3v ga = gx.get(ia), gb = gx.get(ib);
    const D3v u = subd(muld(gb, b.w), muld(ga, a.w));
    const double un = dotd(u, n);
    const D3v gd = addd(muld(n, -un / den), muld(subd(u, muld(n, un)), dl / L));
    gx.put(ia, subd(ga, gd));
    gx.put(ib, addd(gb, gd));
    return -un * dl / den;
}

// VJP of the knot projection (nc::solve_knot with lambda from zero) at the
// positions p with inverse masses p.w: g[4], the adjoints of the moved
// positions, become those of p.  Returns d loss / d alpha.  Reverse mode by
// hand: one pass over the projection's steps (two square roots, five
// quotients), against thirteen of them for a tangent per input.
__device__ __forceinline__ double knot_vjp(const float4 p[4], double alpha, double rest, D3v g[4]) {
    const double w0 = p[0].w, w1 = p[1].w, w2 = p[2].w, w3 = p[3].w;
    const D3v e = subd(d4f(p[1]), d4f(p[0])), f = subd(d4f(p[3]), d4f(p[2]));
    const double el = 1.0 / sqrt(dotd(e, e)), fl = 1.0 / sqrt(dotd(f, f));
    const D3v u = muld(e, el), v = muld(f, fl);
    double c = dotd(u, v);
    const bool clamped = c > 1.0 || c < -1.0;
    c = c > 1.0 ? 1.0 : c < -1.0 ? -1.0 : c;
    // gradients of the cosine, the step along them
    const D3v gw = muld(subd(v, muld(u, c)), el), gf = muld(subd(u, muld(v, c)), fl);
    const double we = w0 + w1, wf = w2 + w3;
    const double iden = 1.0 / (alpha + we * dotd(gw, gw) + wf * dotd(gf, gf));
    const double dl = -(c - rest) * iden;
    // reverse: p1 + gw w1 dl, p0 - gw w0 dl, p3 + gf w3 dl, p2 - gf w2 dl
    const D3v A = subd(muld(g[1], w1), muld(g[0], w0)), B = subd(muld(g[3], w3), muld(g[2], w2));
    const double bdl = dotd(A, gw) + dotd(B, gf);
    const double bden = -bdl * dl * iden;
    const D3v bgw = addd(muld(A, dl), muld(gw, 2.0 * we * bden));
    const D3v bgf = addd(muld(B, dl), muld(gf, 2.0 * wf * bden));
    const D3v q = muld(bgw, el), r = muld(bgf, fl);
    double bc = -bdl * iden - dotd(q, u) - dotd(r, v);
    if (clamped) bc = 0.0;
    const D3v bu = addd(subd(r, muld(q, c)), muld(v, bc));
    const D3v bv = addd(subd(q, muld(r, c)), muld(u, bc));
    // u = e / |e| and the 1 / |e| of gw: along e, then across it
    const D3v be = muld(subd(bu, muld(u, dotd(bu, u) + dotd(bgw, gw))), el);
    const D3v bf = muld(subd(bv, muld(v, dotd(bv, v) + dotd(bgf, gf))), fl);
    g[0] = subd(g[0], be);
    g[1] = addd(g[1], be);
    g[2] = subd(g[2], bf);
    g[3] = addd(g[3], bf);
    return bden;
}

// Forward-mode dual number (value, one tangent) for the bend projection on
// the ground, whose branches a hand-written reverse pass would repeat.
struct Dual {
    double v, d;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual{a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual{a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return Dual{a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    return Dual{a.v / b.v, (a.d * b.v - a.v * b.d) / (b.v * b.v)};
}
__device__ __forceinline__ Dual dsqrt(Dual a) {
    const double r = sqrt(a.v);
    return Dual{r, a.d / (2.0 * r)};
}
struct DV {
    Dual x, y, z;
};
__device__ __forceinline__ DV operator-(DV a, DV b) { return DV{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ DV operator*(DV a, Dual s) { return DV{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ Dual ddot(DV a, DV b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }

// Branches the forward bend projection took (nc::bend_core): active[s]
// when the ground holds particle s's normal motion; frac_src the particle
// whose ground distance limits the step (-1: none, fraction 1), frac_zero
// when that distance is zero; clamp[s] when the new position is lifted back
// to the ground.
struct BendBranches {
    bool active[2];
    int frac_src;
    bool frac_zero;
    bool clamp[2];
};

// The forward's FP32 decisions for one bend with lambda from zero; false
// when the forward leaves the pair unchanged.
__device__ __forceinline__ bool bend_branches(const float4& p0, const float4& p2, const float2& m, float dt2,
                                              float radius, bool ground, BendBranches& b) {
    const float4 p[2] = {p0, p2};
    const V3 diff = xyz(p2) - xyz(p0);
    const float chord = len3(diff);
    if (chord < 1.0e-12f) return false;
    const float value = chord - m.x;
    const V3 dir = vdiv(diff, chord);
    const V3 g[2] = {dir * -1.0f, dir};
    const float alpha = m.y / dt2;
    float free_den = alpha;
    free_den = free_den + p[0].w * lsq(g[0]);
    free_den = free_den + p[1].w * lsq(g[1]);
    if (free_den < 1.0e-16f) return false;
    const float lam = 0.0f;
    const float numerator = -value - alpha * lam;
    const float free_dl = numerator / free_den;
    float den = alpha;
    for (int s = 0; s < 2; ++s) {
        b.active[s] = ground && p[s].z <= radius + 1.0e-9f && g[s].z * free_dl < 0.0f;
        den = den + p[s].w * (lsq(g[s]) - (b.active[s] ? g[s].z * g[s].z : 0.0f));
    }
    if (den < 1.0e-16f) return false;
    const float dl = numerator / den;
    float fraction = 1.0f;
    b.frac_src = -1;
    b.frac_zero = false;
    if (ground) {
        for (int s = 0; s < 2; ++s) {
            if (b.active[s]) continue;
            const float vc = g[s].z * p[s].w * dl;
            if (vc >= 0.0f) continue;
            const float cand = fmaxf(0.0f, p[s].z - radius) / -vc;
            if (cand < fraction) {
                fraction = cand;
                b.frac_src = s;
                b.frac_zero = !(p[s].z - radius > 0.0f);
            }
        }
    }
    const float applied = dl * fraction;
    for (int s = 0; s < 2; ++s) {
        V3 corr = g[s] * (p[s].w * applied);
        if (b.active[s]) corr.z = 0.0f;
        const V3 np = xyz(p[s]) + corr;
        b.clamp[s] = ground && np.z < radius;
    }
    return true;
}

// The bend projection on dual numbers along the forward's branches:
// positions p[2] (the pair's ends), inverse masses w[2], compliance alpha
// (over dt^2); writes out[2].
__device__ __forceinline__ void bend_dual(const DV p[2], const double w[2], Dual alpha, double rest, double radius,
                                          const BendBranches& b, DV out[2]) {
    const Dual zero{0.0, 0.0};
    const Dual one{1.0, 0.0};
    const DV diff = p[1] - p[0];
    const Dual chord = dsqrt(ddot(diff, diff));
    const Dual value = chord - Dual{rest, 0.0};
    const DV dir = diff * (one / chord);
    const DV g[2] = {DV{zero, zero, zero} - dir, dir};
    const Dual numerator = zero - value;
    Dual den = alpha;
    for (int s = 0; s < 2; ++s)
        den = den + Dual{w[s], 0.0} * (ddot(g[s], g[s]) - (b.active[s] ? g[s].z * g[s].z : zero));
    const Dual dl = numerator / den;
    Dual fraction = one;
    if (b.frac_src >= 0) {
        const int s = b.frac_src;
        if (b.frac_zero) {
            fraction = zero;
        } else {
            const Dual vc = g[s].z * Dual{w[s], 0.0} * dl;
            fraction = (p[s].z - Dual{radius, 0.0}) / (zero - vc);
        }
    }
    const Dual applied = dl * fraction;
    for (int s = 0; s < 2; ++s) {
        const Dual k = Dual{w[s], 0.0} * applied;
        DV np{p[s].x + g[s].x * k, p[s].y + g[s].y * k, p[s].z + (b.active[s] ? zero : g[s].z * k)};
        if (b.clamp[s]) np.z = Dual{radius, 0.0};
        out[s] = np;
    }
}

}  // namespace adj

// One item of a constraint colour: the record's points at the positions the
// phase started from, its material and compliance group.
struct AdjointItem {
    uint32_t k;
    uint32_t idx[4];
    float4 p[4];
    float4 m;
    uint32_t group;
};

#define ADJ_THREADS 512u
#define ADJ_PHASES 256u   /* phase records kept in shared memory */
#define ADJ_CLUSTER_MAX 16u

// The reverse sweep of one cloth's taped segment on its cluster of CTAs.
//
// A substep is some twenty dependent phases of at most a few thousand items,
// so the sweep is bound by the latency of a phase: barrier, gather, a chain
// of FP64 quotients and roots.  On one CTA of 256 threads with the adjoint in
// global memory a phase of the 64 x 64 cloth's 2,000 items took eight rounds
// of dependent L2 loads (22.9 ms for 96 substeps).  Here a cluster gives every
// item its own thread, the adjoint lives in the cluster's shared memory, and a
// thread loads its next item (indices, material, taped positions: nothing the
// sweep writes) before the barrier in front of it.  Phases that touch only a
// particle's own adjoint (finalize, ground, contact counts, predict) run on
// its owner, one after the other without barriers.
template <bool kShared>
__device__ __forceinline__ void adjoint_segment(const AdjointArgs& A, uint32_t rank, uint32_t ranks, double* smem) {
    using namespace adj;
    const DeviceCloth& d = *A.cloth;
    const uint32_t n = d.n;
    const uint32_t bottom = A.slots - 1u;   // phases of a substep
    __shared__ uint4 s_phase[ADJ_PHASES];
    for (uint32_t b = threadIdx.x; b < min(bottom, ADJ_PHASES); b += blockDim.x) s_phase[b] = A.phases[b];
    auto phase = [&](uint32_t b) { return b < ADJ_PHASES ? s_phase[b] : A.phases[b]; };
    auto sync = [&]() {
        if (ranks > 1u)
            cooperative_groups::this_cluster().sync();
        else
            __syncthreads();
    };
    const AdjointX<kShared> gx{smem, A.gx, rank, A.shift};
    const uint32_t own = min(rank << A.shift, n), own_end = min(own + (1u << A.shift), n);
    if constexpr (kShared)
        for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x) {
            const double4 v = A.gx[i];
            gx.put(i, D3v{v.x, v.y, v.z});
        }
    double acc[ADJ_MAX_GROUPS + 1u];
    for (uint32_t e = 0; e <= ADJ_MAX_GROUPS; ++e) acc[e] = 0.0;
    const uint32_t damp_slot = A.groups;
    double loss = 0.0;
    unsigned int rough = 0u;
    __shared__ double s_grip[NC_MAX_GRIPS][6];

    // item r of a colour phase, at the positions `pre` the phase started from
    auto load = [&](const uint4& ph, uint32_t r, const float4* pre, AdjointItem& it) {
        const uint32_t k = ph.y + r;
        it.k = k;
        if (ph.x == ADJ_KNOT) {
            const uint4 q = __ldg(d.k_ij + k);
            const float2 m = __ldg(d.k_mat + k);
            it.m = make_float4(m.x, m.y, 0.0f, 0.0f);
            it.idx[0] = q.x;
            it.idx[1] = q.y;
            it.idx[2] = q.z;
            it.idx[3] = q.w;
            it.group = __ldg(A.k_group + k);
#pragma unroll
            for (int e = 0; e < 4; ++e) it.p[e] = __ldg(pre + it.idx[e]);
            return;
        }
        if (ph.x == ADJ_BEND) {
            const uint4 q = __ldg(d.b_ij + k);
            const float2 m = __ldg(d.b_mat + k);
            it.m = make_float4(m.x, m.y, 0.0f, 0.0f);
            it.idx[0] = q.x;
            it.idx[1] = q.z;
            it.group = __ldg(A.b_group + k);
        } else {
            const uint2 q = __ldg(d.d_ij + k);
            it.m = __ldg(d.d_mat + k);
            it.idx[0] = q.x;
            it.idx[1] = q.y;
            it.group = __ldg(A.d_group + k);
        }
        it.p[0] = __ldg(pre + it.idx[0]);
        it.p[1] = __ldg(pre + it.idx[1]);
    };
    // this CTA's slice of a phase's items
    auto slice = [&](uint32_t count, uint32_t& lo, uint32_t& hi) {
        lo = static_cast<uint32_t>(static_cast<unsigned long long>(count) * rank / ranks);
        hi = static_cast<uint32_t>(static_cast<unsigned long long>(count) * (rank + 1u) / ranks);
    };
    // this thread's first item of the next colour phase below (si, b)
    AdjointItem next{};
    auto fetch = [&](uint32_t si, uint32_t b) {
        for (;;) {
            if (b == 0u) {
                if (si == 0u) return;
                --si;
                b = bottom;
            }
            --b;
            const uint4 ph = phase(b);
            if (ph.x != ADJ_DIST && ph.x != ADJ_STRAIN && ph.x != ADJ_BEND && ph.x != ADJ_KNOT) continue;
            uint32_t lo, hi;
            slice(ph.z, lo, hi);
            if (lo + threadIdx.x < hi)
                load(ph, lo + threadIdx.x, A.tape + (static_cast<size_t>(si) * A.slots + b) * n, next);
            return;
        }
    };
    // the sweep of one colour phase's items: each loaded before the one in
    // front of it is computed
    auto colour = [&](const uint4& ph, const float4* pre, auto&& apply) {
        uint32_t lo, hi;
        slice(ph.z, lo, hi);
        for (uint32_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
            const AdjointItem it = next;
            if (r + blockDim.x < hi) load(ph, r + blockDim.x, pre, next);
            apply(it);
        }
    };
    // The sums since the last flush, in a fixed order: lanes, warps, then the
    // cluster's CTAs.  Called at the same substeps of the rollout however its
    // segments are taped, so that one call's bits depend on its arguments
    // alone.  The first CTA adds a flush's parts to the totals at the next
    // one (a cluster has colour phases between, whose barriers order them), so
    // a flush costs none of the cluster's barriers.
    __shared__ double s_red[ADJ_MAX_GROUPS + 2u][ADJ_THREADS / 32u];
    __shared__ double s_part[2][ADJ_CLUSTER_MAX][ADJ_MAX_GROUPS + 2u];
    __shared__ double s_total[ADJ_MAX_GROUPS + 2u];
    if (threadIdx.x <= A.groups + 1u)   // later segments' sums
        s_total[threadIdx.x] = threadIdx.x <= A.groups ? A.grads[threadIdx.x] : *A.loss;
    uint32_t flushes = 0u;
    auto add_parts = [&]() {
        if (rank != 0u || flushes == 0u || threadIdx.x > A.groups + 1u) return;
        double sum = 0.0;
        for (uint32_t r = 0; r < ranks; ++r) sum += s_part[(flushes - 1u) & 1u][r][threadIdx.x];
        s_total[threadIdx.x] += sum;
    };
    auto flush = [&]() {
        __syncthreads();   // s_red is read (a cloth may have no colour phase)
        add_parts();
        for (uint32_t e = 0; e <= A.groups + 1u; ++e) {
            double v = e <= A.groups ? acc[e] : loss;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (threadIdx.x % 32u == 0u) s_red[e][threadIdx.x / 32u] = v;
            if (e <= A.groups) acc[e] = 0.0;
        }
        loss = 0.0;
        __syncthreads();
        if (threadIdx.x <= A.groups + 1u) {
            double sum = 0.0;
            for (uint32_t w = 0; w < blockDim.x / 32u; ++w) sum += s_red[threadIdx.x][w];
            double* part = &s_part[flushes & 1u][rank][threadIdx.x];
            if (ranks > 1u) part = static_cast<double*>(__cluster_map_shared_rank(part, 0u));
            *part = sum;
        }
        ++flushes;
    };
    sync();
    fetch(A.substeps, 0u);
    bool loose = false;   // own-particle phases ran since the last barrier
    for (uint32_t si = A.substeps; si-- > 0u;) {
        const NumiClothConfig& cf = A.cfg[si];
        const float dt = cf.gravityAndTimestep.w;
        const float dt2 = dt * dt;
        const double dtd = dt;
        const float radius = cf.clothMaterial.x;
        const bool ground = cf.constraintCounts.z != 0u;
        const float4* T = A.tape + static_cast<size_t>(si) * A.slots * n;
        const uint32_t step = A.first_substep + si;
        // loss seed at the end of the substep, by the tracked particles' owners
        if (A.loss_every != 0u && (step + 1u) % A.loss_every == 0u) {
            const uint32_t li = (step + 1u) / A.loss_every - 1u;
            const float4* xe = T + static_cast<size_t>(bottom) * n;
            for (uint32_t t = 0; t < A.n_tracked; ++t) {
                const uint32_t i = __ldg(A.tracked + t);
                if (i < own || i >= own_end || (i - own) % blockDim.x != threadIdx.x) continue;
                const double* tg = A.targets + (static_cast<size_t>(li) * A.n_tracked + t) * 3u;
                const D3v diff{static_cast<double>(xe[i].x) - tg[0], static_cast<double>(xe[i].y) - tg[1],
                               static_cast<double>(xe[i].z) - tg[2]};
                loss += dotd(diff, diff);
                gx.put(i, addd(gx.get(i), muld(diff, 2.0)));
            }
            loose = true;
        }
        for (uint32_t b = bottom; b-- > 0u;) {
            const uint4 ph = phase(b);
            const float4* pre = T + static_cast<size_t>(b) * n;     // positions before the phase
            const float4* post = pre + n;                            // after its barrier
            bool crossed = true;   // the phase touches particles of other threads
            if (loose && (ph.x == ADJ_STRAIN || ph.x == ADJ_DIST || ph.x == ADJ_BEND || ph.x == ADJ_KNOT ||
                          ph.x == ADJ_GRIP)) {
                sync();
                loose = false;
            }
            switch (ph.x) {
            case ADJ_YARN:
                // fruit/yarn contact moved the cloth: not differentiated
                crossed = false;
                for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x)
                    if (pre[i].x != post[i].x || pre[i].y != post[i].y || pre[i].z != post[i].z) ++rough;
                break;
            case ADJ_FINAL: {
                // v_end = (x - x_start) / dt, then the cloth/ground Coulomb
                // friction of a grounded particle (nc::finalize_particle):
                // with normal impulse gi = (v_end.z - v_pred.z) / w, sticking
                // (|v_t| / w <= mu gi) zeroes the tangential velocity and
                // sliding removes mu (v_end.z - v_pred.z) along the slip.
                // The adjoint of the predicted normal velocity goes to
                // gprev.w for the predict step.
                crossed = false;
                const float4* xs = T;
                const float4* vs = A.tape_v + static_cast<size_t>(si) * n;
                const float inv_dt = 1.0f / dt;
                const float mu = cf.clothMaterial.z;
                for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x) {
                    if (pre[i].w == 0.0f) {
                        gx.put(i, D3v{0.0, 0.0, 0.0});
                        A.gv[i] = make_double4(0, 0, 0, 0);
                        A.gprev[i] = make_double4(0, 0, 0, 0);
                        continue;
                    }
                    D3v gvv = d3(A.gv[i]);
                    double gvpz = 0.0;
                    if (ground && A.frictions != 0u && pre[i].z <= radius + 1.0e-6f) {
                        // the forward's decisions, in FP32
                        const float w = pre[i].w;
                        const V3 vel = (xyz(pre[i]) - xyz(xs[i])) * inv_dt;
                        float vpz = vs[i].z + cf.gravityAndTimestep.z * dt;
                        if (A.damping != 0.0f) vpz = vpz * (1.0f / (1.0f + A.damping * dt));
                        const float gi = fmaxf(0.0f, (vel.z - vpz) / w);
                        const V3 tv{vel.x, vel.y, 0.0f};
                        const float slip = len3(tv);
                        if (gi > 0.0f && !(slip < 1.0e-10f) && fminf(slip / w, mu * gi) > 0.0f) {
                            if (slip / w <= mu * gi) {
                                gvv.x = 0.0;   // sticking
                                gvv.y = 0.0;
                            } else {
                                // sliding: v_t' = v_t - phi v_t / |v_t|, phi = mu (v.z - v_pred.z)
                                const D3v vd = muld(subd(d4f(pre[i]), d4f(xs[i])), 1.0 / dtd);
                                double vpd = static_cast<double>(vs[i].z) + static_cast<double>(cf.gravityAndTimestep.z) * dtd;
                                if (A.damping != 0.0f) vpd /= 1.0 + static_cast<double>(A.damping) * dtd;
                                const double sl = sqrt(vd.x * vd.x + vd.y * vd.y);
                                const double nx = vd.x / sl, ny = vd.y / sl;
                                const double phi = static_cast<double>(mu) * (vd.z - vpd);
                                const double gn = gvv.x * nx + gvv.y * ny;
                                const double gtx = gvv.x - phi / sl * (gvv.x - nx * gn);
                                const double gty = gvv.y - phi / sl * (gvv.y - ny * gn);
                                const double gphi = -gn;
                                gvv = D3v{gtx, gty, gvv.z + static_cast<double>(mu) * gphi};
                                gvpz = -static_cast<double>(mu) * gphi;
                            }
                        }
                    }
                    gx.put(i, addd(gx.get(i), muld(gvv, 1.0 / dtd)));
                    const D3v gp = muld(gvv, -1.0 / dtd);
                    A.gprev[i] = make_double4(gp.x, gp.y, gp.z, gvpz);
                    A.gv[i] = make_double4(0, 0, 0, 0);
                }
                break;
            }
            case ADJ_STRAIN:
                colour(ph, pre, [&](const AdjointItem& it) {
                    const float4 a = it.p[0], bb = it.p[1], m = it.m;
                    if (!(m.w > 0.0f)) return;
                    const float L = len3(xyz(bb) - xyz(a));
                    const float maxL = m.x * (1.0f + m.w);
                    if (L <= maxL || L < 1.0e-12f) return;
                    if (a.w + bb.w <= 0.0f) return;
                    // x_a += dir w_a (L - maxL)/den: the distance form with rest maxL, alpha 0
                    distance_vjp(gx, it.idx[0], it.idx[1], a, bb, static_cast<double>(maxL), 0.0);
                });
                break;
            case ADJ_DIST:
                colour(ph, pre, [&](const AdjointItem& it) {
                    const float4 a = it.p[0], bb = it.p[1];
                    if (len3(xyz(bb) - xyz(a)) < 1.0e-12f) return;
                    const float alpha = it.m.y / dt2;
                    if ((a.w + bb.w) + alpha <= 0.0f) return;
                    const double alphad = static_cast<double>(it.m.y) / (dtd * dtd);
                    acc[it.group] +=
                        distance_vjp(gx, it.idx[0], it.idx[1], a, bb, static_cast<double>(it.m.x), alphad) * alphad;
                });
                break;
            case ADJ_KNOT:
                colour(ph, pre, [&](const AdjointItem& it) {
                    // the forward's own skip tests, in FP32
                    const float4* p = it.p;
                    const float wl = len3(xyz(p[1]) - xyz(p[0]));
                    const float fl = len3(xyz(p[3]) - xyz(p[2]));
                    if (wl < 1.0e-12f || fl < 1.0e-12f) return;
                    const V3 warp = vdiv(xyz(p[1]) - xyz(p[0]), wl);
                    const V3 weft = vdiv(xyz(p[3]) - xyz(p[2]), fl);
                    const float cosine = fminf(fmaxf(dot3(warp, weft), -1.0f), 1.0f);
                    const V3 gw = vdiv(weft - warp * cosine, wl);
                    const V3 gf = vdiv(warp - weft * cosine, fl);
                    float den = it.m.y / dt2;
                    den = den + p[0].w * lsq(gw * -1.0f);
                    den = den + p[1].w * lsq(gw);
                    den = den + p[2].w * lsq(gf * -1.0f);
                    den = den + p[3].w * lsq(gf);
                    if (den <= 0.0f) return;
                    const double alphad = static_cast<double>(it.m.y) / (dtd * dtd);
                    D3v g[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) g[e] = gx.get(it.idx[e]);
                    acc[it.group] += knot_vjp(p, alphad, static_cast<double>(it.m.x), g) * alphad;
#pragma unroll
                    for (int e = 0; e < 4; ++e) gx.put(it.idx[e], g[e]);
                });
                break;
            case ADJ_BEND:
                colour(ph, pre, [&](const AdjointItem& it) {
                    const float4 p0 = it.p[0], p2 = it.p[1];
                    const float2 m = make_float2(it.m.x, it.m.y);
                    BendBranches br;
                    if (!bend_branches(p0, p2, m, dt2, radius, ground, br)) return;
                    const double alphad = static_cast<double>(m.y) / (dtd * dtd);
                    if (!br.active[0] && !br.active[1] && br.frac_src < 0 && !br.clamp[0] && !br.clamp[1]) {
                        // clear of the ground: the distance form
                        acc[it.group] +=
                            distance_vjp(gx, it.idx[0], it.idx[1], p0, p2, static_cast<double>(m.x), alphad) * alphad;
                        return;
                    }
                    // on the ground: VJP by forward mode along the forward's
                    // branches, one tangent per input (6 coordinates, alpha)
                    const float4 pp[2] = {p0, p2};
                    const D3v u0 = gx.get(it.idx[0]), u1 = gx.get(it.idx[1]);
                    const double w[2] = {p0.w, p2.w};
                    double gin[7];
                    for (int dir = 0; dir < 7; ++dir) {
                        DV pd[2];
                        for (int e = 0; e < 2; ++e)
                            pd[e] = DV{Dual{pp[e].x, dir == 3 * e ? 1.0 : 0.0}, Dual{pp[e].y, dir == 3 * e + 1 ? 1.0 : 0.0},
                                       Dual{pp[e].z, dir == 3 * e + 2 ? 1.0 : 0.0}};
                        DV out[2];
                        bend_dual(pd, w, Dual{alphad, dir == 6 ? 1.0 : 0.0}, static_cast<double>(m.x),
                                  static_cast<double>(radius), br, out);
                        gin[dir] = (u0.x * out[0].x.d + u0.y * out[0].y.d + u0.z * out[0].z.d) +
                                   (u1.x * out[1].x.d + u1.y * out[1].y.d + u1.z * out[1].z.d);
                    }
                    gx.put(it.idx[0], D3v{gin[0], gin[1], gin[2]});
                    gx.put(it.idx[1], D3v{gin[3], gin[4], gin[5]});
                    acc[it.group] += gin[6] * alphad;
                });
                break;
            case ADJ_GRIP: {
                // the first CTA, one thread per grip
                if (!(cf.gripTargetAndActive.w > 0.0f) || d.g_count == 0u) {
                    crossed = false;
                    break;
                }
                if (rank != 0u) break;
                const uint32_t g = threadIdx.x;
                double gg[6] = {0, 0, 0, 0, 0, 0};
                if (g < d.g_count) {
                    const NumiClothGrip grip = A.tape_grip[static_cast<size_t>(si) * d.g_count + g];
                    if (grip.particle.y == cf.gripControl.x) {
                        const uint32_t i = grip.particle.x;
                        const float4 p = pre[i];
                        const float alpha = grip.targetOffsetAndCompliance.w / dt2;
                        if (p.w + alpha > 0.0f) {
                            const float4 qr = make_float4(cf.gripOrientation.x, cf.gripOrientation.y,
                                                          cf.gripOrientation.z, cf.gripOrientation.w);
                            const V3 ro = rotate_q(qr, V3{grip.targetOffsetAndCompliance.x,
                                                          grip.targetOffsetAndCompliance.y,
                                                          grip.targetOffsetAndCompliance.z});
                            const D3v target = addd(D3v{cf.gripTargetAndActive.x, cf.gripTargetAndActive.y,
                                                        cf.gripTargetAndActive.z},
                                                    d3f(ro));
                            const D3v gout = gx.get(i);
                            const double w = p.w;
                            const double al = static_cast<double>(grip.targetOffsetAndCompliance.w) / (dtd * dtd);
                            const double dn = w + al;
                            // x' = (alpha x + w T) / (w + alpha)
                            gx.put(i, muld(gout, al / dn));
                            const D3v gT = muld(gout, w / dn);
                            const D3v xm = subd(d4f(p), target);
                            acc[A.g_group[g]] += dotd(gout, muld(xm, w / (dn * dn))) * al;
                            const D3v rot = crossd(d3f(ro), gT);
                            gg[0] = gT.x;
                            gg[1] = gT.y;
                            gg[2] = gT.z;
                            gg[3] = rot.x;
                            gg[4] = rot.y;
                            gg[5] = rot.z;
                        }
                    }
                }
                if (g < NC_MAX_GRIPS)
                    for (int e = 0; e < 6; ++e) s_grip[g][e] = gg[e];
                __syncthreads();
                if (threadIdx.x == 0 && A.grip_grads != nullptr) {
                    double* out = A.grip_grads + static_cast<size_t>(step) * 6u;
                    for (uint32_t k = 0; k < min(d.g_count, NC_MAX_GRIPS); ++k)
                        for (int e = 0; e < 6; ++e) out[e] += s_grip[k][e];
                }
                break;
            }
            case ADJ_GROUND:
                crossed = false;
                if (ground)
                    for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x)
                        if (radius - pre[i].z > 0.0f) {
                            D3v v = gx.get(i);
                            v.z = 0.0;
                            gx.put(i, v);
                        }
                break;
            case ADJ_BEGIN: {
                // x' = x_s + v' dt, v' = (v_s + g dt) / (1 + c dt)
                crossed = false;
                const float4* vs = A.tape_v + static_cast<size_t>(si) * n;
                const double c = A.damping;
                const double kf = c != 0.0 ? 1.0 / (1.0 + c * dtd) : 1.0;
                const double dk = -dtd / ((1.0 + c * dtd) * (1.0 + c * dtd));
                const D3v grav{cf.gravityAndTimestep.x, cf.gravityAndTimestep.y, cf.gravityAndTimestep.z};
                for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x) {
                    if (pre[i].w == 0.0f) {
                        gx.put(i, D3v{0.0, 0.0, 0.0});
                        A.gv[i] = make_double4(0, 0, 0, 0);
                        continue;
                    }
                    D3v gpos = gx.get(i);
                    // swept ground clamp: the predicted z is set to the radius
                    if (ground && pre[i].z >= radius && post[i].z == radius) gpos.z = 0.0;
                    // v' feeds x' and, through friction, the finalize step
                    const double4 gp = A.gprev[i];
                    D3v gvp = muld(gpos, dtd);
                    gvp.z += gp.w;
                    const D3v v0 = addd(D3v{vs[i].x, vs[i].y, vs[i].z}, muld(grav, dtd));
                    acc[damp_slot] += dotd(gvp, v0) * dk;
                    put(A.gv, i, muld(gvp, kf));
                    gx.put(i, addd(gpos, d3(gp)));
                    A.gprev[i] = make_double4(0, 0, 0, 0);
                }
                break;
            }
            default:   // ADJ_TAIL
                crossed = false;
                break;
            }
            if (crossed) {
                if (ph.x != ADJ_GRIP) fetch(si, b);
                sync();
            } else if (ph.x != ADJ_TAIL) {
                loose = true;
            }
        }
        if (si == 0u || step % A.interval == 0u) flush();
    }
    if constexpr (kShared)
        for (uint32_t i = own + threadIdx.x; i < own_end; i += blockDim.x) put(A.gx, i, gx.get(i));
    if (rough) atomicAdd(A.nonsmooth, rough);
    sync();
    add_parts();
    if (rank == 0u && threadIdx.x <= A.groups + 1u) {
        if (threadIdx.x <= A.groups)
            A.grads[threadIdx.x] = s_total[threadIdx.x];
        else
            *A.loss = s_total[threadIdx.x];
    }
}

// Many cloths' segments, a cluster of CTAs each.
template <bool kShared>
__global__ void __launch_bounds__(ADJ_THREADS, 1) numi_cloth_adjoint_kernel(const AdjointArgs* args, uint32_t ranks) {
    extern __shared__ __align__(16) double nc_adjoint_smem[];
    adjoint_segment<kShared>(args[blockIdx.x / ranks], blockIdx.x % ranks, ranks, nc_adjoint_smem);
}

// Device-to-device copies of many regions in one launch, one CTA per
// region (cloth state checkpoints of a batch).
struct CopyOp {
    const void* src;
    void* dst;
    unsigned long long bytes;
};

__global__ void numi_cloth_copy_kernel(const CopyOp* ops) {
    const CopyOp op = ops[blockIdx.x];
    if ((reinterpret_cast<uintptr_t>(op.src) | reinterpret_cast<uintptr_t>(op.dst) | op.bytes) % 16u == 0u) {
        const float4* s = static_cast<const float4*>(op.src);
        float4* d = static_cast<float4*>(op.dst);
        for (unsigned long long k = threadIdx.x; k < op.bytes / 16u; k += blockDim.x) d[k] = s[k];
    } else {
        const unsigned char* s = static_cast<const unsigned char*>(op.src);
        unsigned char* d = static_cast<unsigned char*>(op.dst);
        for (unsigned long long k = threadIdx.x; k < op.bytes; k += blockDim.x) d[k] = s[k];
    }
}
