// Lennard-Jones Metropolis sweep: PairwiseCutoff<Isotropic<Shifted<LennardJones>>> (and the overlap
// penalty and the other isotropic potentials, in FP64).
//
// delta_energy_one (hoomd-interaction/src/pairwise_cutoff.rs:919-941) sums the pair energy of
// the trial site and of the current site over every other site within r_cut; the Metropolis
// test (hoomd-mc/src/parallel_sweep.rs:267-268) accepts when dH <= 0, else draws u and accepts
// when u < exp(-dH / kT). At rho = 0.8 with r_cut = 2.5 a space holds ~13 bodies, so a colour
// pass has few trials (~5k for 2^19 bodies) with ~340 candidates each, and a sweep 112 passes. All of
// them run in one launch in dataflow order (hmc_flow.cuh): a trial's latency then no longer adds
// up to a pass's, and the launches are gone.
//
// FP32 + recheck: FP32 pair energies together with a rigorous bound B on |dU32 - dU64| (r^2 error
// from the fixed-point sites, propagated through dE/dr^2; rounding of the energy formula;
// summation chains; the FP64 sum's own error). A decision that B cannot change is taken from the
// FP32 sums; otherwise the warp recomputes dU in FP64. Any FP64 sum that another order could
// decide differently is counted (order_ambiguous), so decisions equal the FP64 pass.
//
// Bound: the dependent chain of a trial (L2 latency of the staging copies, the acquire and release
// of the progress words, FP64 wraps) and issue slots; DRAM is idle (the state stays in L2).
// Measured, ten sweeps with the frame's copy: 2^19 sites FP32 29.4 -> 13.7 ms, 20,011 sites FP64
// 18.3 -> 6.9 ms, 64 replicas of 8,192 FP32 44.0 -> 21.3 ms, against one launch per colour pass
// with a warp per trial. (Trials with few candidates: lj_staging.)
#include <cuda_runtime.h>

#include <type_traits>

#include "hmc_flow.cuh"

namespace hmc {
namespace {

constexpr float kU32 = 5.9604645e-8f;  // 2^-24

// FP32 pair energy and a bound on its error against the exact energy of the FP64 sites, for
// a pair with r2 below the band's upper end (the caller skips pairs outside the cut-off).
// The r^2 error is bounded without a square root: sum |d_a| <= sqrt(3) r and
// r <= (r^2 + 1) / 2, so |r2_32 - r2| <= 3.5 E ((r^2 + 1)/2 + E) + lj_rel_err r^2 (lj_setup_for).
__device__ __forceinline__ void lj_pair32(const Pair& P, float r2, float& e, float& err) {
    if (r2 >= P.lj_rcut2_lo32) {  // the FP64 pass may or may not count this pair
        e = 0.f;
        err = P.lj_band_energy;
        return;
    }
    const float E = P.lj_disp_err;
    const float dr2 = 3.5f * E * (0.5f * (r2 + 1.f) + E) + P.lj_rel_err * r2;
    const float inv = __frcp_rn(r2);
    const float sr2 = P.lj_sigma2_32 * inv;
    const float sr6 = sr2 * sr2 * sr2;
    const float b = P.lj_four_eps32 * sr6;  // 4 eps (sigma/r)^6
    const float a = b * sr6;                // 4 eps (sigma/r)^12
    e = (a - b) - P.lj_e_shift32;
    // |dE/dr^2| <= (6a + 3b) / r^2; 1.1 covers its variation over [r2 - dr2, r2 + dr2] and the
    // FP32 evaluation of this bound; 25 u32 covers the roundings of the energy formula and of 4 eps.
    err = 1.1f * ((6.f * a + 3.f * b) * (dr2 * inv) + 25.f * kU32 * (a + b + fabsf(P.lj_e_shift32)));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ uint32_t warp_maxu(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// FP64 energy of site ta against the stencil fs, skipping slot self: the warp takes the stencil's
// candidates 32 at a time, each lane sums its own in that order, then a butterfly reduction (every
// lane ends with the same values). mag receives sum |e| (for order_ambiguous). For injected moves
// and the tuner, whose sites may lie in different spaces.
template <int DIM>
__device__ __forceinline__ void lj_energy64(const Geometry& g, const Arrays& A, const Pair& P, const double* ta,
                                            const FlatStencil& fs, uint32_t self, uint32_t lane, double& ea,
                                            double& mag) {
    double a = 0.0, am = 0.0;
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < fs.total; j0 += 32u) {
        const uint32_t j = j0 + lane;
        uint32_t part;
        const uint32_t q = flat_slot(fs, j, part);
        if (j >= fs.total || q == self) continue;
        const double4 v = ldg4(A.sorted_s + q);
        const double sv[3] = {v.x, v.y, v.z};
        const double ra = ref_dist2<DIM>(g, ta, sv);
        const double x = soft_pair64<true>(P, ra);
        a = dadd(a, x);
        am += soft_pair_mag(P, ra, x);
    }
    ea = warp_sum(a);
    mag = warp_sum(am);
}

struct Sums32 {
    float e_new, e_old, err, mag;
    uint32_t terms;
};

// FP32 energies of the trial site t32 and the current site c32 (fixed_site) against the stencil fs
// of their common space, with error bounds (hmc_eval_moves).
template <int DIM>
__device__ __forceinline__ Sums32 lj_energy32(const Geometry& g, const Arrays& A, const Pair& P, const int4& t32, const int4& c32,
                                               const FlatStencil& fs, uint32_t self, uint32_t lane) {
    Sums32 s{0.f, 0.f, 0.f, 0.f, 0u};
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < fs.total; j0 += 32u) {
        const uint32_t j = j0 + lane;
        uint32_t part;
        const uint32_t q = flat_slot(fs, j, part);
        if (j >= fs.total || q == self) continue;
        const int4 o = __ldg(reinterpret_cast<const int4*>(A.sorted_off) + q);
        const float r2[2] = {fixed_dist2<DIM>(g, t32, o), fixed_dist2<DIM>(g, c32, o)};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (!(r2[i] < P.lj_rcut2_hi32)) continue;
            float e, err;
            lj_pair32(P, r2[i], e, err);
            (i == 0 ? s.e_new : s.e_old) += e;
            s.err += err;
            s.mag += fabsf(e);
            s.terms += 1;
        }
    }
    s.e_new = warp_sumf(s.e_new);
    s.e_old = warp_sumf(s.e_old);
    s.err = warp_sumf(s.err);
    s.mag = warp_sumf(s.mag);
    s.terms = warp_maxu(s.terms);
    return s;
}

// ---- the sweep --------------------------------------------------------------------------------
// What the random streams of the trials of colour sets [L.round, L.round_end) give, one thread per
// trial (generate_trial_moves, parallel_sweep.rs:231-278): the body (IndexedRandom::choose), the
// displacement (Ball::sample) and the Metropolis uniform, from Counter(step, substep + set,
// seed).index(space). None of it depends on a site, so it is computed for all of a launch's trials
// at once with every lane busy, and k_flow_lj, which gives a trial a warp, does not repeat it in
// 32 lanes. The FP32 pass also gets -kT ln u as a pair of FP32 bounds (metropolis_bounds), which
// spares its decision two exponentials.
// Each space's progress is set to the first colour set; the ticket starts at 0.
struct DrawRecord {
    uint32_t k;      // the chosen body's slot; kNoTrial: the replica runs no such colour set
    uint32_t m;      // packed multi-index of the space
    float w_lo, w_hi;
};

// Bounds around w = -kT ln u, the energy below which u < exp(-dU / kT): dU < w_lo accepts and
// dU > w_hi rejects for certain. The exponent's slack of 1e-11 covers the rounding of dU / kT
// (|dU / kT| <= 37 where u >= 2^-53 decides), of the reference's exp and of log here (each a few
// ulp). u = 0 is left to the FP64 sums.
__device__ __forceinline__ void metropolis_bounds(double u, double kt, float& lo, float& hi) {
    const double x = -log(u);
    lo = u > 0.0 ? __double2float_rd(kt * (x - 1e-11)) : -INFINITY;
    hi = u > 0.0 ? __double2float_ru(kt * (x + 1e-11)) : INFINITY;
}

template <int DIM, bool BATCH>
__global__ void __launch_bounds__(128) k_draw_lj(Geometry g, Arrays A, Launch L, Batch B) {
    grid_dependency_wait();
    allow_dependent_launch();
    if (BATCH && L.round == kRoundFromDevice) {  // a captured sweep's rounds loop
        L.round = *B.round_dev;
        L.round_end += L.round;
    }
    const FlowRange f = flow_range(A.stats, L.round, L.round_end, 1u << DIM);
    if (blockIdx.x == 0 && threadIdx.x == 0) A.stats->ticket = L.flow.stall == kStallTrial ? 1u : 0u;
    const uint32_t stride = BATCH ? B.color_stride : g.color_stride;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += gridDim.x * blockDim.x) {
        uint32_t round, color, entry;
        flow_item(f, i, round, color, entry);
        if (!BATCH) entry = flow_rotated(A.stats->color_count[color], round, color, 1u << DIM, g.shape[0], entry);
        const size_t e = (size_t)color * stride + entry;
        const uint32_t packed = __ldg(A.color_cells + e);
        uint32_t m[3] = {0, 0, 0};
        unpack_m<DIM>(packed, m);
        const Replica* R = BATCH ? B.rep + __ldg(B.color_rep + e) : nullptr;
        const Geometry& G = BATCH ? R->g : g;
        const uint32_t cell = cell_index<DIM>(G, m), base = BATCH ? R->cell_base : 0u;
        if (round == f.r0) A.progress[base + cell] = f.r0;
        if (BATCH && round >= R->rounds) {
            A.draw_i[i] = make_uint4(kNoTrial, packed, 0u, 0u);
            continue;
        }
        const uint32_t start = __ldg(A.cell_start + base + cell);
        const uint32_t count = __ldg(A.cell_start + base + cell + 1) - start;
        Sfc64 rng = make_rng(BATCH ? R->step : L.step, (BATCH ? R->substep : L.substep) + round,
                             BATCH ? R->seed : L.seed, (uint64_t)cell);
        const uint32_t k = start + canon_range_u32(rng, count);
        double dv[3];
        ball_sample<DIM>(rng, BATCH ? R->max_move : L.max_move, A.zig_x, A.zig_f, dv);
        const double u = uniform01(rng);
        float lo, hi;
        metropolis_bounds(u, BATCH ? R->kt : L.kt, lo, hi);
        A.draw_d[i] = make_double4(dv[0], dv[1], DIM == 3 ? dv[2] : 0.0, u);
        A.draw_i[i] = make_uint4(k, packed, __float_as_uint(lo), __float_as_uint(hi));
    }
}

// The team of W warps that decides one trial shares this: the non-empty parts of the trial's
// stencil (stencil_part) as ranges of the candidate number j (slot = base + j for j < end), the
// staged sites of the candidates (FP32: fixed point), the trial, and per warp the pairs inside the
// cut-off that wait for their energies and the partial sums. Batches: the trial's replica too, since
// its fields would else come from L2 after every acquire.
struct StencilPart {
    uint32_t base, end;
};
constexpr int kStage = 384;  // candidates staged at a time (a stencil of 2^19 sites at 0.8 holds ~345)
constexpr int kDirect = 0;   // of trials with few candidates: their lanes load the sites (lj_staging)
template <bool FP32, bool BATCH, int W, int STAGE>
struct alignas(16) Team {
    // candidates between two staging steps; direct loads need none
    static constexpr bool staged = STAGE > 0;
    static constexpr uint32_t stage = staged ? STAGE : 0x80000000u;
    using Site = typename std::conditional<FP32, int4, double4>::type;
    Site site[staged ? STAGE : 1];
    union {
        float2 q32[64];
        double2 q64[64];
    } list[W];
    StencilPart part[18];
    unsigned long long bar;
    double sum64[W][3];
    float2 sum32[W];
    double t[3], s[3];  // the trial site and (FP64) the current site
    int4 t32, s32;      // the same in fixed point (FP32)
    uint32_t n_parts, total, self, valid;
    uint32_t lost;      // a thread's wait for staged sites ran out (mbar_wait)
    typename std::conditional<BATCH, Replica, uint32_t>::type rep;
};

template <int W>
__device__ __forceinline__ void team_sync() {
    if (W == 1)
        __syncwarp();
    else
        __syncthreads();  // a block is one team
}
// team_sync, and whether v holds in any thread of the team (the same answer for all).
template <int W>
__device__ __forceinline__ bool team_any(bool v) {
    return W == 1 ? __any_sync(0xffffffffu, v) != 0 : __syncthreads_or(v) != 0;
}

// The stencil around space m into the team's scratch, by one warp, with the candidate number of slot k.
template <int DIM, typename T>
__device__ __forceinline__ void team_parts(const Geometry& g, const uint32_t* __restrict__ cs, const uint32_t* m,
                                           uint32_t k, uint32_t lane, T& S) {
    const unsigned full = 0xffffffffu;
    uint32_t lo = 0, len = 0;
    float s0, s1;
    if (lane < 2u * kRows<DIM>) stencil_part<DIM>(g, cs, m, (int)(lane >> 1), (lane & 1u) != 0, lo, len, s0, s1);
    uint32_t x = len;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(full, x, o);
        if (lane >= o) x += y;
    }
    const unsigned has = __ballot_sync(full, len > 0);
    if (len > 0) {
        S.part[__popc(has & ((1u << lane) - 1u))] = {lo - (x - len), x};
        if (k - lo < len) S.self = k - lo + (x - len);
    }
    if (lane == 31) {
        S.total = x;
        S.n_parts = __popc(has);
    }
    __syncwarp();
}

// Candidates [c0, c0 + T::stage) into the team's staging buffer by one warp, one bulk copy per part:
// every copy is in flight at once, where a walk over the candidates in global memory waits for a
// load per step or two.
template <bool FP32, typename T>
__device__ __forceinline__ void team_stage(const Arrays& A, uint32_t c0, uint32_t lane, T& S, const FlowLimit& limit) {
    using Site = typename T::Site;
    const Site* src;
    if constexpr (FP32)
        src = reinterpret_cast<const Site*>(A.sorted_off);
    else
        src = A.sorted_s;
    const uint32_t c1 = min(c0 + T::stage, S.total);
    if (lane == 0)
        mbar_expect(&S.bar, (c1 - c0) * (uint32_t)sizeof(Site) + (limit.stall == kStallCopy ? 16u : 0u));
    __syncwarp();
    if (lane < S.n_parts) {
        const StencilPart p = S.part[lane];
        const uint32_t b = max(lane == 0 ? 0u : S.part[lane - 1].end, c0), e = min(p.end, c1);
        if (b < e) bulk_copy(S.site + (b - c0), src + (p.base + b), (e - b) * (uint32_t)sizeof(Site), &S.bar);
    }
}

// dU in FP32 of the team's trial with a bound on its error against the FP64 sums: its warps take
// the staged candidates 32 at a time and list the pairs inside the cut-off band (1 in 6); the pair
// energies are evaluated 32 listed pairs at a time, so that those ~60 instructions run with every
// lane busy (two evaluations per trial instead of one per 32 candidates with five lanes). `phase`:
// the parity of the staging barrier, the first chunk already on its way. Where a copy does not arrive in
// time (mbar_wait) S.lost is set before a barrier of the team, and the caller drops the result: the next
// wait lies behind another barrier, so all threads read the same.
template <int DIM, int W, typename T>
__device__ __forceinline__ void lj_delta32(const Geometry& g, const Arrays& A, const Pair& P, uint32_t lane, uint32_t warp, T& S,
                                           uint32_t& phase, const FlowLimit& limit, float& d32, float& bound) {
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    float2* list = S.list[warp].q32;
    const uint32_t total = S.total;
    const int4 t32 = S.t32, s32 = S.s32;
    const float cut2 = P.lj_rcut2_hi32;
    float d = 0.f, err = 0.f, mag = 0.f;
    uint32_t listed = 0, rounds = 1, part = 0;
    auto evaluate = [&](uint32_t at) {
        const float2 r2 = list[at];
        float e, x;
        if (r2.x < cut2) {
            lj_pair32(P, r2.x, e, x);
            d += e;
            err += x;
            mag += fabsf(e);
        }
        if (r2.y < cut2) {
            lj_pair32(P, r2.y, e, x);
            d -= e;
            err += x;
            mag += fabsf(e);
        }
    };
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < total; c0 += T::stage) {
        if (c0 > 0) {
            if (team_any<W>(S.lost != 0u)) break;  // the chunk before has been read
            if (warp == 0) team_stage<true>(A, c0, lane, S, limit);
        }
        if constexpr (T::staged) {
            mbar_wait(&S.bar, phase, A.stats, limit, &S.lost);
            phase ^= 1u;
        }
        const uint32_t n = min(T::stage, total - c0), self = S.self - c0;
#pragma unroll 2
        for (uint32_t j0 = 32u * warp; j0 < n; j0 += 32u * W) {
            const uint32_t j = j0 + lane;
            int4 o;
            if constexpr (T::staged) {
                o = S.site[j];  // (j < T::stage; stale beyond n)
            } else {
                while (j < n && j >= S.part[part].end) ++part;
                o = j < n ? __ldcg(reinterpret_cast<const int4*>(A.sorted_off) + (S.part[part].base + j)) : t32;
            }
            const float rn = fixed_dist2<DIM>(g, t32, o), ro = fixed_dist2<DIM>(g, s32, o);
            const bool need = fminf(rn, ro) < cut2 && j < n && j != self;
            const unsigned b = __ballot_sync(full, need);
            if (need) list[listed + __popc(b & below)] = make_float2(rn, ro);
            listed += __popc(b);
            if (listed >= 32u) {
                __syncwarp();
                listed -= 32u;
                evaluate(listed + lane);
                rounds += 1;
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (lane < listed) evaluate(lane);
    // summation chains (per lane, the reduction, the warps' sums, the final difference), FP64's own
    // error
    const float chain = (float)(2u * rounds + 7u + W) * kU32 * 1.01f + 1e-9f;
    d32 = warp_sumf(d);
    bound = warp_sumf(err + chain * mag);
    if (W > 1) {
        if (lane == 0) S.sum32[warp] = make_float2(d32, bound);
        team_sync<W>();
        d32 = bound = 0.f;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            d32 += S.sum32[w].x;
            bound += S.sum32[w].y;
        }
    }
    bound += kU32 * fabsf(d32) + 1e-9f;
}

// FP64 energies of the trial site ta and of the current site tb against the stencil's candidates,
// and sum |e| over both (order_ambiguous), by the team. Like lj_delta32 the pairs inside the
// cut-off are listed first and their energies evaluated 32 at a time; a pair outside adds an exact
// zero and is left out. STAGED: S of the candidates comes from the staging buffer; else it is
// wrap(sorted_b) (the recheck of the FP32 pass, which does not keep S).
// INTERIOR: no space of the stencil is the first of an axis (which straddles the box boundary) or
// reached across the wrap, and an axis has six spaces or more: every site of the stencil then lies
// within 2 w <= L / 3 of the trial on each axis and any image at least 4 w away, so
// ref_dist2 would choose the site itself.
template <int DIM, bool GENERIC, bool INTERIOR, bool STAGED, int W, typename T>
__device__ __forceinline__ void lj_energies64(const Geometry& g, const Arrays& A, const Pair& P, const double* ta,
                                              const double* tb, uint32_t lane, uint32_t warp, T& S, uint32_t& phase,
                                              const FlowLimit& limit, double& ea, double& eb, double& mag) {
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    const double cut2 = !GENERIC || P.penalty == 0u ? P.lj_rcut2 : (P.penalty == 1u ? P.op_rcut2 : P.uv_rcut2);
    double2* list = S.list[warp].q64;
    const uint32_t total = S.total;
    double a = 0.0, b = 0.0, am = 0.0;
    uint32_t listed = 0, part = 0;
    auto evaluate = [&](uint32_t at) {
        const double2 r2 = list[at];
        const double x = soft_pair64<GENERIC>(P, r2.x), y = soft_pair64<GENERIC>(P, r2.y);
        a = dadd(a, x);
        b = dadd(b, y);
        am += GENERIC ? soft_pair_mag(P, r2.x, x) : fabs(x);
        am += GENERIC ? soft_pair_mag(P, r2.y, y) : fabs(y);
    };
    auto dist2 = [&](const double* t, const double* s) -> double {
        if (!INTERIOR) return ref_dist2<DIM>(g, t, s);
        double r2 = 0.0;
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            const double x = dsub(t[k], s[k]);
            r2 = dadd(r2, dmul(x, x));
        }
        return r2;
    };
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < total; c0 += T::stage) {
        if constexpr (STAGED && T::staged) {
            if (c0 > 0) {
                if (team_any<W>(S.lost != 0u)) break;  // the chunk before has been read
                if (warp == 0) team_stage<false>(A, c0, lane, S, limit);
            }
            mbar_wait(&S.bar, phase, A.stats, limit, &S.lost);
            phase ^= 1u;
        }
        const uint32_t n = min(T::stage, total - c0), self = S.self - c0;
#pragma unroll 1
        for (uint32_t j0 = 32u * warp; j0 < n; j0 += 32u * W) {
            const uint32_t j = j0 + lane;
            double rn = cut2, ro = cut2;
            if (j < n && j != self) {
                double sv[3];
                if constexpr (STAGED && T::staged) {
                    const double4 v = S.site[j];
                    sv[0] = v.x, sv[1] = v.y, sv[2] = v.z;
                } else {
                    while (c0 + j >= S.part[part].end) ++part;
                    const double4 v = ldcg4((STAGED ? A.sorted_s : A.sorted_b) + (S.part[part].base + c0 + j));
                    sv[0] = v.x, sv[1] = v.y, sv[2] = v.z;
                    if (!STAGED) wrap_inv<DIM>(g.L, g.invL, sv);
                }
                rn = dist2(ta, sv);
                ro = dist2(tb, sv);
            }
            const bool need = rn < cut2 || ro < cut2;
            const unsigned h = __ballot_sync(full, need);
            if (need) list[listed + __popc(h & below)] = make_double2(rn, ro);
            listed += __popc(h);
            if (listed >= 32u) {
                __syncwarp();
                listed -= 32u;
                evaluate(listed + lane);
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (!T::staged && total <= 32u && listed == 0u) {  // no pair: sums of zeros
        ea = eb = mag = 0.0;
        return;
    }
    if (lane < listed) evaluate(lane);
    ea = warp_sum(a);
    eb = warp_sum(b);
    mag = warp_sum(am);
    if (W > 1) {
        if (lane == 0) {
            S.sum64[warp][0] = ea;
            S.sum64[warp][1] = eb;
            S.sum64[warp][2] = mag;
        }
        team_sync<W>();
        ea = eb = mag = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            ea = dadd(ea, S.sum64[w][0]);
            eb = dadd(eb, S.sum64[w][1]);
            mag += S.sum64[w][2];
        }
    }
}

// The Metropolis test of the team's trial, slot k in space m (parallel_sweep.rs:267-268): FP32 sums
// first (FP32), the FP64 sums when their bound could change the decision. The candidates of
// the stencil in the team's scratch are on their way into its staging buffer; not decided where S.lost
// is set then.
template <int DIM, bool FP32, bool GENERIC, int W, typename T>
__device__ __forceinline__ bool lj_decide(const Geometry& g, const Arrays& A, const Pair& P, double kt,
                                          const uint32_t* m, uint32_t k, double u, float w_lo, float w_hi,
                                          uint32_t lane, uint32_t warp, T& S, uint32_t& phase, const FlowLimit& limit,
                                          PairStats& pst, uint8_t& flags) {
    float d32 = 0.f;
    if constexpr (FP32) {
        float b;
        lj_delta32<DIM, W>(g, A, P, lane, warp, S, phase, limit, d32, b);
        if (lane == 0 && warp == 0) pst.checks += 2u * (S.total - 1u);
        const float lo = __fsub_rd(d32, b), hi = __fadd_ru(d32, b);
        if (hi <= 0.f) return true;  // dU64 <= 0 for certain: accepted without a uniform
        if (lo > 0.f && hi < w_lo) return true;
        if (lo > 0.f && lo > w_hi) return false;
        flags |= kTrialRechecked;  // (also where a sum is not finite: every comparison is false)
    }
    const double t[3] = {S.t[0], S.t[1], DIM == 3 ? S.t[2] : 0.0};
    double si[3] = {S.s[0], S.s[1], DIM == 3 ? S.s[2] : 0.0};
    bool interior = !FP32;
    if (FP32) {
        const double4 b4 = ldcg4(A.sorted_b + k);
        si[0] = b4.x, si[1] = b4.y, si[2] = b4.z;
        wrap_inv<DIM>(g.L, g.invL, si);
    }
#pragma unroll
    for (int a = 0; a < DIM; ++a) interior = interior && g.shape[a] >= 6 && m[a] >= 2 && m[a] + 2 <= g.shape[a];
    double e_new, e_old, mag;
    if (!FP32 && interior)
        lj_energies64<DIM, GENERIC, !FP32, !FP32, W>(g, A, P, t, si, lane, warp, S, phase, limit, e_new, e_old, mag);
    else
        lj_energies64<DIM, GENERIC, false, !FP32, W>(g, A, P, t, si, lane, warp, S, phase, limit, e_new, e_old, mag);
    const double du = dsub(e_new, e_old);
    // order_ambiguous is false where dU lies well off 0 and u well off e0, or where no pair was in range:
    // the tests here imply its own (mag >= |dU| and S.total < 2^24 make order_bound less than 1e-8 mag) and
    // spare its divisions, and the exponential where dU < 0.
    bool accept = du <= 0.0;
    const double b = 1e-8 * mag;
    const bool few = S.total < (1u << 24) && mag > 1e-200;
    if (!(few && du < -b) && !(du == 0.0 && mag == 0.0 && u < 1.0 - 1e-15)) {
        const double e0 = exp(ddiv(-du, kt));
        if (!(few && du > b && b < 0.99e-3 * kt && fabs(u - e0) * kt > e0 * (4.1 * b + 1.1e-14 * kt)) &&
            order_ambiguous(du, mag, S.total, u, kt, e0))
            flags |= kTrialAmbiguous;
        accept = accept || u < e0;
    }
    if (lane == 0 && warp == 0) {
        if (FP32) {
            pst.rechecks++;
            const double err = fabs((double)d32 - du);
            pst.max_err = err > pst.max_err ? err : pst.max_err;
        }
        if (flags & kTrialAmbiguous) pst.ambiguous++;
    }
    return accept;
}

// The sweep: one team of W warps per trial in dataflow order (hmc_flow.cuh), all colour passes of
// colour sets [L.round, L.round_end) in one launch. BATCH: over every replica of a batch, with the
// box, checkerboard, pair parameters and kT of the trial's replica. INJ: the probe mode, team w
// decides injected trial w against the unchanged state (no order, no commit).
// The proposal (B + displacement, W1 = wrap, the space check, T = wrap(W1), fixed-point site) and the
// commit run on one lane per axis of the team's first warp; the proposal needs the own space's
// last colour set only and is done before the wait for the neighbours.
template <int DIM, bool FP32, bool GENERIC, bool BATCH, bool INJ, int WARPS, int MINB, int W, int STAGE>
__global__ void __launch_bounds__(32 * WARPS, MINB)
    k_flow_lj(Geometry g0, Arrays A, Pair P0, Launch L, Batch B, Injected J) {
    static_assert(W == 1 || W == WARPS, "a team is a warp or a block");
    constexpr unsigned full = 0xffffffffu;
    constexpr uint32_t kTeams = WARPS / W, kNear = DIM == 3 ? 27u : 9u, kOwn = kNear / 2;
    using TeamT = Team<FP32, BATCH, W, STAGE>;
    __shared__ TeamT s_team[kTeams];
    __shared__ FlowRange s_range;
    __shared__ uint32_t s_item[2];
    const uint32_t lane = threadIdx.x & 31u, axis = lane < DIM ? lane : 0u;
    const uint32_t warp = W == 1 ? 0u : threadIdx.x >> 5;  // within the team
    TeamT& S = s_team[W == 1 ? threadIdx.x >> 5 : 0u];
    if (lane == 0 && warp == 0) {
        mbar_init(&S.bar);
        S.lost = 0;
    }
    if (!INJ) {
        grid_dependency_wait();
        if (threadIdx.x == 0) {
            uint32_t round = L.round, round_end = L.round_end;
            if (BATCH && round == kRoundFromDevice) {
                round = *B.round_dev;
                round_end += round;
            }
            s_range = flow_range(A.stats, round, round_end, 1u << DIM);
        }
    }
    __syncthreads();
    const uint32_t n = INJ ? J.n : s_range.n;
    const uint32_t team = blockIdx.x * kTeams + (W == 1 ? threadIdx.x >> 5 : 0u), n_teams = gridDim.x * kTeams;
    auto take = [&]() -> uint32_t { return lane == 0 && warp == 0 ? atomicAdd(&A.stats->ticket, 1u) : 0u; };
    uint32_t n_accepted = 0, phase = 0, turn = 0;
    PairStats pst;
    uint32_t next = INJ ? team : take();
    for (;;) {
        uint32_t item = next;
        if (!INJ) {
            item = __shfl_sync(full, next, 0);
            if (W > 1) {
                // (two words: a thread may still read the last one's when a replica's entry is skipped)
                if (threadIdx.x == 0) s_item[turn] = item;
                __syncthreads();
                item = s_item[turn];
                turn ^= 1u;
            }
        }
        if (item >= n) break;
        next = INJ ? item + n_teams : take();  // in flight while this trial runs
        uint32_t m[3] = {0, 0, 0}, k, r = 0, round = 0;
        uint8_t flags = 0;
        if constexpr (INJ) {
            const uint64_t body = J.bodies[item];
            k = A.slot_of_body[body];
            unpack_m<DIM>(A.body_m[body], m);
            const double4 w4 = J.trial[item];
            double x[3] = {w4.x, w4.y, DIM == 3 ? w4.z : 0.0};
            uint32_t mt[3];
            if (!(point_to_space<DIM>(g0, x, mt) && cell_index<DIM>(g0, mt) == cell_index<DIM>(g0, m))) {
                if (lane == 0) {
                    J.decisions[item] = 0;
                    J.flags[item] = kTrialOutsideSpace;
                }
                continue;
            }
            wrap_inv<DIM>(g0.L, g0.invL, x);
            const double4 s4 = ldg4(A.sorted_s + k);
            if (lane == 0) {
                S.t[0] = x[0], S.t[1] = x[1], S.t[2] = x[2];
                S.s[0] = s4.x, S.s[1] = s4.y, S.s[2] = s4.z;
                S.t32 = fixed_site<DIM>(g0, x);
                S.s32 = __ldg(reinterpret_cast<const int4*>(A.sorted_off) + k);
            }
            const double u = J.u[item];
            float w_lo, w_hi;
            metropolis_bounds(u, L.kt, w_lo, w_hi);
            team_parts<DIM>(g0, A.cell_start, m, k, lane, S);
            team_stage<FP32>(A, 0, lane, S, L.flow);
            const bool accept = lj_decide<DIM, FP32, GENERIC, W>(g0, A, P0, L.kt, m, k, u, w_lo, w_hi, lane, warp, S,
                                                                 phase, L.flow, pst, flags);
            if (S.lost) break;
            if (lane == 0) {
                J.decisions[item] = accept;
                J.flags[item] = flags;
            }
            __syncwarp();
        } else {
            const uint4 di = __ldg(A.draw_i + item);
            if (BATCH) {
                if (di.x == kNoTrial) continue;  // the replica has finished its colour sets
                uint32_t color, entry;
                flow_item(s_range, item, round, color, entry);
                r = __ldg(B.color_rep + (size_t)color * B.color_stride + entry);
            } else {
                round = s_range.r0 + item / s_range.per_set;
            }
            const double u = __ldg(reinterpret_cast<const double*>(A.draw_d + item) + 3);
            k = di.x;
            unpack_m<DIM>(di.y, m);
            if constexpr (BATCH) {
                if (warp == 0) {
                    static_assert(sizeof(Replica) % 8 == 0, "copied in 8-byte words");
                    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(B.rep + r);
                    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&S.rep);
#pragma unroll
                    for (uint32_t i = 0; i < (sizeof(Replica) / 8 + 31) / 32; ++i)
                        if (i * 32 + lane < sizeof(Replica) / 8) dst[i * 32 + lane] = __ldg(src + i * 32 + lane);
                    __syncwarp();
                }
            }
            const Replica* R;
            if constexpr (BATCH)
                R = &S.rep;
            else
                R = nullptr;
            const Geometry& g = BATCH ? R->g : g0;
            const Pair& P = BATCH ? R->p : P0;
            const uint32_t ma = axis == 0 ? m[0] : (axis == 1 ? m[1] : m[2]);
            double ta = 0.0;
            if (warp == 0) {
                const uint32_t base = BATCH ? R->cell_base : 0u;
                const double dv = __ldg(reinterpret_cast<const double*>(A.draw_d + item) + axis);
                uint32_t color = 0;
#pragma unroll
                for (int a = 0; a < DIM; ++a) color = (color << 1) | (m[a] & 1u);
                uint32_t space = 0, need = 0;
                if (lane < kNear) flow_need<DIM>(g, m, color, round, lane, space, need);
                const uint32_t* word = A.progress + base + space;
                bool ok = lane >= kNear;
                team_parts<DIM>(g, A.cell_start + base, m, k, lane, S);
                bool going = flow_wait(word, need, 1u << kOwn, ok, A.stats, L.flow);
                __syncwarp();
                const AxisGeometry ax = axis_geometry<DIM>(g, axis);
                const double b = __ldcg(reinterpret_cast<const double*>(A.sorted_b + k) + axis);
                // the current site
                if constexpr (FP32) {
                    const int s = __ldcg(reinterpret_cast<const int*>(A.sorted_off + k) + axis);
                    if (lane < DIM) reinterpret_cast<int*>(&S.s32)[lane] = s;
                } else {
                    const double s = __ldcg(reinterpret_cast<const double*>(A.sorted_s + k) + axis);
                    if (lane < DIM) S.s[lane] = s;
                }
                const double w1 = wrap_axis(ax.L, ax.invL, dadd(b, dv));  // W1 = wrap(propose(..))
                const bool inside = __all_sync(full, axis_in_space(ax.origin, ax.width, ax.invW, ax.shape, ma, w1));
                ta = wrap_axis(ax.L, ax.invL, w1);  // the trial site T = wrap(W1)
                if (lane < DIM) {
                    S.t[lane] = ta;
                    if (FP32) reinterpret_cast<int*>(&S.t32)[lane] = fixed_axis(ax.invL, ta);
                }
                if (inside && going) going = flow_wait(word, need, full, ok, A.stats, L.flow);
                if (lane == 0) S.valid = going ? (inside ? 1u : 0u) : 2u;
                __syncwarp();
                if constexpr (TeamT::staged) {
                    if (inside && going) {
                        fence_proxy_async();
                        team_stage<FP32>(A, 0, lane, S, L.flow);
                    }
                }
            }
            team_sync<W>();
            const uint32_t valid = S.valid;
            if (valid == 2u) break;  // the launch is given up
            if (valid == 1u) {
                const bool accept =
                    lj_decide<DIM, FP32, GENERIC, W>(g, A, P, BATCH ? R->kt : L.kt, m, k, u, __uint_as_float(di.z),
                                                     __uint_as_float(di.w), lane, warp, S, phase, L.flow, pst, flags);
                if (TeamT::staged && S.lost) break;  // not decided, the whole team gives up
                if (accept && warp == 0) {
                    // update_body_properties: body = T, site = wrap(body)
                    const AxisGeometry ax = axis_geometry<DIM>(g, axis);
                    const double sv = wrap_axis(ax.L, ax.invL, ta);
                    if (lane < DIM) {
                        reinterpret_cast<double*>(A.sorted_b + k)[lane] = ta;
                        if (FP32)
                            reinterpret_cast<int*>(A.sorted_off + k)[lane] = fixed_axis(ax.invL, sv);
                        else
                            reinterpret_cast<double*>(A.sorted_s + k)[lane] = sv;
                        reinterpret_cast<double*>(A.body_pos + A.sorted_body[k])[lane] = ta;
                    }
                    n_accepted += lane == 0;
                    if (BATCH && lane == 0) atomicAdd(B.accepted + r, 1ull);
                }
            }
            __syncwarp();
            if (lane == 0 && warp == 0)
                store_release(A.progress + (BATCH ? R->cell_base : 0u) + cell_index<DIM>(g, m), round + 1u);
        }
    }
    flush_stats(A.stats, pst, n_accepted);
}

// Injected moves: warp per move. delta_h gets dU64 (stencils around the trial's space for the
// final energy and around the body's space for the initial energy); the decision follows the
// precision mode with the given uniform.
template <int DIM, bool FP32>
__global__ void __launch_bounds__(128) k_eval_lj(Geometry g, Arrays A, Pair P, const uint64_t* bodies,
                                                 const double4* trial, const double* uu, double kt, uint32_t n,
                                                 uint8_t* decisions, uint8_t* rechecked, double* delta_h) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    PairStats pst;
    if (i < n) {
        const uint32_t k = A.slot_of_body[bodies[i]];
        const double4 w4 = trial[i];
        double t[3] = {w4.x, w4.y, DIM == 3 ? w4.z : 0.0};
        wrap_inv<DIM>(g.L, g.invL, t);
        const double4 s4 = ldg4(A.sorted_s + k);
        const double si[3] = {s4.x, s4.y, s4.z};
        uint32_t mt[3], mi[3];
        const bool ok = point_to_space<DIM>(g, t, mt) && point_to_space<DIM>(g, si, mi);
        uint8_t dec = 0, rech = 0;
        double du = 0.0;
        if (ok) {
            const FlatStencil ft = flat_stencil<DIM>(g, A.cell_start, mt, lane);
            const FlatStencil fi = flat_stencil<DIM>(g, A.cell_start, mi, lane);
            double e_new, e_old;
            double mag_new, mag_old;
            lj_energy64<DIM>(g, A, P, t, ft, k, lane, e_new, mag_new);
            lj_energy64<DIM>(g, A, P, si, fi, k, lane, e_old, mag_old);
            du = dsub(e_new, e_old);
            const double u = uu[i];
            bool dec64 = du <= 0.0 || u < exp(ddiv(-du, kt));
            dec = dec64 ? 1 : 0;
            if (FP32) {
                // FP32 sums need a common space for both sites: when the trial left the body's
                // space, they are evaluated in FP64 as the sweep never sees such a trial.
                const bool same = mt[0] == mi[0] && mt[1] == mi[1] && (DIM == 2 || mt[2] == mi[2]);
                if (same) {
                    const int4 c32 = __ldg(reinterpret_cast<const int4*>(A.sorted_off) + k);
                    const Sums32 s = lj_energy32<DIM>(g, A, P, fixed_site<DIM>(g, t), c32, ft, k, lane);
                    const float d32 = s.e_new - s.e_old;
                    const float b = s.err + (float)(s.terms + 7) * kU32 * s.mag * 1.01f + kU32 * fabsf(d32) +
                                    1e-9f * (s.mag + 1.f);
                    int d = -1;
                    if (isfinite(d32) && isfinite(b)) {
                        const double lo = (double)d32 - b, hi = (double)d32 + b;
                        if (hi <= 0.0) {
                            d = 1;
                        } else if (lo > 0.0) {
                            const double t_hi = exp(-lo / kt) * (1.0 + 1e-12), t_lo = exp(-hi / kt) * (1.0 - 1e-12);
                            d = u < t_lo ? 1 : (u >= t_hi ? 0 : -1);
                        }
                    }
                    if (d < 0) {
                        rech = 1;
                        d = dec64 ? 1 : 0;  // the FP64 recheck
                    }
                    dec = (uint8_t)d;
                } else {
                    rech = 1;
                }
            }
        } else if (lane == 0) {
            atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
        }
        if (lane == 0) {
            decisions[i] = dec;
            rechecked[i] = rech;
            delta_h[i] = du;
        }
    }
    flush_stats(A.stats, pst, 0u);
}

// The sequential-stream tuner for Lennard-Jones and the overlap penalty (tune_stream_run):
// dH = E_final - E_initial in FP64 (the warp over the stencils of the trial site's and of the
// current site's spaces), then the reference's test: rejected at dH = inf, accepted at dH <= 0
// without a uniform, else the stream's next uniform against exp(-dH / kT). A decision that
// another summation order could change (order_ambiguous; also a dH <= 0 whose bound reaches
// above 0, where another order would draw a uniform) is counted in J.ambiguous.
template <int DIM>
__global__ void __launch_bounds__(32) k_tune_stream_lj(TuneJob* jobs, uint32_t n_jobs) {
    if (blockIdx.x >= n_jobs) return;
    TuneJob& J = jobs[blockIdx.x];
    const Geometry& g = J.g;
    const Arrays& A = J.a;
    const Pair& P = J.p;
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long ambiguous = 0;
    tune_stream_run(
        J, [&](Sfc64& rng, double m, uint32_t b, double* x, double*) { tune_translate<DIM>(rng, g, A, m, b, x); },
        [&](Sfc64& rng, uint32_t b, const double* x, const double*) -> bool {
            double t[3] = {x[0], x[1], x[2]};
            wrap_inv<DIM>(g.L, g.invL, t);
            const uint32_t k = A.slot_of_body[b];
            const double4 s4 = ldg4(A.sorted_s + k);
            const double si[3] = {s4.x, s4.y, s4.z};
            uint32_t mt[3] = {0, 0, 0}, mi[3] = {0, 0, 0};
            if (!(point_to_space<DIM>(g, t, mt) && point_to_space<DIM>(g, si, mi))) {
                if (lane == 0) atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
                return false;
            }
            const FlatStencil ft = flat_stencil<DIM>(g, A.cell_start, mt, lane);
            const FlatStencil fi = flat_stencil<DIM>(g, A.cell_start, mi, lane);
            double e_new, e_old, mag_new, mag_old;
            lj_energy64<DIM>(g, A, P, t, ft, k, lane, e_new, mag_new);
            if (e_new == __longlong_as_double(0x7ff0000000000000ll)) return false;  // the reference stops here
            lj_energy64<DIM>(g, A, P, si, fi, k, lane, e_old, mag_old);
            const double du = dsub(e_new, e_old);
            if (!(du != __longlong_as_double(0x7ff0000000000000ll))) return false;
            const uint32_t n = ft.total + fi.total;
            const double mag = mag_new + mag_old;
            if (du <= 0.0) {
                if (isfinite(mag) && du + order_bound(du, mag, n) > 0.0) ambiguous++;
                return true;
            }
            const double u = uniform01(rng);
            const double e0 = exp(ddiv(-du, J.kt));
            if (order_ambiguous(du, mag, n, u, J.kt, e0)) ambiguous++;
            return u < e0;
        });
    if (lane == 0) J.ambiguous = ambiguous;
}

// Total pair energy, pairs (i < j) in FP64 (PairwiseCutoff::total_energy,
// pairwise_cutoff.rs:720-745); one thread per body, a warp's sums added atomically (one atomic per
// body, all on one word, took most of the kernel). Away from the box's ends no image of a site is nearer
// than the site (see lj_energies64), so the distance needs no ghost rule there. 2^17 sites at 0.8 with a cut-off
// of 2.5: 402 us with both and a pair's energy where it is found, 352 us without both, 303 us with the
// pairs in range collected (pairs_in_range).
template <int DIM>
__global__ void k_energy_lj(Geometry g, Arrays A, Pair P, uint32_t n, double* out) {
    __shared__ double s_list[4][64];
    double e = 0.0;
    const auto dist = [&](const double* t, const double* s, const uint32_t* m) {
        bool interior = true;
#pragma unroll
        for (int a = 0; a < DIM; ++a) interior = interior && g.shape[a] >= 6 && m[a] >= 2 && m[a] + 2 <= g.shape[a];
        if (!interior) return ref_dist2<DIM>(g, t, s);
        double r2 = 0.0;
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const double d = dsub(t[a], s[a]);
            r2 = dadd(r2, dmul(d, d));
        }
        return r2;
    };
    // (the other soft energies test the cut-off themselves)
    pairs_in_range<DIM>(g, A, n, blockIdx.x * blockDim.x + threadIdx.x, P.penalty ? INFINITY : P.lj_rcut2,
                        s_list[threadIdx.x >> 5], dist, [&](double r2) { e += lj_pair64(P, r2); });
    e = warp_sum(e);
    if ((threadIdx.x & 31u) == 0 && e != 0.0) atomicAdd(out, e);
}

}  // namespace

namespace {
using LjKernel = void (*)(Geometry, Arrays, Pair, Launch, Batch, Injected);

// The compiled launch variants 1 .. 4 of kLjShapes and kBatchLjShapes: teams of 1, 2, 4 and 8 warps.
struct LjVariant {
    LjKernel kernel;
    uint32_t warps, team;  // per block, per trial
};
// Variant 0: the largest team of which the chip holds about as many as one colour has trials (`list`):
// a larger team decides a trial in less time, but fewer fit (148 SMs hold about 440 of 8 warps, 890 of
// 4, 1,780 of 2). And no warp without two steps of candidates (a stencil's mean number).
// Four sweeps of n sites at density 0.8, teams of 1 / 2 / 4 / 8 warps, us, FP32: n = 16,384 (216
// trials a colour) 5971 / 4565 / 3712 / 3469; 65,536 (512) 6404 / 4617 / 3713 / 3835; 131,072 (1,000)
// 6895 / 5102 / 4331 / 6467; 262,144 (2,197) 6239 / 5284 / 6670 / 12043; 2-D (40 candidates), 65,536 sites
// (3,844): 654 / 990 / 1575 / 2802.
uint32_t lj_team_variant(uint32_t list, double candidates) {
    const uint32_t by_trials = list > 2300 ? 1u : (list > 1060 ? 2u : (list > 480 ? 3u : 4u));
    const uint32_t by_steps = candidates < 128 ? 1u : (candidates < 192 ? 2u : (candidates < 256 ? 3u : 4u));
    return by_trials < by_steps ? by_trials : by_steps;
}
// How a one-warp trial gets its sites: staged, or (few candidates) loaded by its lanes, in a kernel for few
// trials, which is not short of registers, or for many, nine blocks an SM. The staging buffers let an SM
// hold 24 warps (FP64: 16), too few where a trial is short and a colour has more trials than that; and a
// copy's way through the barrier is longer than a load. A sweep, us, FP64 (FP32) staged / few / many: 2-D
// at density 0.3 (17 candidates), 800 spaces a colour 84 / 83 / 85 (81 / 79 / 80), 3,000 95 / 89 / 98
// (88 / 88 / 94), 5,000 127 / 112 / 102 (102 / 107 / 100), 30,000 507 / 424 / 312 (358 / 401 / 291); 3-D at
// 0.1 (43), 3,000 157 / 168 / 184 (141 / 145 / 160), 5,000 204 / 189 / 195 (159 / 175 / 171), 30,000
// 1016 / 898 / 694 (715 / 822 / 627); 3-D at 0.03 (13), 3,000 114 / 109 / 120 (157 / 155 / 167). A launch per
// colour pass took 318 (360), 729 (817) and 132 (327) us for the last of each.
enum LjStaging { kLjStaged, kLjFew, kLjMany };
LjStaging lj_staging(uint32_t list, double candidates) {
    if (list >= 4500 && candidates <= 96) return kLjMany;
    return candidates <= 24 ? kLjFew : kLjStaged;
}
template <int DIM, bool FP32, bool GENERIC, bool BATCH>
LjVariant lj_kernel(uint32_t v, LjStaging sites) {
    // single-warp teams share a block: FP32 staging buffers of four, FP64 of two fit 48 KB
    constexpr int N = FP32 ? 4 : 2;
    switch (v) {
        case 2: return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, 2, FP32 ? 12 : 8, 2, kStage>, 2, 2};
        case 3: return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, 4, 6, 4, kStage>, 4, 4};
        case 4: return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, 8, 3, 8, kStage>, 8, 8};
        default:
            if (sites == kLjMany) return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, 4, 9, 1, kDirect>, 4, 1};
            if (sites == kLjFew) return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, 4, 4, 1, kDirect>, 4, 1};
            return {k_flow_lj<DIM, FP32, GENERIC, BATCH, false, N, FP32 ? 6 : 8, 1, kStage>, N, 1};
    }
}
LjVariant lj_kernel(int dim, bool fp32, bool generic, bool batch, uint32_t variant, uint32_t list, double per_space) {
    static_assert(n_shapes(kLjShapes) == 5 && n_shapes(kBatchLjShapes) == 5, "the rule and four kernels");
    const uint32_t v = variant == 0 || variant > 4 ? lj_team_rule(dim, list, per_space) : variant;
    const LjStaging w = lj_staging(list, per_space * (dim == 3 ? 27 : 9));
    if (batch) {
        if (dim == 2) return fp32 ? lj_kernel<2, true, false, true>(v, w) : lj_kernel<2, false, false, true>(v, w);
        return fp32 ? lj_kernel<3, true, false, true>(v, w) : lj_kernel<3, false, false, true>(v, w);
    }
    if (generic) return dim == 2 ? lj_kernel<2, false, true, false>(v, w) : lj_kernel<3, false, true, false>(v, w);
    if (dim == 2) return fp32 ? lj_kernel<2, true, false, false>(v, w) : lj_kernel<2, false, false, false>(v, w);
    return fp32 ? lj_kernel<3, true, false, false>(v, w) : lj_kernel<3, false, false, false>(v, w);
}

// The two kernels of a range of colour sets whose longest colour list has at most `list` entries.
// The flow kernel gets a team for each trial of two colour lists (the trials behind the running
// colour wait at most for it), at most one resident wave.
cudaError_t launch_flow(int dim, bool batch, const LjVariant& v, const Geometry& g, const Arrays& a, const Pair& p,
                        const Launch& l, const Batch& b, uint32_t list, cudaStream_t s) {
    if (list == 0) return cudaSuccess;
    using DrawKernel = void (*)(Geometry, Arrays, Launch, Batch);
    const DrawKernel d = dim == 2 ? (batch ? k_draw_lj<2, true> : k_draw_lj<2, false>)
                                  : (batch ? k_draw_lj<3, true> : k_draw_lj<3, false>);
    const uint64_t entries = ((uint64_t)list << dim) * 16u;
    uint64_t blocks = (entries + 127) / 128;
    const uint64_t wave_d = (uint64_t)resident_wave((const void*)d);
    PassLaunch pd((uint32_t)(blocks < wave_d ? blocks : wave_d), l.overlap_previous != 0, s);
    cudaError_t e = cudaLaunchKernelEx(&pd.cfg, d, g, a, l, b);
    if (e != cudaSuccess) return e;
    blocks = ((uint64_t)list * 2 * v.team + v.warps - 1) / v.warps;
    const uint64_t wave = (uint64_t)resident_wave((const void*)v.kernel, (int)(32 * v.warps));
    PassLaunch pl((uint32_t)(blocks < wave ? blocks : wave), l.overlap_previous != 0, s, 32 * v.warps);
    return cudaLaunchKernelEx(&pl.cfg, v.kernel, g, a, p, l, b, Injected{});
}
}  // namespace

uint32_t lj_team_rule(int dim, uint32_t list, double per_space) {
    return lj_team_variant(list, per_space * (dim == 3 ? 27 : 9));
}

cudaError_t launch_flow_lj(int dim, bool fp32, bool generic, const Geometry& g, const Arrays& a, const Pair& p,
                           const Launch& l, cudaStream_t s, uint32_t variant) {
    return launch_flow(dim, false, lj_kernel(dim, fp32, generic, false, variant, g.color_stride, (double)l.n_bodies / g.n_cells),
                       g, a, p, l, Batch{},
                       g.color_stride, s);
}

cudaError_t launch_flow_batch_lj(int dim, bool fp32, const Batch& b, const Arrays& a, uint32_t round,
                                 uint32_t round_end, const FlowLimit& limit, cudaStream_t s, uint32_t variant) {
    Launch l{};
    l.flow = limit;
    l.overlap_previous = 1;
    l.round = round;
    l.round_end = round_end;
    return launch_flow(dim, true, lj_kernel(dim, fp32, false, true, variant, b.color_stride, (double)b.n_bodies / b.n_cells),
                       Geometry{}, a, Pair{}, l, b,
                       b.color_stride, s);
}

cudaError_t launch_tune_stream_lj(int dim, TuneJob* jobs, uint32_t n_jobs, cudaStream_t s) {
    if (n_jobs == 0) return cudaSuccess;
    if (dim == 2)
        k_tune_stream_lj<2><<<n_jobs, 32, 0, s>>>(jobs, n_jobs);
    else
        k_tune_stream_lj<3><<<n_jobs, 32, 0, s>>>(jobs, n_jobs);
    return cudaGetLastError();
}

cudaError_t launch_trials_lj(int dim, bool fp32, const Geometry& g, const Arrays& a, const Pair& p, double kt,
                             const Injected& j, cudaStream_t s) {
    if (j.n == 0) return cudaSuccess;
    Launch l{};
    l.kt = kt;
    // single-warp teams, as the sweep's variant 1
    const LjKernel k = dim == 2 ? (fp32 ? k_flow_lj<2, true, false, false, true, 4, 6, 1, kStage>
                                        : k_flow_lj<2, false, true, false, true, 2, 8, 1, kStage>)
                                : (fp32 ? k_flow_lj<3, true, false, false, true, 4, 6, 1, kStage>
                                        : k_flow_lj<3, false, true, false, true, 2, 8, 1, kStage>);
    const uint32_t warps = fp32 ? 4u : 2u, n = (j.n + warps - 1) / warps;
    const uint32_t wave = (uint32_t)resident_wave((const void*)k, (int)(32 * warps));
    k<<<n < wave ? n : wave, 32 * warps, 0, s>>>(g, a, p, l, Batch{}, j);
    return cudaGetLastError();
}

cudaError_t launch_eval_lj(int dim, bool fp32, const Geometry& g, const Arrays& a, const Pair& p,
                           const uint64_t* bodies, const double4* trial, const double* u, double kt, uint32_t n,
                           uint8_t* decisions, uint8_t* rechecked, double* delta_h, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = (n + 3) / 4;
    if (dim == 2) {
        if (fp32)
            k_eval_lj<2, true><<<blocks, 128, 0, s>>>(g, a, p, bodies, trial, u, kt, n, decisions, rechecked, delta_h);
        else
            k_eval_lj<2, false><<<blocks, 128, 0, s>>>(g, a, p, bodies, trial, u, kt, n, decisions, rechecked, delta_h);
    } else {
        if (fp32)
            k_eval_lj<3, true><<<blocks, 128, 0, s>>>(g, a, p, bodies, trial, u, kt, n, decisions, rechecked, delta_h);
        else
            k_eval_lj<3, false><<<blocks, 128, 0, s>>>(g, a, p, bodies, trial, u, kt, n, decisions, rechecked, delta_h);
    }
    return cudaGetLastError();
}

cudaError_t launch_energy_lj(int dim, const Geometry& g, const Arrays& a, const Pair& p, uint32_t n, double* out,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (dim == 2)
        k_energy_lj<2><<<(n + 127) / 128, 128, 0, s>>>(g, a, p, n, out);
    else
        k_energy_lj<3><<<(n + 127) / 128, 128, 0, s>>>(g, a, p, n, out);
    return cudaGetLastError();
}

}  // namespace hmc
