// Sweeps of few hard spheres or disks in dataflow order (hmc_flow.cuh): PairwiseCutoff<HardSphere> under
// Translate, all colour passes of a sweep in one launch.
//
// A colour pass gives a trial to one lane (hmc_kernels.cu): ~27 pair tests behind a chain of dependent
// loads. That is cheapest where a colour holds trials enough to hide the chain, but a small box is one
// chain after another, and a launch after another. Here nine lanes share a trial, three trials a warp: a
// lane takes one row of the 3^d spaces around the trial (three spaces in 3-D, one in 2-D), so what a
// trial waits for is its neighbours' progress, one load of sites, the pair tests and the commit.
// Measured (us per sweep with the cell-list rebuild, one lane per trial against this): 3-D at packing
// fraction 0.50, 16,384 spheres FP32 238 / 125, FP64 480 / 163; 50,021 spheres FP32 231 / 138, FP64
// 459 / 178; 2-D at 0.65, 16,384 disks FP32 77 / 71, FP64 87 / 71. A colour level of 50,021 spheres
// takes 7 us, of 4,096 disks 3.4 us: latency of the chain (waiting warps outnumber working ones).
// Without gain here, so left out: loading the next trials' draws and ranges ahead, relaxed polls
// with one fence (4,096 disks 66 instead of 61 us), more than four blocks per SM (50,021 spheres
// 2.74 ms for 20 sweeps with four, 3.1 ms with six or three).
#include <cuda_runtime.h>

#include <type_traits>

#include "hmc_flow.cuh"

namespace hmc {
namespace {

constexpr uint32_t kTrials = 3, kLanes = 9;  // trials of a warp, lanes of a trial
template <int DIM>
constexpr int kSpaces = DIM == 3 ? 3 : 1;    // spaces of a lane

// What the random streams of the trials of colour sets [L.round, L.round_end) give, one thread per trial:
// the chosen body's slot, the space and the displacement. Also the spaces' progress, and the ticket.
template <int DIM>
__global__ void __launch_bounds__(128) k_draw_sphere(Geometry g, Arrays A, Launch L) {
    grid_dependency_wait();
    allow_dependent_launch();
    const FlowRange f = flow_range(A.stats, L.round, L.round_end, 1u << DIM);
    if (blockIdx.x == 0 && threadIdx.x == 0) A.stats->ticket = L.flow.stall == kStallTrial ? 1u : 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += gridDim.x * blockDim.x) {
        uint32_t round, color, entry;
        flow_item(f, i, round, color, entry);
        entry = flow_rotated(A.stats->color_count[color], round, color, 1u << DIM, g.shape[0], entry);
        const uint32_t packed = __ldg(A.color_cells + (size_t)color * g.color_stride + entry);
        uint32_t m[3] = {0, 0, 0};
        unpack_m<DIM>(packed, m);
        const uint32_t cell = cell_index<DIM>(g, m);
        if (round == f.r0) A.progress[cell] = f.r0;
        const uint32_t start = __ldg(A.cell_start + cell);
        const uint32_t count = __ldg(A.cell_start + cell + 1) - start;
        Sfc64 rng = make_rng(L.step, L.substep + round, L.seed, (uint64_t)cell);
        const uint32_t k = start + canon_range_u32(rng, count);
        double dv[3];
        ball_sample<DIM>(rng, L.max_move, A.zig_x, A.zig_f, dv);
        A.draw_d[i] = make_double4(dv[0], dv[1], DIM == 3 ? dv[2] : 0.0, 0.0);
        A.draw_i[i] = make_uint4(k, packed, 0u, 0u);
    }
}

// The part of trial space m's stencil that lane `row` (< 9) of the trial takes: up to three spaces, each with
// its offset in spaces from m, its bodies' slots [start, end) and the progress the trial needs of it.
template <int DIM>
struct RowSpaces {
    uint32_t cell[kSpaces<DIM>], start[kSpaces<DIM>], end[kSpaces<DIM>], need[kSpaces<DIM>];
    int d0, d1;  // 3-D: the row's offset on the slow axes (2-D: on both axes)
};
template <int DIM>
__device__ __forceinline__ void row_spaces(const Geometry& g, const uint32_t* __restrict__ cs, const uint32_t* m,
                                           uint32_t color, uint32_t round, uint32_t row, bool active,
                                           RowSpaces<DIM>& R) {
    R.d0 = (int)(row / 3u) - 1;
    R.d1 = (int)(row % 3u) - 1;
    const uint32_t n0 = wrap_index((int)m[0] + R.d0, g.shape[0]), n1 = wrap_index((int)m[1] + R.d1, g.shape[1]);
    // two spaces on an axis: -1 and +1 are the same one
    active = active && !(g.shape[0] == 2 && R.d0 < 0) && !(g.shape[1] == 2 && R.d1 < 0);
#pragma unroll
    for (int i = 0; i < kSpaces<DIM>; ++i) {
        uint32_t cell = n0 * g.shape[1] + n1, c = ((n0 & 1u) << 1) | (n1 & 1u);
        bool on = active;
        if (DIM == 3) {
            const uint32_t n2 = wrap_index((int)m[2] + i - 1, g.shape[2]);
            cell = cell * g.shape[2] + n2;
            c = (c << 1) | (n2 & 1u);
            on = on && !(g.shape[2] == 2 && i == 0);
        }
        R.cell[i] = cell;
        R.start[i] = on ? __ldg(cs + cell) : 0u;
        R.end[i] = on ? __ldg(cs + cell + 1) : 0u;
        R.need[i] = round + (c < color ? 1u : 0u);
    }
}

__device__ __forceinline__ float4 ldcg_site(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ double4 ldcg_site(const double4* p) { return ldcg4(p); }

// Wait until space cell[i] has finished need[i] colour sets for every i in `pending` of every lane. False: the
// launch is given up.
template <int N>
__device__ __forceinline__ bool sphere_wait(const uint32_t* progress, const uint32_t* cell, const uint32_t* need,
                                            unsigned pending, DeviceStats* stats, const FlowLimit& limit) {
    const unsigned full = 0xffffffffu;
    unsigned long long t0 = 0;
    for (uint32_t spins = 0;; ++spins) {
        uint32_t v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = (pending >> i) & 1u ? load_acquire(progress + cell[i]) : 0u;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (v[i] >= need[i]) pending &= ~(1u << i);
        if (!__any_sync(full, pending != 0u)) return true;
        __nanosleep(20);
        if ((spins & 1023u) == 1023u) {
            const unsigned long long now = global_ns();
            if (t0 == 0) t0 = now;
            bool stop = *(volatile unsigned int*)&stats->error_flags != 0u;
            if (now - t0 > limit.wait_ns) {
                atomicOr(&stats->error_flags, kErrFlowTimeout);
                stop = true;
            }
            if (__any_sync(full, stop)) return false;
        }
    }
}

// The reference's FP64 squared distance of site t and slot q. S of the slot is wrap(B).
template <int DIM>
__device__ __forceinline__ double sphere_dist2_fp64(const Geometry& g, const double4* sorted_b, double tx, double ty,
                                                 double tz, uint32_t q) {
    const double t[3] = {tx, ty, tz};
    const double4 b4 = ldcg4(sorted_b + q);
    double sv[3] = {b4.x, b4.y, b4.z};
    wrap_inv<DIM>(g.L, g.invL, sv);
    return ref_dist2<DIM>(g, t, sv);
}

// INJ: the probe mode (Injected): injected trials are decided against the unchanged state.
template <int DIM, bool FP32, bool INJ, int MINB>
__global__ void __launch_bounds__(128, MINB) k_flow_sphere(Geometry g, Arrays A, Pair P, Launch L, Injected J) {
    constexpr unsigned full = 0xffffffffu;
    constexpr int SP = kSpaces<DIM>;
    using Site = typename std::conditional<FP32, float4, double4>::type;
    __shared__ FlowRange s_range;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t trial = lane / kLanes, row = lane - trial * kLanes;  // trial 3: the five spare lanes
    const uint32_t head = trial * kLanes;
    const unsigned mine = (0x1ffu << head) & 0x7ffffffu;  // the trial's lanes
    const uint32_t axis = DIM == 3 ? row % 3u : row & 1u;
    const AxisGeometry ax = axis_geometry<DIM>(g, axis);
    if (!INJ) {
        grid_dependency_wait();
        if (threadIdx.x == 0) s_range = flow_range(A.stats, L.round, L.round_end, 1u << DIM, kTrials);
        __syncthreads();
    }
    const FlowRange& f = s_range;
    const uint32_t n_units = INJ ? (J.n + kTrials - 1u) / kTrials : f.n_units;
    const uint32_t n_warps = gridDim.x * 4u;
    auto take = [&]() -> uint32_t { return lane == 0 ? atomicAdd(&A.stats->ticket, 1u) : 0u; };
    uint32_t n_accepted = 0;
    PairStats st;
    uint32_t next = INJ ? blockIdx.x * 4u + (threadIdx.x >> 5) : take();
    for (;;) {
        const uint32_t unit = INJ ? next : __shfl_sync(full, next, 0);
        if (unit >= n_units) break;
        next = INJ ? unit + n_warps : take();  // in flight while these trials run
        uint32_t round = 0, color = 0, m[3] = {0, 0, 0}, k = 0;
        bool valid;
        double x = 0.0;
        uint8_t flag = 0;
        if constexpr (INJ) {
            const uint32_t i = unit * kTrials + trial;
            valid = trial < kTrials && i < J.n;
            if (valid) {
                const uint64_t body = J.bodies[i];
                k = A.slot_of_body[body];
                const double4 w = J.trial[i];
                const double w1[3] = {w.x, w.y, DIM == 3 ? w.z : 0.0};
                valid = point_to_space<DIM>(g, w1, m);
                if (!valid) {
                    atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
                } else {
                    if (cell_index<DIM>(g, m) != A.body_cell[body]) flag |= kTrialOutsideSpace;
                    x = axis == 0 ? w1[0] : (axis == 1 ? w1[1] : w1[2]);
                }
            }
        } else {
            uint32_t entry;
            flow_unit(f, unit, round, color, entry);
            entry = entry * kTrials + trial;
            valid = trial < kTrials && entry < f.count[color];
            if (valid) {
                const uint32_t e = (round - f.r0) * f.per_set + f.prefix[color] + entry;
                const uint2 d = __ldg(reinterpret_cast<const uint2*>(A.draw_i + e));
                k = d.x;
                unpack_m<DIM>(d.y, m);
                x = __ldg(reinterpret_cast<const double*>(A.draw_d + e) + axis);
            }
        }
        const bool has = valid;
        RowSpaces<DIM> R;
        row_spaces<DIM>(g, A.cell_start, m, color, round, row, has, R);
        // The trial site, an axis a lane. The own space's bodies move in its own trials only, so the
        // proposal needs no more than the trial of the colour set before.
        const uint32_t ma = axis == 0 ? m[0] : (axis == 1 ? m[1] : m[2]), cell = cell_index<DIM>(g, m);
        double ta = 0.0;
        if (INJ) {
            ta = wrap_axis(ax.L, ax.invL, x);  // T = wrap(W1), as delta_energy_one wraps the site
        } else {
            if (round > f.r0 && !sphere_wait<1>(A.progress, &cell, &round, has ? 1u : 0u, A.stats, L.flow))
                break;  // given up
            const double b = has ? __ldcg(reinterpret_cast<const double*>(A.sorted_b + k) + axis) : 0.0;
            const double w1 = wrap_axis(ax.L, ax.invL, dadd(b, x));  // W1 = wrap(propose(..))
            const bool inside = axis_in_space(ax.origin, ax.width, ax.invW, ax.shape, ma, w1);
            ta = wrap_axis(ax.L, ax.invL, w1);
            const unsigned in = __ballot_sync(full, inside);
            valid = valid && (in & mine) == mine;
            // a trial that leaves its space is rejected whatever lies around
            if (has && !valid && row == 0) store_release(A.progress + cell, round + 1u);
            if (!__any_sync(full, valid)) continue;
        }
        double t[3] = {__shfl_sync(full, ta, head), __shfl_sync(full, ta, head + 1u),
                       DIM == 3 ? __shfl_sync(full, ta, head + 2u) : 0.0};
        float4 t32 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (FP32) {
            const float o = offset_axis(ax.L, ax.origin, ax.width, ma, ta);
            t32 = make_float4(__shfl_sync(full, o, head), __shfl_sync(full, o, head + 1u),
                              DIM == 3 ? __shfl_sync(full, o, head + 2u) : 0.f, 0.f);
        }
        if (!INJ) {
            // the neighbours' progress (an empty space's is never waited for)
            unsigned pending = 0;
#pragma unroll
            for (int i = 0; i < SP; ++i)
                if (valid && R.end[i] > R.start[i] && R.need[i] > f.r0) pending |= 1u << i;
            if (!sphere_wait<SP>(A.progress, R.cell, R.need, pending, A.stats, L.flow)) break;  // given up
        }
        // the first site of each space
        const Site* sites = FP32 ? reinterpret_cast<const Site*>(A.sorted_off) : reinterpret_cast<const Site*>(A.sorted_s);
        Site v[SP];
#pragma unroll
        for (int i = 0; i < SP; ++i)
            if (valid && R.end[i] > R.start[i]) v[i] = ldcg_site(sites + R.start[i]);
        bool hit = false, near = false;
        if (valid) {
#pragma unroll
            for (int i = 0; i < SP; ++i) {
                Site s = v[i];
                for (uint32_t q = R.start[i]; q < R.end[i];) {
                    if (q != k) {
                        st.checks++;
                        if constexpr (FP32) {
                            const float s0 = (float)R.d0 * g.w32[0], s1 = DIM == 3 ? (float)R.d1 * g.w32[1] : 0.f;
                            const float d2 = fp32_dist2<DIM>(g, t32, s, s0, s1, DIM == 3 ? i - 1 : R.d1);
                            hit |= d2 < P.sig2_lo32;
                            if (d2 >= P.sig2_lo32 && d2 < P.sig2_hi32) {
                                near = true;
                                const double r2 = sphere_dist2_fp64<DIM>(g, A.sorted_b, t[0], t[1], t[2], q);
                                const double err = fabs((double)d2 - r2);
                                st.rechecks++;
                                st.max_err = err > st.max_err ? err : st.max_err;
                                hit |= r2 < P.sigma2;
                            }
                        } else {
                            const double sv[3] = {s.x, s.y, s.z};
                            hit |= ref_dist2<DIM>(g, t, sv) < P.sigma2;
                        }
                    }
                    if (hit || ++q >= R.end[i]) break;
                    s = ldcg_site(sites + q);
                }
            }
        }
        const unsigned hits = __ballot_sync(full, hit);
        const bool clear = valid && (hits & mine) == 0u;
        if constexpr (INJ) {
            const unsigned checked = __ballot_sync(full, near) & mine;
            const uint32_t i = unit * kTrials + trial;
            if (trial < kTrials && i < J.n && row == 0) {
                J.decisions[i] = clear;
                J.flags[i] = flag | (checked ? kTrialRechecked : 0);
            }
        } else {
            // update_body_properties: body = wrap(W1) = T, site = wrap(body)
            if (clear && row < (uint32_t)DIM) {
                reinterpret_cast<double*>(A.sorted_b + k)[axis] = ta;
                reinterpret_cast<double*>(A.body_pos + __ldg(A.sorted_body + k))[axis] = ta;
                const double sv = wrap_axis(ax.L, ax.invL, ta);
                if (FP32)
                    reinterpret_cast<float*>(A.sorted_off + k)[axis] = offset_axis(ax.L, ax.origin, ax.width, ma, sv);
                else
                    reinterpret_cast<double*>(A.sorted_s + k)[axis] = sv;
            }
            n_accepted += clear && row == 0;
            __syncwarp();
            if (valid && row == 0) store_release(A.progress + cell, round + 1u);
        }
    }
    flush_stats(A.stats, st, n_accepted);
}

template <int DIM, bool FP32>
using FlowSphere = void (*)(Geometry, Arrays, Pair, Launch, Injected);

template <int DIM, bool FP32>
cudaError_t launch(const Geometry& g, const Arrays& a, const Pair& p, const Launch& l, cudaStream_t s,
                   uint32_t variant) {
    // the draws: a thread per trial of two colour sets, at most one resident wave
    const auto d = k_draw_sphere<DIM>;
    const uint64_t per_set = (uint64_t)g.color_stride << DIM, wave_d = (uint64_t)resident_wave((const void*)d);
    uint64_t blocks = (2u * per_set + 127u) / 128u;
    PassLaunch pd((uint32_t)(blocks < wave_d ? blocks : wave_d), l.overlap_previous != 0, s);
    cudaError_t e = cudaLaunchKernelEx(&pd.cfg, d, g, a, l);
    if (e != cudaSuccess) return e;
    // the compiled launch variants, in the order of kSphereFlowShapes
    static constexpr FlowSphere<DIM, FP32> kernels[] = {k_flow_sphere<DIM, FP32, false, 4>,
                                                        k_flow_sphere<DIM, FP32, false, 6>};
    static_assert(n_shapes(kSphereFlowShapes) == 2, "a kernel per variant");
    const auto k = kernels[variant < 2 ? variant : 0];
    // warps for the trials of two colours, at most one resident wave
    blocks = ((uint64_t)g.color_stride * 2u + 4u * kTrials - 1u) / (4u * kTrials);
    const uint64_t wave = (uint64_t)resident_wave((const void*)k);
    PassLaunch pl((uint32_t)(blocks < wave ? blocks : wave), l.overlap_previous != 0, s);
    return cudaLaunchKernelEx(&pl.cfg, k, g, a, p, l, Injected{});
}

}  // namespace

cudaError_t launch_flow_sphere(int dim, bool fp32, const Geometry& g, const Arrays& a, const Pair& p, const Launch& l,
                               cudaStream_t s, uint32_t variant) {
    if (l.n_active == 0) return cudaSuccess;
    if (dim == 2) return fp32 ? launch<2, true>(g, a, p, l, s, variant) : launch<2, false>(g, a, p, l, s, variant);
    return fp32 ? launch<3, true>(g, a, p, l, s, variant) : launch<3, false>(g, a, p, l, s, variant);
}

cudaError_t launch_flow_trials_sphere(int dim, bool fp32, const Geometry& g, const Arrays& a, const Pair& p,
                                      const Injected& j, cudaStream_t s) {
    if (j.n == 0) return cudaSuccess;
    const auto k = dim == 2 ? (fp32 ? k_flow_sphere<2, true, true, 4> : k_flow_sphere<2, false, true, 4>)
                            : (fp32 ? k_flow_sphere<3, true, true, 4> : k_flow_sphere<3, false, true, 4>);
    k<<<(j.n + 4u * kTrials - 1u) / (4u * kTrials), 128, 0, s>>>(g, a, p, Launch{}, j);
    return cudaGetLastError();
}

}  // namespace hmc
