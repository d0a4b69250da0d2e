// Dataflow order of a sweep's trials: one launch runs every colour pass of a range of colour sets.
//
// A colour pass per launch waits for its slowest trial before the next colour starts, and the
// passes that give a trial a warp hold too few trials to hide that (2^19 Lennard-Jones sites:
// 112 passes of 4,913 trials, 26 us each, the SMs issuing 36 % of the cycles). But a trial
// depends only on the 3^d spaces around its own: it needs the moves of the colours before its
// own from this colour set, and of the others from the one before. So the trials are numbered
// in the passes' order (colour set, colour, list entry), warps take the numbers in that order
// (an atomic ticket), and a warp waits only for the spaces around its trial: progress[space]
// counts the colour sets that the space has finished. Every trial sees the sites that it would
// see in the pass order, so the trajectory is the same.
//
// Every wait ends: a trial waits only for trials with smaller numbers, each of which a running
// warp holds or has finished (a warp takes the next number while it works on its present one, but
// works in number order), so the smallest unfinished trial never waits. The waits carry a time
// limit all the same (FlowLimit): a warp whose wait runs out raises kErrFlowTimeout and gives its trial
// up undecided, the others stop at their next wait, and the state is left with part of the sweep done.
//
// Memory order: sites that the launch changes are read through L2 (ld.global.cg; an L1 line could
// be stale) after an acquire of the neighbours' progress, and written before a release of the own.
#pragma once

#include <cuda_runtime.h>

#include "hmc_device.cuh"

namespace hmc {

// The colour sets [r0, r1) one launch runs, and where its trials stand: trial number e is entry e of
// the draws (k_draw_*: what the trial's random stream gives, which depends on no site). A kernel
// whose warps take several trials at a time takes units of `group` trials of one colour, numbered
// in the same order (trials of two colours may touch and cannot wait for one another in one warp).
struct FlowRange {
    uint32_t r0, r1;
    uint32_t count[8];   // trials of colour c in one colour set
    uint32_t prefix[8];  // of the colours before c
    uint32_t per_set;    // of one colour set
    uint32_t n;          // of the range
    uint32_t unit_prefix[8], units_per_set, n_units;
};

__device__ __forceinline__ FlowRange flow_range(const DeviceStats* st, uint32_t round, uint32_t round_end,
                                                uint32_t colors, uint32_t group = 1) {
    FlowRange f;
    f.r0 = round;
    f.r1 = min(round_end, st->rounds);
    f.per_set = f.units_per_set = 0;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
        f.prefix[c] = f.per_set;
        f.unit_prefix[c] = f.units_per_set;
        f.count[c] = c < colors ? st->color_count[c] : 0u;
        f.per_set += f.count[c];
        f.units_per_set += (f.count[c] + group - 1u) / group;
    }
    const uint32_t sets = st->error_flags != 0u || f.r1 <= f.r0 ? 0u : f.r1 - f.r0;
    f.n = sets * f.per_set;
    f.n_units = sets * f.units_per_set;
    return f;
}

// Number e in a range with these prefixes: its colour set (absolute), colour and place in the colour.
__device__ __forceinline__ void flow_place(uint32_t r0, const uint32_t* prefix, uint32_t per_set, uint32_t e,
                                           uint32_t& round, uint32_t& color, uint32_t& entry) {
    const uint32_t s = e / per_set, rem = e - s * per_set;
    round = r0 + s;
    color = 0;
    entry = rem;
#pragma unroll
    for (uint32_t c = 1; c < 8; ++c)
        if (rem >= prefix[c] && prefix[c] < per_set) {
            color = c;
            entry = rem - prefix[c];
        }
}
__device__ __forceinline__ void flow_item(const FlowRange& f, uint32_t e, uint32_t& round, uint32_t& color,
                                          uint32_t& entry) {
    flow_place(f.r0, f.prefix, f.per_set, e, round, color, entry);
}
__device__ __forceinline__ void flow_unit(const FlowRange& f, uint32_t u, uint32_t& round, uint32_t& color,
                                          uint32_t& entry) {
    flow_place(f.r0, f.unit_prefix, f.units_per_set, u, round, color, entry);
}

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Read of a value that the running launch may have changed on another SM.
__device__ __forceinline__ double4 ldcg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldcg(q), b = __ldcg(q + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Neighbour space `lane` (< 3^DIM) of space m of colour `color`, and the progress a trial of
// colour set `round` needs there: round + 1 of the colours before its own (they move first within
// a colour set), round of the others and of its own space.
template <int DIM>
__device__ __forceinline__ void flow_need(const Geometry& g, const uint32_t* m, uint32_t color, uint32_t round,
                                          uint32_t lane, uint32_t& space, uint32_t& need) {
    uint32_t v = lane, n[3] = {0, 0, 0}, c = 0;
    int d[3];
#pragma unroll
    for (int a = DIM - 1; a >= 0; --a) {
        d[a] = (int)(v % 3u) - 1;
        v /= 3u;
    }
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
        n[a] = wrap_index((int)m[a] + d[a], g.shape[a]);
        c = (c << 1) | (n[a] & 1u);
    }
    space = cell_index<DIM>(g, n);
    need = round + (c < color ? 1u : 0u);
}

// The place in a colour's list of `count` spaces that the `entry`-th trial of the colour takes in
// colour set `round`. The lists are sorted by space, slowest axis first, so trials started close
// together lie in one slab of the box and need the slabs around it that the colour before has just
// left, except at the list's two ends, which touch across the periodic boundary: the first trials
// of a colour would wait for the last of the colour before. Every colour therefore starts two
// spaces of the slow axis (one of its own planes) further on than the colour before.
__device__ __forceinline__ uint32_t flow_rotated(uint32_t count, uint32_t round, uint32_t color,
                                                 uint32_t colors, uint32_t planes, uint32_t entry) {
    const uint32_t level = (round * colors + color) % (planes / 2u);  // planes is even
    const uint32_t shift = (uint32_t)((uint64_t)count * level / (planes / 2u));
    const uint32_t e = entry + shift;
    return e >= count ? e - count : e;
}

// Poll a lane's progress word until it reaches `need` (ok: it has) in every lane of `lanes`. False:
// the launch is given up (another warp's or this one's time limit).
__device__ __forceinline__ bool flow_wait(const uint32_t* word, uint32_t need, unsigned lanes, bool& ok,
                                          DeviceStats* stats, const FlowLimit& limit) {
    const unsigned full = 0xffffffffu;
    unsigned long long t0 = 0;
    for (uint32_t spins = 0;; ++spins) {
        if (!ok) ok = load_acquire(word) >= need;
        if ((__ballot_sync(full, ok) & lanes) == lanes) return true;
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

// The same for lanes with up to N words each (bit i of pending: word words[first + i * stride] is
// still short): returns once no lane has a pending word among those of `mask`.
template <uint32_t N>
__device__ __forceinline__ bool flow_wait_words(const uint32_t* progress, const uint2* words, uint32_t first,
                                           uint32_t stride, unsigned& pending, unsigned mask, DeviceStats* stats,
                                           const FlowLimit& limit) {
    const unsigned full = 0xffffffffu;
    unsigned long long t0 = 0;
    for (uint32_t spins = 0;; ++spins) {
        uint32_t v[N], need[N];
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            v[i] = need[i] = 0;
            if ((pending >> i) & 1u) {
                const uint2 w = words[first + i * stride];
                need[i] = w.y;
                v[i] = load_acquire(progress + w.x);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < N; ++i)
            if (v[i] >= need[i]) pending &= ~(1u << i);
        if (!__any_sync(full, (pending & mask) != 0u)) return true;
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

// ---- staging by bulk copies ------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Copy `bytes` (a multiple of 16, both addresses 16-byte aligned) and count them on the barrier.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Orders the generic proxy's view of global memory (sites that other SMs have written and this
// thread has acquired) before the bulk copies that follow.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ bool mbar_try(unsigned long long* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0u;
}
// Wait for the barrier's phase of the given parity. Where the copies do not arrive within the limit `lost`
// is set, and the caller gives the trial up; the barrier is then waited for once more as long, since the
// block's shared memory must not be given back while copies into it are on their way.
static __device__ __noinline__ void mbar_wait_long(unsigned long long* bar, uint32_t parity, DeviceStats* stats,
                                                   unsigned long long wait_ns, uint32_t* lost) {
    unsigned long long t0 = global_ns();
    bool late = false;
    while (!mbar_try(bar, parity)) {
        const unsigned long long now = global_ns();
        if (now - t0 <= wait_ns) continue;
        if (late) return;
        atomicOr(&stats->error_flags, kErrFlowTimeout);
        *lost = 1u;
        late = true;
        t0 = now;
    }
}
__device__ __forceinline__ void mbar_wait(unsigned long long* bar, uint32_t parity, DeviceStats* stats,
                                          const FlowLimit& limit, uint32_t* lost) {
    for (uint32_t i = 0; i < 16u; ++i)  // (a try suspends the warp for a while)
        if (mbar_try(bar, parity)) return;
    mbar_wait_long(bar, parity, stats, limit.wait_ns, lost);
}

// One axis of wrap_inv, point_to_space and cell_offsets: the lanes of a warp that share a trial
// take an axis each.
__device__ __forceinline__ double wrap_axis(double L, double invL, double x) {
    double lam = div_fixed(x, L, invL);
    lam = dsub(lam, round(lam));
    if (lam == 0.5) lam = -0.5;
    return dmul(lam, L);
}
// Whether x lies in space m of the axis (point_to_space's index equals m).
__device__ __forceinline__ bool axis_in_space(double origin, double width, double invW, uint32_t shape, uint32_t m,
                                              double x) {
    const double f = floor(div_fixed(dsub(x, origin), width, invW));
    if (!(f >= 0.0) || f > 4.0e9) return false;
    uint32_t idx = (uint32_t)f;
    if (idx == shape) idx = 0;
    return idx == m;
}
__device__ __forceinline__ float offset_axis(double L, double origin, double width, uint32_t m, double s) {
    double off = dsub(dsub(s, origin), dmul((double)m, width));
    if (off > 1.5 * width)
        off = dsub(off, L);
    else if (off < -0.5 * width)
        off = dadd(off, L);
    return __double2float_rn(off);
}

// The box and checkerboard of one axis.
struct AxisGeometry {
    double L, invL, origin, width, invW;
    uint32_t shape;
};
template <int DIM>
__device__ __forceinline__ AxisGeometry axis_geometry(const Geometry& g, uint32_t a) {
    return {g.L[a], g.invL[a], g.origin[a], g.width[a], g.invW[a], g.shape[a]};
}

}  // namespace hmc
