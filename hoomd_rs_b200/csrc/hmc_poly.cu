// Hard convex polyhedra: PairwiseCutoff<HardShape<Convex<ConvexPolyhedron>>> with
// Translate<Cartesian<3>> and Rotate<Versor> trial moves.
//
// The pair test is Convex::intersects_at_global (hoomd-geometry/src/convex.rs:154-170): a
// circumsphere rejection, pair_system_to_local (hoomd-vector/src/lib.rs:878-888) and
// XenoCollide / Minkowski portal refinement (hoomd-geometry/src/xenocollide.rs:172-414) over
// the support function of the vertex table (shape/convex_polytope.rs:222-244). Every
// product, sum and fused multiply-add below follows the reference's expression order, so
// the FP64 decision is the reference's.
//
// The sweep gives a warp four trials (k_flow_poly3): each group of 8 lanes computes its trial and
// prefilters its candidates by circumsphere, and the warp runs the full tests of all four trials'
// remaining candidates together. Injected moves (k_eval_poly3) take
// one warp per move and the stencil's candidates 32 at a time, with an early exit by vote.
// FP32 + recheck: a candidate whose FP32 centre distance clears the circumsphere by more
// than the FP32 error bound is skipped; every other candidate runs the FP64 test, so the
// decisions equal the FP64 pass.
#include <cuda_runtime.h>

#include <type_traits>

#include "hmc_flow.cuh"
#include "hmc_serial.cuh"

namespace hmc {
namespace {

struct Q {
    double s, x, y, z;
};
struct V3 {
    double x, y, z;
};

__device__ __forceinline__ double dot3(const V3& a, const V3& b) {  // mul_add fold from 0.0
    return dfma(a.z, b.z, dfma(a.y, b.y, dfma(a.x, b.x, 0.0)));
}
__device__ __forceinline__ V3 cross3(const V3& a, const V3& b) {  // cartesian.rs:604-610
    return {dsub(dmul(a.y, b.z), dmul(a.z, b.y)), dsub(dmul(a.z, b.x), dmul(a.x, b.z)),
            dsub(dmul(a.x, b.y), dmul(a.y, b.x))};
}
__device__ __forceinline__ V3 sub3(const V3& a, const V3& b) { return {dsub(a.x, b.x), dsub(a.y, b.y), dsub(a.z, b.z)}; }
__device__ __forceinline__ V3 neg3(const V3& a) { return {-a.x, -a.y, -a.z}; }

// Quaternion::mul (quaternion.rs:408-415).
__device__ __forceinline__ Q qmul(const Q& a, const Q& b) {
    const V3 av{a.x, a.y, a.z}, bv{b.x, b.y, b.z};
    const double sc = dsub(dmul(a.s, b.s), dot3(av, bv));
    const V3 c = cross3(av, bv);
    return {sc, dadd(dadd(dmul(bv.x, a.s), dmul(av.x, b.s)), c.x), dadd(dadd(dmul(bv.y, a.s), dmul(av.y, b.s)), c.y),
            dadd(dadd(dmul(bv.z, a.s), dmul(av.z, b.s)), c.z)};
}
// Versor::rotate (quaternion.rs:740-747).
__device__ __forceinline__ V3 vrotate(const Q& q, const V3& v) {
    const V3 qv{q.x, q.y, q.z};
    const double k1 = dsub(dmul(q.s, q.s), dot3(qv, qv));
    const V3 c = cross3(qv, v);
    const double k2 = dmul(2.0, q.s);
    const double k3 = dmul(2.0, dot3(qv, v));
    return {dadd(dadd(dmul(v.x, k1), dmul(c.x, k2)), dmul(qv.x, k3)),
            dadd(dadd(dmul(v.y, k1), dmul(c.y, k2)), dmul(qv.y, k3)),
            dadd(dadd(dmul(v.z, k1), dmul(c.z, k2)), dmul(qv.z, k3))};
}

struct M3 {
    V3 r[3];
};
// RotationMatrix::from(Versor) (quaternion.rs:642-690).
__device__ __forceinline__ M3 mat_from(const Q& q) {
    const double a = q.s, b = q.x, c = q.y, d = q.z;
    M3 m;
    m.r[0] = {dsub(dsub(dadd(dmul(a, a), dmul(b, b)), dmul(c, c)), dmul(d, d)),
              dsub(dmul(dmul(2.0, b), c), dmul(dmul(2.0, a), d)), dadd(dmul(dmul(2.0, b), d), dmul(dmul(2.0, a), c))};
    m.r[1] = {dadd(dmul(dmul(2.0, b), c), dmul(dmul(2.0, a), d)),
              dsub(dadd(dsub(dmul(a, a), dmul(b, b)), dmul(c, c)), dmul(d, d)),
              dsub(dmul(dmul(2.0, c), d), dmul(dmul(2.0, a), b))};
    m.r[2] = {dsub(dmul(dmul(2.0, b), d), dmul(dmul(2.0, a), c)), dadd(dmul(dmul(2.0, c), d), dmul(dmul(2.0, a), b)),
              dadd(dsub(dsub(dmul(a, a), dmul(b, b)), dmul(c, c)), dmul(d, d))};
    return m;
}
__device__ __forceinline__ V3 mat_rotate(const M3& m, const V3& v) {
    return {dot3(m.r[0], v), dot3(m.r[1], v), dot3(m.r[2], v)};
}
__device__ __forceinline__ M3 transpose(const M3& m) {
    return {{{m.r[0].x, m.r[1].x, m.r[2].x}, {m.r[0].y, m.r[1].y, m.r[2].y}, {m.r[0].z, m.r[1].z, m.r[2].z}}};
}

// ConvexPolytope::support_mapping: argmax of ((v0 n0) + v1 n1) + v2 n2, first maximum wins.
// Unrolled by four so that the vertex loads of several iterations are in flight together (the
// comparisons stay in order). For cubes this measured the same as rolled (1.69e8 trial moves/s,
// FP32), for the 2-D squares' support2 +3 %; a shared-memory copy of the table gained nothing.
__device__ __forceinline__ V3 support(const double4* __restrict__ verts, uint32_t nv, const V3& n) {
    uint32_t arg = 0;
    double best = -INFINITY;
#pragma unroll 4
    for (uint32_t i = 0; i < nv; ++i) {
        const double4 v = ldg4(verts + i);
        const double x = dadd(dadd(dmul(v.x, n.x), dmul(v.y, n.y)), dmul(v.z, n.z));
        if (x > best) {
            best = x;
            arg = i;
        }
    }
    const double4 v = ldg4(verts + arg);
    return {v.x, v.y, v.z};
}

struct Minkowski {
    const double4* verts;
    uint32_t nv;
    V3 vij;
    M3 q, qinv;
    // composite_support_mapping (xenocollide.rs:318-328)
    __device__ __forceinline__ V3 operator()(const V3& n) const {
        const V3 sb = support(verts, nv, mat_rotate(qinv, n));
        V3 r = mat_rotate(q, sb);
        r = {dadd(r.x, vij.x), dadd(r.y, vij.y), dadd(r.z, vij.z)};
        const V3 sa = support(verts, nv, neg3(n));
        return sub3(r, sa);
    }
};

constexpr int kXenoMaxIter = 1024;  // xenocollide.rs:38

// collide for N = 3 (xenocollide.rs:172-291, :361-414). The iteration caps return overlap,
// as the reference does.
__device__ __noinline__ bool collide3d(const double4* verts, uint32_t nv, const V3& vij, const Q& oij) {
    Minkowski s;
    s.verts = verts;
    s.nv = nv;
    s.vij = vij;
    s.q = mat_from(oij);
    s.qinv = transpose(s.q);
    const double TOL = 2e-12;
    const V3 v0 = vij;
    if (fabs(v0.x) < TOL && fabs(v0.y) < TOL && fabs(v0.z) < TOL) return true;
    V3 v1 = s(neg3(v0));
    if (dot3(v1, v0) > 0.0) return false;
    V3 n = cross3(v1, v0);
    if (fabs(n.x) < TOL && fabs(n.y) < TOL && fabs(n.z) < TOL) return true;
    V3 v2 = s(n);
    if (dot3(v2, n) < 0.0) return false;
    n = cross3(sub3(v1, v0), sub3(v2, v0));
    if (dot3(n, v0) > 0.0) {
        const V3 t = v1;
        v1 = v2;
        v2 = t;
        n = neg3(n);
    }
    V3 v3;
    for (int count = 1;; ++count) {
        if (count >= kXenoMaxIter) return true;
        v3 = s(n);
        if (dot3(v3, n) <= 0.0) return false;
        if (dot3(cross3(v1, v3), v0) < 0.0) {
            v2 = v3;
            n = cross3(sub3(v1, v0), sub3(v2, v0));
            continue;
        }
        if (dot3(cross3(v3, v2), v0) < 0.0) {
            v1 = v3;
            n = cross3(sub3(v1, v0), sub3(v2, v0));
            continue;
        }
        break;
    }
    V3 p0 = v1, p1 = v2, p2 = v3;
    for (int count = 1;; ++count) {
        V3 nn = cross3(sub3(p1, p0), sub3(p2, p0));
        if (dot3(sub3(p0, v0), nn) < 0.0) nn = neg3(nn);
        if (dot3(p0, nn) >= 0.0) return true;
        const V3 vn = s(nn);
        if (dot3(vn, nn) < 0.0) return false;
        const double tol = dmul(TOL, dsqrt(dot3(nn, nn)));
        if (fabs(dot3(sub3(vn, p0), nn)) < tol) return false;
        if (fabs(dot3(p0, nn)) < tol) return true;
        const V3 vp = cross3(vn, v0);
        const bool t1 = dot3(vp, p0) > 0.0, t2 = dot3(vp, p1) > 0.0, t3 = dot3(vp, p2) > 0.0;
        if (t1 && t2)
            p0 = vn;
        else if (t1 && !t2)
            p2 = vn;
        else if (!t1 && t3)
            p1 = vn;
        else
            p0 = vn;
        if (count >= kXenoMaxIter) return true;
    }
}

// Trial site t (position) with versor qi against the site of slot q (position S via the image
// rule, versor sorted_q[q]): HardShape::site_pair_energy -> intersects_at_global.
__device__ __forceinline__ bool poly_overlap64(const Geometry& g, const Arrays& A, const double4* verts, uint32_t nv,
                                               double rcut2, const double* t, const Q& qi, const double* sj, uint32_t q) {
    double d[3];
    const double d2 = ref_disp<3>(g, t, sj, d);
    if (d2 >= rcut2) return false;  // r_self.distance_squared(r_other) >= r_cut^2
    const V3 rab{-d[0], -d[1], -d[2]};  // image - t, exactly -(t - image)
    const double4 o4 = ldg4(A.sorted_q + q);
    const Q qj{o4.x, o4.y, o4.z, o4.w};
    const Q ia{qi.s, -qi.x, -qi.y, -qi.z};  // Versor::inverted = conjugate
    const V3 vij = vrotate(ia, rab);
    const Q oij = qmul(ia, qj);
    return collide3d(verts, nv, vij, oij);
}

// Rotate<Versor>::propose (rotate/versor.rs:40-71, 112-123): Gaussian rotation vector with
// standard deviation sigma, rejected beyond pi, lifted by the exponential map (versor_draw), composed
// in front of the current orientation.
__device__ __forceinline__ Q versor_draw(Sfc64& rng, double sigma, const double* zx, const double* zf) {
    for (;;) {
        double s0 = dadd(0.0, dmul(sigma, standard_normal(rng, zx, zf)));
        double s1 = dadd(0.0, dmul(sigma, standard_normal(rng, zx, zf)));
        double s2 = dadd(0.0, dmul(sigma, standard_normal(rng, zx, zf)));
        const V3 sv{s0, s1, s2};
        const double theta = dsqrt(dot3(sv, sv));
        if (theta > 3.141592653589793) continue;
        double sh, ch;
        portable_sincos(dmul(0.5, theta), &sh, &ch);
        double vf = ddiv(sh, theta);
        if (!isfinite(vf)) vf = 0.5;
        return Q{ch, dmul(s0, vf), dmul(s1, vf), dmul(s2, vf)};
    }
}
__device__ __forceinline__ Q versor_move(Sfc64& rng, double sigma, const double* zx, const double* zf, const Q& q) {
    return qmul(versor_draw(rng, sigma, zx, zf), q);
}

struct PolyShape {
    const double4* verts;
    uint32_t nv;
    double rcut2;     // (R_a + R_b)^2
    float rcut2_hi32; // FP32 threshold: at or above this, outside the circumsphere for certain
    float site_err;   // per-axis error of a displacement of fixed-point sites beyond its FP32 roundings
    float bound_scale;  // widens the FP32 bounds of the pair tests (1; tests: HMC_B200_FP32_BAND_SCALE)
};

__device__ __forceinline__ bool warp_any(bool v) { return __any_sync(0xffffffffu, v); }

// Overlap of the trial (t, qi; fixed-point site t32) with any candidate of the stencil fs,
// skipping slot self (injected moves, the tuner). The warp takes the stencil's candidates 32 at a
// time across its rows, and a vote after each step stops the warp at the first overlap. FP32: the
// circumsphere prefilter in FP32 under the bound.
template <bool FP32>
__device__ __forceinline__ bool poly_overlaps(const Geometry& g, const Arrays& A, const PolyShape& sh, const double* t,
                                              const Q& qi, const int4& t32, const FlatStencil& fs, uint32_t self,
                                              uint32_t lane, PairStats& st) {
#pragma unroll 1
    for (uint32_t j0 = 0; j0 < fs.total; j0 += 32) {
        const uint32_t j = j0 + lane;
        uint32_t part;
        const uint32_t q = flat_slot(fs, j, part);
        bool hit = false;
        if (j < fs.total && q != self) {
            bool test = true;
            st.checks++;
            if (FP32) {
                test = fixed_dist2<3>(g, t32, __ldg(reinterpret_cast<const int4*>(A.sorted_off) + q)) < sh.rcut2_hi32;
                if (test) st.rechecks++;
            }
            if (test) {
                // shapes keep S in both precision modes (the FP32 pass only prefilters)
                const double4 s4 = ldg4(A.sorted_s + q);
                const double sj[3] = {s4.x, s4.y, s4.z};
                hit = poly_overlap64(g, A, sh.verts, sh.nv, sh.rcut2, t, qi, sj, q);
            }
        }
        if (warp_any(hit)) return true;
    }
    return false;
}

// A round's trial moves of convex polyhedra under the approximate overlap for every colour list
// (generate_trial_moves, parallel_sweep.rs:231-278, up to delta_energy_one), one thread per trial: the
// chosen body, Translate (Ball::sample) or Rotate<Versor>, W1 = wrap(propose(..)), the space check, the
// trial site T = wrap(W1) and the Metropolis uniform; k_sweep_poly3_soft, which gives a trial a warp, reads
// them instead of computing each move in 32 lanes.
__global__ void __launch_bounds__(128) k_propose_poly3(Geometry g, Arrays A, Launch L, uint32_t rotate) {
    const DeviceStats* st = A.stats;
    if (st->error_flags != 0u || L.round >= st->rounds) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 8u * g.color_stride; i += gridDim.x * blockDim.x) {
        const uint32_t c = i / g.color_stride, w = i - c * g.color_stride;
        if (w >= st->color_count[c]) continue;
        uint32_t m[3] = {0, 0, 0};
        unpack_m<3>(__ldg(A.color_cells + i), m);
        const uint32_t cell = cell_index<3>(g, m);
        const uint32_t start = __ldg(A.cell_start + cell);
        const uint32_t count = __ldg(A.cell_start + cell + 1) - start;
        Sfc64 rng = make_rng(L.step, L.substep, L.seed, (uint64_t)cell);
        const uint32_t k = start + canon_range_u32(rng, count);
        const double4 b4 = A.sorted_b[k];
        double x[3] = {b4.x, b4.y, b4.z};
        const double4 q4 = A.sorted_q[k];
        Q qi{q4.x, q4.y, q4.z, q4.w};
        if (rotate) {
            qi = versor_move(rng, L.max_move, A.zig_x, A.zig_f, qi);
        } else {
            double dv[3];
            ball_sample<3>(rng, L.max_move, A.zig_x, A.zig_f, dv);
            for (int a = 0; a < 3; ++a) x[a] = dadd(x[a], dv[a]);
        }
        const double u = uniform01(rng);  // the Metropolis uniform, the stream's next draw after the move
        wrap_inv<3>(g.L, g.invL, x);  // W1 = wrap(propose(..))
        uint32_t mt[3];
        if (!(point_to_space<3>(g, x, mt) && cell_index<3>(g, mt) == cell)) {
            A.trial_k[i] = kNoTrial;
            continue;
        }
        double t[3] = {x[0], x[1], x[2]};
        wrap_inv<3>(g.L, g.invL, t);
        A.trial_t[i] = make_double4(t[0], t[1], t[2], u);
        A.trial_q[i] = make_double4(qi.s, qi.x, qi.y, qi.z);
        A.trial_k[i] = k;
    }
}

// ---- the sweep --------------------------------------------------------------------------------
// What the random streams of the trials of colour sets [L.round, L.round_end) give, one thread per
// trial (generate_trial_moves, parallel_sweep.rs:231-278): the chosen body's slot and space in
// draw_i, and in draw_d the displacement (Ball::sample) or the rotation's versor (Rotate<Versor>), which
// depend on no site. Each space's progress is set to the first colour set; the ticket starts at 0.
__global__ void __launch_bounds__(128) k_draw_poly3(Geometry g, Arrays A, Launch L, uint32_t rotate) {
    grid_dependency_wait();
    allow_dependent_launch();
    const FlowRange f = flow_range(A.stats, L.round, L.round_end, 8);
    if (blockIdx.x == 0 && threadIdx.x == 0) A.stats->ticket = L.flow.stall == kStallTrial ? 1u : 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += gridDim.x * blockDim.x) {
        uint32_t round, color, entry;
        flow_item(f, i, round, color, entry);
        entry = flow_rotated(A.stats->color_count[color], round, color, 8, g.shape[0], entry);
        const uint32_t packed = __ldg(A.color_cells + (size_t)color * g.color_stride + entry);
        uint32_t m[3];
        unpack_m<3>(packed, m);
        const uint32_t cell = cell_index<3>(g, m);
        if (round == f.r0) A.progress[cell] = f.r0;
        const uint32_t start = __ldg(A.cell_start + cell);
        const uint32_t count = __ldg(A.cell_start + cell + 1) - start;
        Sfc64 rng = make_rng(L.step, L.substep + round, L.seed, (uint64_t)cell);
        const uint32_t k = start + canon_range_u32(rng, count);
        double4 d;
        if (rotate) {
            const Q dq = versor_draw(rng, L.max_move, A.zig_x, A.zig_f);
            d = make_double4(dq.s, dq.x, dq.y, dq.z);
        } else {
            double dv[3];
            ball_sample<3>(rng, L.max_move, A.zig_x, A.zig_f, dv);
            d = make_double4(dv[0], dv[1], dv[2], 0.0);
        }
        A.draw_d[i] = d;
        A.draw_i[i] = make_uint4(k, packed, 0u, 0u);
    }
}

// The shape's vertices in a block's shared memory: FP64 for the support mapping's values, FP32 to
// find which vertex it is, with the largest coordinate.
struct ShapeTable {
    float4 v32[32];
    double v[32][3];
    uint32_t nv;
    float vmax;
    float bound_scale;  // PolyShape's
};

// ConvexPolytope::support_mapping (support above): which vertex has the first maximum of ((v0 n0) + v1
// n1) + v2 n2.
__device__ __noinline__ uint32_t support64(const ShapeTable& T, V3 n) {
    uint32_t arg = 0;
    double best = -INFINITY;
    for (uint32_t i = 0; i < T.nv; ++i) {
        const double x = dadd(dadd(dmul(T.v[i][0], n.x), dmul(T.v[i][1], n.y)), dmul(T.v[i][2], n.z));
        if (x > best) {
            best = x;
            arg = i;
        }
    }
    return arg;
}

// One pair test in steps: XenoCollide (collide3d) written so that every step is one composite support
// mapping followed by the little that depends on the phase; the lanes of a warp then share the
// support mappings, which are nearly all of the work, whatever phase each is in.
struct PairLane {
    V3 v0, p0, p1, p2, n;  // v0; the portal; the direction of the next support mapping
    M3 q;                  // orientation of the other shape in the trial's frame
    uint32_t phase, count;
};

// composite_support_mapping (xenocollide.rs:318-328) in direction n by the two lanes of a pair test:
// role 0 finds the trial shape's vertex in direction -n, role 1 the other's in direction q^T n.
// FP32: the vertex is looked for in FP32 first: with |v_a| <= vmax, vertices and the components of the
// direction d that is searched rounded once and three roundings per sum, a product is off by at most
// 6 u32 vmax |d|_1, so a maximum ahead of the runner-up by more than 64 u32 vmax |d|_1 is the FP64
// maximum too (also where d = q^T n of a versor that is not of unit length is longer than n); else (ties, as along the edges of a portal) the FP64
// products decide. FP32 takes 8 instructions per vertex against 17 (FP64 issues at half rate).
template <bool FP32>
__device__ __forceinline__ V3 pair_support(const ShapeTable& T, const M3& q, const V3& vij, const V3& n, uint32_t role,
                                           unsigned active) {
    const V3 dir = role ? mat_rotate(transpose(q), n) : neg3(n);
    uint32_t mine = 0;
    if constexpr (FP32) {
        const float x = (float)dir.x, y = (float)dir.y, z = (float)dir.z;
        float first = -INFINITY, second = -INFINITY;
#pragma unroll 4
        for (uint32_t i = 0; i < T.nv; ++i) {
            const float4 v = T.v32[i];
            const float p = v.x * x + v.y * y + v.z * z;
            second = fmaxf(second, fminf(first, p));
            mine = p > first ? i : mine;
            first = fmaxf(first, p);
        }
        const float gap = 64.f * 5.9604645e-8f * 1.01f * T.bound_scale * T.vmax * (fabsf(x) + fabsf(y) + fabsf(z)) + 1e-35f;
        if (!(first - second > gap)) mine = support64(T, dir);
    } else {
        mine = support64(T, dir);
    }
    const uint32_t other = __shfl_xor_sync(active, mine, 1);
    const uint32_t ia = role ? other : mine, ib = role ? mine : other;
    V3 r = mat_rotate(q, V3{T.v[ib][0], T.v[ib][1], T.v[ib][2]});
    r = {dadd(r.x, vij.x), dadd(r.y, vij.y), dadd(r.z, vij.z)};
    return sub3(r, V3{T.v[ia][0], T.v[ia][1], T.v[ia][2]});
}

// The step after a support mapping v: -1 undecided (s.n: the next direction), else the result. The
// phases are collide3d's: 0 the first support, 1 the second, 2 portal discovery (p0, p1, p2 = v1, v2,
// v3), 3 portal refinement. Each expression is collide3d's own; lanes in different phases share the
// first test (in phase 0 n = -v0, and v . v0 > 0 is v . n < 0, the products being exactly negated)
// and the portal's normal.
__device__ __forceinline__ int pair_step(PairLane& s, const V3& v) {
    const double TOL = 2e-12;
    const double along = dot3(v, s.n);
    if (s.phase == 2 ? along <= 0.0 : along < 0.0) return 0;
    if (s.phase < 2) {
        if (s.phase == 0) {
            s.p0 = v;
            s.n = cross3(v, s.v0);
            s.phase = 1;
            return fabs(s.n.x) < TOL && fabs(s.n.y) < TOL && fabs(s.n.z) < TOL ? 1 : -1;
        }
        s.p1 = v;
        s.n = cross3(sub3(s.p0, s.v0), sub3(s.p1, s.v0));
        if (dot3(s.n, s.v0) > 0.0) {
            const V3 t = s.p0;
            s.p0 = s.p1;
            s.p1 = t;
            s.n = neg3(s.n);
        }
        s.phase = 2;
        s.count = 1;
        return -1;
    }
    if (s.phase == 2) {
        bool again = true;
        if (dot3(cross3(s.p0, v), s.v0) < 0.0)
            s.p1 = v;
        else if (dot3(cross3(v, s.p1), s.v0) < 0.0)
            s.p0 = v;
        else
            again = false;
        if (again) {
            s.n = cross3(sub3(s.p0, s.v0), sub3(s.p1, s.v0));
            s.count += 1;
            return s.count >= kXenoMaxIter ? 1 : -1;
        }
        s.p2 = v;
        s.count = 1;
        s.phase = 3;
    } else {
        // |x| < TOL sqrt(n . n), the root only where x^2 does not rule it out by far
        const double nn2 = dot3(s.n, s.n), far2 = 1.5 * TOL * TOL * nn2;
        const double x0 = dot3(sub3(v, s.p0), s.n), x1 = dot3(s.p0, s.n);
        if (!(x0 * x0 > far2 && x1 * x1 > far2)) {
            const double tol = dmul(TOL, dsqrt(nn2));
            if (fabs(x0) < tol) return 0;
            if (fabs(x1) < tol) return 1;
        }
        const V3 vp = cross3(v, s.v0);
        const bool t1 = dot3(vp, s.p0) > 0.0, t2 = dot3(vp, s.p1) > 0.0, t3 = dot3(vp, s.p2) > 0.0;
        if (t1 && !t2)
            s.p2 = v;
        else if (!t1 && t3)
            s.p1 = v;
        else
            s.p0 = v;
        if (s.count >= kXenoMaxIter) return 1;
        s.count += 1;
    }
    // the refinement loop's head: the portal's normal away from v0; the origin inside: overlap
    V3 nn = cross3(sub3(s.p1, s.p0), sub3(s.p2, s.p0));
    if (dot3(sub3(s.p0, s.v0), nn) < 0.0) nn = neg3(nn);
    s.n = nn;
    return dot3(s.p0, nn) >= 0.0 ? 1 : -1;
}

// FP32 form of the first test of XenoCollide (phase 0: v1 . v0 > 0, the shapes are separated along the
// line of centres), which ends 7 in 10 of the pairs inside the circumsphere. With v0 and the relative
// orientation M by the FP64 path's formulas in FP32 from d (the other site minus the trial's),
// v1 . v0 = |v0|^2 - max_a a . v0 - max_b b . (-M^T v0). An FP32 value above its error bound decides:
// the FP64 test is then positive too, whichever of tied vertices it takes (its own roundings
// are of order 1e-15). Bound, with si, sj = |q|^2 (1 for versors) and D = |d|_1: v0 is off by at most 16 u32
// si D per component, M by 28 u32 si sj per entry (Cauchy's inequality over the quaternion products),
// M^T v0 by 106 u32 si^2 sj D, so the value by 110 u32 T, T = si D (si D + 3 vmax (1 + si sj)); the
// sites' own error moves it by 2 T / D times its 1-norm. 128 u32 leaves room for the bound's roundings.
__device__ __forceinline__ bool separated32(const ShapeTable& T, float dx, float dy, float dz, float4 qi, float4 qj,
                                            float site_err) {
    // ia = conj(qi) = (s, -x, -y, -z); v0 = vrotate(ia, d); o = ia qj; M = mat_from(o)
    const float s = qi.x, x = -qi.y, y = -qi.z, z = -qi.w;
    const float si = s * s + x * x + y * y + z * z, sj = qj.x * qj.x + qj.y * qj.y + qj.z * qj.z + qj.w * qj.w;
    const float k1 = s * s - (x * x + y * y + z * z), k2 = 2.f * s, k3 = 2.f * (x * dx + y * dy + z * dz);
    const float vx = dx * k1 + (y * dz - z * dy) * k2 + x * k3;
    const float vy = dy * k1 + (z * dx - x * dz) * k2 + y * k3;
    const float vz = dz * k1 + (x * dy - y * dx) * k2 + z * k3;
    const float a = s * qj.x - (x * qj.y + y * qj.z + z * qj.w);
    const float b = qj.y * s + x * qj.x + (y * qj.w - z * qj.z);
    const float c = qj.z * s + y * qj.x + (z * qj.y - x * qj.w);
    const float d = qj.w * s + z * qj.x + (x * qj.z - y * qj.y);
    // -M^T v0
    const float bx = -((a * a + b * b - c * c - d * d) * vx + 2.f * (b * c + a * d) * vy + 2.f * (b * d - a * c) * vz);
    const float by = -(2.f * (b * c - a * d) * vx + (a * a - b * b + c * c - d * d) * vy + 2.f * (c * d + a * b) * vz);
    const float bz = -(2.f * (b * d + a * c) * vx + 2.f * (c * d - a * b) * vy + (a * a - b * b - c * c + d * d) * vz);
    float ha = -INFINITY, hb = -INFINITY;
#pragma unroll 4
    for (uint32_t i = 0; i < T.nv; ++i) {
        const float4 v = T.v32[i];
        ha = fmaxf(ha, v.x * vx + v.y * vy + v.z * vz);
        hb = fmaxf(hb, v.x * bx + v.y * by + v.z * bz);
    }
    const float D = fabsf(dx) + fabsf(dy) + fabsf(dz);
    const float scale = T.bound_scale * si * (si * D + 3.f * T.vmax * (1.f + si * sj));
    return vx * vx + vy * vy + vz * vz - ha - hb > scale * (128.f * 5.9604645e-8f * D + 6.f * site_err);
}

// A warp decides kGroup trials at a time, kGroupLanes lanes for each where a trial's own work is done;
// the kWarps warps of a block go through the steps together (k_flow_poly3).
constexpr uint32_t kGroup = 4, kGroupLanes = 32 / kGroup, kWarps = 4;
constexpr uint32_t kPairs = 128;  // pairs a warp lists before it tests them
struct alignas(16) PolyTeam {
    uint2 step[kGroup][32];  // a trial's stencil in steps of kGroupLanes candidates: first slot, length
    uint2 near[kGroup][28];  // the progress words around each trial's space and the values it needs
    uint32_t pair_q[kPairs];
    uint8_t pair_g[kPairs];
    double t[kGroup][3], q[kGroup][4];  // the trials: site T and versor
    float4 q32[kGroup];                 // the versor in FP32
    int4 t32[kGroup];                   // T in fixed point
};

// The pair of the trial (t, q of the warp's trial `mine`) and slot q: pair_system_to_local as
// poly_overlap64 does it. 0: outside the circumsphere, 1: overlap (coincident centres), -1: to be tested.
__device__ __forceinline__ int pair_begin(const Geometry& g, const Arrays& A, double rcut2, const PolyTeam& S,
                                          uint32_t mine, uint32_t q, PairLane& s) {
    const double4 s4 = ldcg4(A.sorted_s + q), o4 = ldcg4(A.sorted_q + q);
    const double t[3] = {S.t[mine][0], S.t[mine][1], S.t[mine][2]}, sj[3] = {s4.x, s4.y, s4.z};
    double d[3];
    if (!(ref_disp<3>(g, t, sj, d) < rcut2)) return 0;
    const Q ia{S.q[mine][0], -S.q[mine][1], -S.q[mine][2], -S.q[mine][3]};
    s.v0 = vrotate(ia, V3{-d[0], -d[1], -d[2]});
    s.q = mat_from(qmul(ia, Q{o4.x, o4.y, o4.z, o4.w}));
    s.n = neg3(s.v0);
    s.phase = 0;
    return fabs(s.v0.x) < 2e-12 && fabs(s.v0.y) < 2e-12 && fabs(s.v0.z) < 2e-12 ? 1 : -1;
}

// The pair tests of a warp's n listed pairs, two lanes each: bit g of the result is set when trial g
// overlaps. Two lanes that have their result take the next pair, so that the tests' different
// lengths leave few lanes idle; pairs of a trial that is known to overlap are dropped.
template <bool FP32>
__device__ __forceinline__ uint32_t test_pairs(const Geometry& g, const Arrays& A, const ShapeTable& T, double rcut2,
                                               const PolyTeam& S, uint32_t n, uint32_t lane, uint32_t mask) {
    const unsigned full = 0xffffffffu;
    const uint32_t role = lane & 1u;
    uint32_t head = 0, mine = 0;
    bool busy = false;
    PairLane s;
    for (;;) {
        const unsigned idle = __ballot_sync(full, !busy && role == 0u);
        const uint32_t n_idle = __popc(idle);
        uint32_t hit = 0;
        if (head < n && n_idle >= 4u) {
            const uint32_t at = head + __popc(idle & ((1u << (lane & ~1u)) - 1u));
            head += min(n_idle, n - head);
            if (!busy && at < n) {
                mine = S.pair_g[at];
                if (!((mask >> mine) & 1u)) {
                    const int b = pair_begin(g, A, rcut2, S, mine, S.pair_q[at], s);
                    busy = b < 0;
                    if (b == 1) hit = 1u << mine;
                }
            }
        } else if (n_idle == 16u) {
            return mask;
        }
        const unsigned active = __ballot_sync(full, busy);
        if (busy) {
            const V3 v = pair_support<FP32>(T, s.q, s.v0, s.n, role, active);
            const int res = pair_step(s, v);
            busy = res < 0;
            if (res == 1) hit = 1u << mine;
        }
        mask |= __reduce_or_sync(full, hit);
        busy = busy && !((mask >> mine) & 1u);
    }
}

// The listed pairs through XenoCollide's first test, which ends 7 in 10 of them; returns how many
// are left (at the list's front, in order). FP32: separated32, a lane per pair. FP64: the test itself,
// two lanes per pair.
template <bool FP32>
__device__ __forceinline__ uint32_t poly_screen(const Geometry& g, const Arrays& A, const PolyShape& sh,
                                                const ShapeTable& T, PolyTeam& S, uint32_t n, uint32_t lane) {
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    constexpr uint32_t per = FP32 ? 32 : 16;
    uint32_t kept = 0;
#pragma unroll 1
    for (uint32_t p0 = 0; p0 < n; p0 += per) {
        const uint32_t p = p0 + (FP32 ? lane : lane >> 1);
        uint32_t q = 0, mine = 0;
        bool keep = p < n;
        if (keep) {
            q = S.pair_q[p];
            mine = S.pair_g[p];
        }
        if constexpr (FP32) {
            if (keep) {
                const int4 o = __ldcg(reinterpret_cast<const int4*>(A.sorted_off) + q), t = S.t32[mine];
                const double4 o4 = ldcg4(A.sorted_q + q);
                keep = !separated32(T, (float)(int)((uint32_t)o.x - (uint32_t)t.x) * g.fix[0],
                                    (float)(int)((uint32_t)o.y - (uint32_t)t.y) * g.fix[1],
                                    (float)(int)((uint32_t)o.z - (uint32_t)t.z) * g.fix[2], S.q32[mine],
                                    make_float4((float)o4.x, (float)o4.y, (float)o4.z, (float)o4.w), sh.site_err);
            }
        } else {
            PairLane s;
            if (keep) keep = pair_begin(g, A, sh.rcut2, S, mine, q, s) != 0;  // (an overlap is found again)
            const unsigned active = __ballot_sync(full, keep);
            if (keep) keep = !(dot3(pair_support<false>(T, s.q, s.v0, s.n, lane & 1u, active), s.v0) > 0.0);
            if (lane & 1u) keep = false;  // one entry per pair
        }
        const unsigned b = __ballot_sync(full, keep);
        if (keep) {  // (in place: no entry is written beyond those already read)
            S.pair_q[kept + __popc(b & below)] = q;
            S.pair_g[kept + __popc(b & below)] = (uint8_t)mine;
        }
        kept += __popc(b);
        __syncwarp();
    }
    return kept;
}

// The warp's trials (slot k, space m; valid the same in a trial's lanes) against their stencils: the
// circumsphere test (FP32: under the error bound), 8 lanes per trial and a row of the stencil in
// steps of 8 candidates; then the pairs that need the full test are listed, those with the closest centres
// first (they overlap most often), and tested. Returns the trials that overlap. The circumsphere loop
// only collects bits, so the loads of its steps are in flight together (bulk copies into shared
// memory, as for Lennard-Jones, took longer: the rows are 9 candidates long); the list is written
// once per 32 steps by a scan over the lanes.
template <bool FP32, bool SYNC>
__device__ __forceinline__ uint32_t poly_decide(const Geometry& g, const Arrays& A, const PolyShape& sh,
                                                const ShapeTable& T, const uint32_t* m, uint32_t k, bool valid,
                                                uint32_t lane, PolyTeam& S, const uint3& lo, const uint3& len,
                                                PairStats& st) {
    const unsigned full = 0xffffffffu;
    const uint32_t grp = lane / kGroupLanes, sub = lane % kGroupLanes;
    // this lane's parts as steps [a, a + sum) of the trial's
    const uint32_t ls[3] = {lo.x, lo.y, lo.z}, ns[3] = {len.x, len.y, len.z};
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) sum += valid ? (ns[i] + kGroupLanes - 1) / kGroupLanes : 0u;
    uint32_t end = sum;
#pragma unroll
    for (uint32_t o = 1; o < kGroupLanes; o <<= 1) {
        const uint32_t y = __shfl_up_sync(full, end, o, kGroupLanes);
        if (sub >= o) end += y;
    }
    const uint32_t steps = __shfl_sync(full, end, kGroupLanes - 1, kGroupLanes);
    const uint32_t longest = __reduce_max_sync(full, steps);
    const int4 t32 = S.t32[grp];
    const double t[3] = {S.t[grp][0], S.t[grp][1], S.t[grp][2]};
    const float near32 = 0.45f * sh.rcut2_hi32;
    const double near64 = 0.45 * sh.rcut2;
    const unsigned bv = __ballot_sync(full, valid && sub == 0u);
    uint32_t which = 0, mask = 0;  // bit i: trial i
#pragma unroll
    for (uint32_t i = 0; i < kGroup; ++i) which |= ((bv >> (i * kGroupLanes)) & 1u) << i;
    bool first_pass = true;
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < longest || (SYNC && first_pass); s0 += 32u) {
        __syncwarp();  // the steps before have been read
        if (valid) {
            uint32_t at = end - sum;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                for (uint32_t c = 0; c < ns[i]; c += kGroupLanes, ++at)
                    if (at - s0 < 32u) S.step[grp][at - s0] = make_uint2(ls[i] + c, min(ns[i] - c, kGroupLanes));
        }
        __syncwarp();
        const uint32_t n = steps > s0 ? min(32u, steps - s0) : 0u, n_max = min(32u, longest - s0);
        uint32_t need = 0, close = 0;  // bit i: candidate `sub` of step i
#pragma unroll 2
        for (uint32_t i = 0; i < n_max; ++i) {
            const uint2 p = S.step[grp][i];  // (stale beyond n)
            const uint32_t q = p.x + sub;
            const bool ok = i < n && sub < p.y && q != k;
            bool in, cl;
            if constexpr (FP32) {
                const int4 o = ok ? __ldcg(reinterpret_cast<const int4*>(A.sorted_off) + q) : make_int4(0, 0, 0, 0);
                const float d2 = fixed_dist2<3>(g, t32, o);
                in = d2 < sh.rcut2_hi32;
                cl = d2 < near32;
            } else {
                // the circumsphere test that opens poly_overlap64
                const double4 s4 = ok ? ldcg4(A.sorted_s + q) : make_double4(0.0, 0.0, 0.0, 0.0);
                const double sj[3] = {s4.x, s4.y, s4.z};
                double d[3];
                const double d2 = ref_disp<3>(g, t, sj, d);
                in = d2 < sh.rcut2;
                cl = d2 < near64;
            }
            need |= (ok && in ? 1u : 0u) << i;
            close |= (ok && cl ? 1u : 0u) << i;
            st.checks += ok ? 1u : 0u;
        }
        if (FP32) st.rechecks += __popc(need);
        if ((mask >> grp) & 1u) need = 0;
        while (__any_sync(full, need != 0u) || (SYNC && first_pass)) {
            // this lane's places: the close pairs of all lanes first, then the others
            uint32_t x = __popc(need & close) | (__popc(need & ~close) << 16);
            const uint32_t own = x;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(full, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t all = __shfl_sync(full, x, 31), n_close = all & 0xffffu, n_pairs = n_close + (all >> 16);
            uint32_t at_close = (x - own) & 0xffffu, at_far = n_close + ((x - own) >> 16);
            uint32_t left = need;
            while (left) {
                const uint32_t i = (uint32_t)__ffs(left) - 1u, bit = 1u << i;
                left &= left - 1u;
                const uint32_t at = close & bit ? at_close++ : at_far++;
                if (at < kPairs) {
                    S.pair_q[at] = S.step[grp][i].x + sub;
                    S.pair_g[at] = (uint8_t)grp;
                    need &= ~bit;
                }
            }
            __syncwarp();
            if (SYNC && first_pass) __syncthreads();
            const uint32_t listed = poly_screen<FP32>(g, A, sh, T, S, min(n_pairs, kPairs), lane);
            if (SYNC && first_pass) __syncthreads();
            first_pass = false;
            mask = test_pairs<FP32>(g, A, T, sh.rcut2, S, listed, lane, mask);
            if ((mask >> grp) & 1u) need = 0;
            __syncwarp();
        }
        if ((mask & which) == which && !(SYNC && first_pass)) break;  // every trial is decided
    }
    return mask;
}

// The stencils around the spaces m of the warp's trials (valid the same in a trial's lanes): lane `sub`
// < 6 of a trial has the slots of parts 3 sub .. 3 sub + 2, so the loads of all trials are in flight
// together.
__device__ __forceinline__ void poly_parts(const Geometry& g, const Arrays& A, const uint32_t* m, bool valid, uint32_t sub,
                                           uint3& lo, uint3& len) {
    uint32_t l[3], n[3];
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i) {
        const uint32_t p = 3u * sub + i;
        float s0, s1;
        l[i] = n[i] = 0;
        if (valid && p < 2u * kRows<3>)
            stencil_part<3>(g, A.cell_start, m, (int)(p >> 1), (p & 1u) != 0, l[i], n[i], s0, s1);
    }
    lo = make_uint3(l[0], l[1], l[2]);
    len = make_uint3(n[0], n[1], n[2]);
}

// The sweep of hard convex polyhedra: a block takes kWarps x kGroup trials of one colour (one unit) in
// dataflow order (hmc_flow.cuh), all colour passes of colour sets [L.round, L.round_end) in one
// launch. The trials of a unit are neighbours in their colour's list, so they wait for the same
// slab of the box. INJ: the probe mode, warp w decides injected trials kGroup w .. against the
// unchanged state.
// Bound: instruction fetch. The four steps of a unit (set-up, circumspheres, screen, XenoCollide) are
// some 2,000 instructions; with every warp at its own place among them the schedulers found no
// instruction in a third of the cycles, so the block's warps take the steps together (a barrier before
// each): 24.6 -> 20.9 ms on 2^18 cubes at packing fraction 0.55, ten sweeps of each move (FP32;
// FP64 44.7 -> 30.6; the sweeps alone, 22.5 with the frame's copy). One launch per colour pass with four
// trials per warp and a lane per pair test: 42.0 ms (FP64 44.3).
template <bool FP32, bool INJ, int MINB>
__global__ void __launch_bounds__(32 * kWarps, MINB)
    k_flow_poly3(Geometry g, Arrays A, PolyShape sh, Launch L, uint32_t rotate, Injected J) {
    constexpr unsigned full = 0xffffffffu;
    // each lane polls up to kWords of its trial's 27 progress words: word sub + i lanes, i < kWords;
    // the own space's is word 13
    constexpr uint32_t kWords = (27 + kGroupLanes - 1) / kGroupLanes;
    constexpr uint32_t kOwnLane = 13 % kGroupLanes, kOwnBit = 1u << (13 / kGroupLanes);
    __shared__ PolyTeam s_team[kWarps];
    __shared__ uint32_t s_unit;
    __shared__ FlowRange s_range;
    __shared__ ShapeTable T;
    const uint32_t lane = threadIdx.x & 31u, grp = lane / kGroupLanes, sub = lane % kGroupLanes;
    PolyTeam& S = s_team[threadIdx.x >> 5];
    if (threadIdx.x < 32u) {
        float vmax = 0.f;
        if (threadIdx.x < sh.nv) {
            const double4 v = ldg4(sh.verts + threadIdx.x);
            T.v[threadIdx.x][0] = v.x, T.v[threadIdx.x][1] = v.y, T.v[threadIdx.x][2] = v.z;
            T.v32[threadIdx.x] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
            vmax = __double2float_ru(fmax(fabs(v.x), fmax(fabs(v.y), fabs(v.z))));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(full, vmax, o));
        if (threadIdx.x == 0) T.vmax = vmax, T.nv = sh.nv, T.bound_scale = sh.bound_scale;
    }
    if (!INJ) {
        grid_dependency_wait();
        if (threadIdx.x == 0) s_range = flow_range(A.stats, L.round, L.round_end, 8, kGroup * kWarps);
    }
    __syncthreads();
    const FlowRange& f = s_range;
    const uint32_t n = INJ ? (J.n + kGroup - 1) / kGroup : f.n_units;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t n_accepted = 0;
    PairStats st;
    uint32_t next = INJ ? warp : (threadIdx.x == 0 ? atomicAdd(&A.stats->ticket, 1u) : 0u);
    for (;;) {
        uint32_t unit = next;
        if (!INJ) {
            if (threadIdx.x == 0) s_unit = next;
            __syncthreads();
            unit = s_unit;
        }
        if (unit >= n) break;
        if (INJ) next = unit + n_warps;
        else if (threadIdx.x == 0) next = atomicAdd(&A.stats->ticket, 1u);
        uint32_t m[3] = {0, 0, 0}, k = 0, round = 0, e = 0;
        bool valid = false;
        double ta = 0.0;
        Q qi{1.0, 0.0, 0.0, 0.0};
        uint8_t flag = 0;
        const uint32_t axis = sub < 3 ? sub : 0u;
        if constexpr (INJ) {
            const uint32_t w = unit * kGroup + grp;
            if (w < J.n) {
                const uint64_t body = J.bodies[w];
                k = A.slot_of_body[body];
                const double4 w4 = J.trial[w], q4 = J.trial_q[w];
                double x[3] = {w4.x, w4.y, w4.z};
                qi = Q{q4.x, q4.y, q4.z, q4.w};
                valid = point_to_space<3>(g, x, m);
                if (!valid)
                    atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
                else if (cell_index<3>(g, m) != A.body_cell[body])
                    flag |= kTrialOutsideSpace;
                wrap_inv<3>(g.L, g.invL, x);
                ta = axis == 0 ? x[0] : (axis == 1 ? x[1] : x[2]);
            }
        } else {
            uint32_t color, entry;
            flow_unit(f, unit, round, color, entry);
            entry = (entry * kWarps + (threadIdx.x >> 5)) * kGroup + grp;
            valid = entry < f.count[color];
            uint4 di = make_uint4(0u, 0u, 0u, 0u);
            e = (round - f.r0) * f.per_set + f.prefix[color] + entry;
            if (valid) di = __ldg(A.draw_i + e);
            k = di.x;
            unpack_m<3>(di.y, m);
        }
        const bool listed = valid;  // the group has a trial (its space is finished below)
        uint3 lo, len;
        poly_parts(g, A, m, valid, sub, lo, len);
        if (!INJ && valid) {
            const uint32_t color = ((m[0] & 1u) << 2) | ((m[1] & 1u) << 1) | (m[2] & 1u);
#pragma unroll 1
            for (uint32_t i = sub; i < 27u; i += kGroupLanes) {
                uint2 w;
                flow_need<3>(g, m, color, round, i, w.x, w.y);
                S.near[grp][i] = w;
            }
        }
        __syncwarp();
        if constexpr (!INJ) {
            unsigned pending = 0;
            if (valid) pending = (1u << kWords) - 1u;
            if (sub + (kWords - 1u) * kGroupLanes >= 27u) pending &= ~(1u << (kWords - 1u));
            // the own space first: the proposal needs no other
            bool going = flow_wait_words<kWords>(A.progress, S.near[grp], sub, kGroupLanes, pending,
                                                 sub == kOwnLane ? kOwnBit : 0u, A.stats, L.flow);
            __syncwarp();
            const AxisGeometry ax = axis_geometry<3>(g, axis);
            const uint32_t ma = axis == 0 ? m[0] : (axis == 1 ? m[1] : m[2]);
            double x = 0.0, w1 = 0.0;
            if (valid) {
                const double* draw = reinterpret_cast<const double*>(A.draw_d + e);
                x = __ldcg(reinterpret_cast<const double*>(A.sorted_b + k) + axis);
                const double4 q4 = ldcg4(A.sorted_q + k);
                qi = Q{q4.x, q4.y, q4.z, q4.w};
                if (rotate)
                    qi = qmul(Q{__ldg(draw), __ldg(draw + 1), __ldg(draw + 2), __ldg(draw + 3)}, qi);
                else
                    x = dadd(x, __ldg(draw + axis));
                w1 = wrap_axis(ax.L, ax.invL, x);  // W1 = wrap(propose(..))
            }
            const bool in_axis = !valid || axis_in_space(ax.origin, ax.width, ax.invW, ax.shape, ma, w1);
            const unsigned in = __ballot_sync(full, in_axis);
            constexpr unsigned all = (1u << kGroupLanes) - 1u;
            valid = valid && ((in >> (grp * kGroupLanes)) & all) == all;
            if (valid) ta = wrap_axis(ax.L, ax.invL, w1);  // the trial site T = wrap(W1)
            if (!valid) pending = 0;
            if (going)
                going = flow_wait_words<kWords>(A.progress, S.near[grp], sub, kGroupLanes, pending, ~0u, A.stats,
                                                    L.flow);
            if (!going) valid = false;
            if (__syncthreads_or(!going)) break;
            __syncwarp();
        }
        if (valid) {
            if (sub < 3u) {
                S.t[grp][sub] = ta;
                reinterpret_cast<int*>(&S.t32[grp])[sub] = fixed_axis(g.invL[axis], ta);
            }
            if (sub == 3u) {
                S.q[grp][0] = qi.s, S.q[grp][1] = qi.x, S.q[grp][2] = qi.y, S.q[grp][3] = qi.z;
                S.q32[grp] = make_float4((float)qi.s, (float)qi.x, (float)qi.y, (float)qi.z);
            }
        }
        __syncwarp();
        const uint32_t mask = poly_decide<FP32, !INJ>(g, A, sh, T, m, k, valid, lane, S, lo, len, st);
        const bool accept = valid && !((mask >> grp) & 1u);
        if constexpr (INJ) {
            const uint32_t w = unit * kGroup + grp;
            if (sub == 0 && w < J.n) {
                J.decisions[w] = accept;
                J.flags[w] = flag;
            }
        } else {
            if (accept) {
                // update_body_properties: body = T, site = wrap(body)
                const uint32_t body = A.sorted_body[k];
                if (sub < 3u) {
                    const double tc = S.t[grp][sub], sv = wrap_axis(g.L[axis], g.invL[axis], tc);
                    reinterpret_cast<double*>(A.sorted_b + k)[sub] = tc;
                    reinterpret_cast<double*>(A.sorted_s + k)[sub] = sv;
                    if (FP32) reinterpret_cast<int*>(A.sorted_off + k)[sub] = fixed_axis(g.invL[axis], sv);
                    reinterpret_cast<double*>(A.body_pos + body)[sub] = tc;
                }
                const double4 q4 = make_double4(S.q[grp][0], S.q[grp][1], S.q[grp][2], S.q[grp][3]);
                if (sub == 3u) A.sorted_q[k] = A.body_ori[body] = q4;
                n_accepted += sub == 0u;
            }
            __syncwarp();
            if (listed && sub == 0u) store_release(A.progress + cell_index<3>(g, m), round + 1u);
        }
        __syncwarp();
    }
    flush_stats(A.stats, st, n_accepted);
}

// ---- the insertion hamiltonian: approximate shape overlap -----------------------------------
// Anisotropic::site_pair_energy (anisotropic.rs:120-135) of ApproximateShapeOverlap
// (approximate_shape_overlap.rs:122-131) for the site t with versor qi against the site sj (image
// rule) with versor qj: 0 at a centre distance >= r_cut, else pair_system_to_local and
// IntersectsAt::approximate_separation_distance (hoomd-geometry/src/lib.rs:307-325): the
// direction v / |v| (lib.rs:632-639; the last axis for v = 0, cartesian.rs:313-318) and d grown
// by `resolution` while Convex::intersects_at (convex.rs:130-143: the bounding spheres,
// |w|^2 <= (R + R)^2, then XenoCollide) holds at w = v + direction * d; the energy is
// OverlapPenalty(-d).
__device__ __forceinline__ double shape_overlap3(const Geometry& g, const PolyShape& sh, const ShapeOverlap& so,
                                                 const double* t, const Q& qi, const double* sj, const Q& qj,
                                                 uint32_t& capped) {
    double d[3];
    const double d2 = ref_disp<3>(g, t, sj, d);
    if (dsqrt(d2) >= so.rcut) return 0.0;
    const V3 rab{-d[0], -d[1], -d[2]};  // image - t
    const Q ia{qi.s, -qi.x, -qi.y, -qi.z};
    const V3 v = vrotate(ia, rab);
    const Q oij = qmul(ia, qj);
    const double norm = dsqrt(dot3(v, v));
    const V3 dir = norm == 0.0 ? V3{0.0, 0.0, 1.0} : V3{ddiv(v.x, norm), ddiv(v.y, norm), ddiv(v.z, norm)};
    double sep = 0.0;
    for (uint32_t step = 0;; ++step) {
        const V3 w{dadd(v.x, dmul(dir.x, sep)), dadd(v.y, dmul(dir.y, sep)), dadd(v.z, dmul(dir.z, sep))};
        if (!(dot3(w, w) <= so.rr) || !collide3d(sh.verts, sh.nv, w, oij)) break;
        if (step >= so.max_steps) {
            capped = 1;
            break;
        }
        sep = dadd(sep, so.resolution);
    }
    return separation_penalty(so, sep);
}

// ParallelSweep colour pass under the approximate shape overlap (FP64 in both precision modes):
// one warp per trial from k_propose_poly3 (soft), the stencil's candidates 32 at a time. Each lane
// adds the pair energies of the trial (T, q) and of the body's current site (S, q_k) against its
// candidates; butterfly sums give E_final and E_initial (delta_energy_one, pairwise_cutoff.rs:
// 919-941: an infinite pair makes E_final infinite and the move is rejected) and the Metropolis
// test (parallel_sweep.rs:267-268) uses the uniform drawn after the move.
__global__ void __launch_bounds__(128) k_sweep_poly3_soft(Geometry g, Arrays A, PolyShape sh, ShapeOverlap so,
                                                          Launch L) {
    if (L.early_wait) grid_dependency_wait();  // first pass: the rebuild's arrays are read at once
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t n_accepted = 0, capped = 0;
    PairStats pst;
    const uint32_t n_active = active_count(A, L.color, L.round);
    for (uint32_t w = warp; w < n_active; w += n_warps) {
        const size_t e = (size_t)L.color * g.color_stride + w;
        const uint32_t k = __ldg(A.trial_k + e);
        if (k == kNoTrial) continue;  // warp-uniform: the move left its space
        uint32_t m[3] = {0, 0, 0};
        unpack_m<3>(__ldg(A.color_cells + e), m);
        const double4 t4 = ldg4(A.trial_t + e);
        const double t[3] = {t4.x, t4.y, t4.z};
        const double u = t4.w;
        const double4 q4 = ldg4(A.trial_q + e);
        const Q qt{q4.x, q4.y, q4.z, q4.w};
        const FlatStencil fs = flat_stencil<3>(g, A.cell_start, m, lane);
        grid_dependency_wait();  // the previous colour's moves are visible from here on
        allow_dependent_launch();
        const double4 s4 = ldg4(A.sorted_s + k);
        const double si[3] = {s4.x, s4.y, s4.z};
        const double4 o4 = ldg4(A.sorted_q + k);
        const Q qk{o4.x, o4.y, o4.z, o4.w};
        double a = 0.0, b = 0.0, mag = 0.0;
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < fs.total; j0 += 32) {
            const uint32_t j = j0 + lane;
            uint32_t part;
            const uint32_t q = flat_slot(fs, j, part);
            if (j < fs.total && q != k) {
                const double4 c4 = ldg4(A.sorted_s + q);
                const double sj[3] = {c4.x, c4.y, c4.z};
                const double4 cq = ldg4(A.sorted_q + q);
                const Q qj{cq.x, cq.y, cq.z, cq.w};
                const double x = shape_overlap3(g, sh, so, t, qt, sj, qj, capped);
                const double y = shape_overlap3(g, sh, so, si, qk, sj, qj, capped);
                a = dadd(a, x);
                b = dadd(b, y);
                mag += fabs(x) + fabs(y);
                pst.checks += 2;
            }
        }
        const double e_new = warp_sum64(a), e_old = warp_sum64(b);
        mag = warp_sum64(mag);
        const double du = dsub(e_new, e_old);
        const double e0 = exp(ddiv(-du, L.kt));
        if (lane == 0 && order_ambiguous(du, mag, fs.total, u, L.kt, e0)) pst.ambiguous++;
        if ((du <= 0.0 || u < e0) && lane == 0) {
            n_accepted++;
            double sv[3] = {t[0], t[1], t[2]};
            wrap_inv<3>(g.L, g.invL, sv);
            const uint32_t body = A.sorted_body[k];
            A.sorted_b[k] = make_double4(t[0], t[1], t[2], 0.0);
            A.sorted_s[k] = make_double4(sv[0], sv[1], sv[2], 0.0);
            A.sorted_off[k] = cell_offsets<3>(g, sv, m);
            A.sorted_q[k] = make_double4(qt.s, qt.x, qt.y, qt.z);
            A.body_pos[body] = make_double4(t[0], t[1], t[2], 0.0);
            A.body_ori[body] = make_double4(qt.s, qt.x, qt.y, qt.z);
        }
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, capped != 0u) && lane == 0) atomicOr(&A.stats->error_flags, kErrIterationCap);
    grid_dependency_wait();
    allow_dependent_launch();
    flush_stats(A.stats, pst, n_accepted);
}

// PairwiseCutoff::total_energy (pairwise_cutoff.rs:720-745) under the approximate shape overlap:
// one thread per body i adds the pairs with the bodies j > i of its stencil in i's frame (the
// reference's site_tag_i < site_tag_j; tags are body indices here), summed with atomics.
__global__ void k_energy_poly3_soft(Geometry g, Arrays A, PolyShape sh, ShapeOverlap so, uint32_t n, double* out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t capped = 0;
    if (k < n) {
        const uint32_t bi = A.sorted_body[k];
        const double4 s4 = A.sorted_s[k];
        const double t[3] = {s4.x, s4.y, s4.z};
        const double4 o4 = A.sorted_q[k];
        const Q qi{o4.x, o4.y, o4.z, o4.w};
        uint32_t m[3];
        uint32_t c = A.body_cell[bi];
        for (int a = 2; a >= 0; --a) {
            m[a] = c % g.shape[a];
            c /= g.shape[a];
        }
        double e = 0.0;
        for_each_neighbor<3>(g, A.cell_start, m, [&](uint32_t q, const float*) -> bool {
            if (A.sorted_body[q] <= bi) return false;
            const double4 c4 = A.sorted_s[q];
            const double sj[3] = {c4.x, c4.y, c4.z};
            const double4 cq = A.sorted_q[q];
            e = dadd(e, shape_overlap3(g, sh, so, t, qi, sj, Q{cq.x, cq.y, cq.z, cq.w}, capped));
            return false;
        });
        atomicAdd(out, e);
    }
    if (capped) atomicOr(&A.stats->error_flags, kErrIterationCap);
}

// QuickInsert's insertion loop (k_quick_insert in hmc_serial.cu) for convex polyhedra under the
// approximate shape overlap, one warp: a UniformIn body draws its position per axis, then a
// uniform random versor (StandardUniform for Versor, quaternion.rs:863-885: four standard normals,
// scalar first, divided by sqrt(|v|^2 + s^2)); only whether the insertion energy is infinite or
// positive matters, and single pairs decide both.
__global__ void __launch_bounds__(32) k_quick_insert_poly3(Geometry g, Arrays A, SerialGrid G, PolyShape sh,
                                                           ShapeOverlap so, Launch L, QuickInsertArgs q, BodyTags T,
                                                           unsigned long long* out) {
    const uint32_t lane = threadIdx.x;
    if (A.stats->error_flags) return;
    Sfc64 rng = make_rng(L.step, L.substep, L.seed, 0);
    uint32_t n = q.n0, capped = 0;
    uint64_t inserted = 0, overlapping = 0, rejected = 0;
    for (uint64_t attempt = 0; attempt < q.attempts; ++attempt) {
        double x[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double u = dsub(as_double(0x3FF0000000000000ULL | (rng.next_u64() >> 12)), 1.0);
            x[a] = dadd(dmul(u, q.scale[a]), q.low[a]);
        }
        const double sc = standard_normal(rng, A.zig_x, A.zig_f);
        V3 vv;
        vv.x = standard_normal(rng, A.zig_x, A.zig_f);
        vv.y = standard_normal(rng, A.zig_x, A.zig_f);
        vv.z = standard_normal(rng, A.zig_x, A.zig_f);
        const double norm = dsqrt(dadd(dot3(vv, vv), dmul(sc, sc)));
        const Q o{ddiv(sc, norm), ddiv(vv.x, norm), ddiv(vv.y, norm), ddiv(vv.z, norm)};
        double t[3] = {x[0], x[1], x[2]};
        wrap_inv<3>(g.L, g.invL, t);
        uint32_t m[3] = {0, 0, 0}, cell;
        serial_cell<3>(g, G, t, m);
        bool inf = false, pos = false;
        if (lane_cell<3>(G, m, lane, &cell)) {
            const uint32_t cnt = G.size[cell];
            for (uint32_t kk = 0; kk < cnt && !inf; ++kk) {
                const uint32_t j = G.items[(size_t)cell * G.cap + kk];
                const double4 s4 = G.site[j];
                const double sv[3] = {s4.x, s4.y, s4.z};
                const double4 oj = A.body_ori[j];
                const double e = shape_overlap3(g, sh, so, t, o, sv, Q{oj.x, oj.y, oj.z, oj.w}, capped);
                inf = e == __longlong_as_double(0x7ff0000000000000ll);
                pos = pos || e > 0.0;
            }
        }
        inf = __any_sync(0xffffffffu, inf);
        pos = __any_sync(0xffffffffu, pos);
        if (inf) {
            rejected++;
            continue;
        }
        if (n >= q.capacity) {
            if (lane == 0) atomicOr(&A.stats->error_flags, kErrCellOverflow);
            break;
        }
        if (lane == 0) {
            grid_append<3>(g, A, G, T, n, x);
            A.body_ori[n] = make_double4(o.s, o.x, o.y, o.z);
        }
        __syncwarp();
        n++;
        inserted++;
        if (pos) overlapping++;
        if (inserted == q.to_insert || overlapping >= q.allowed) break;
        if (A.stats->error_flags) break;
    }
    if (__any_sync(0xffffffffu, capped != 0u) && lane == 0) atomicOr(&A.stats->error_flags, kErrIterationCap);
    if (lane == 0) {
        out[0] = inserted;
        out[1] = overlapping;
        out[2] = rejected;
        out[3] = n;
    }
}

// Injected moves (position and versor): warp per move, decision in the requested mode.
template <bool FP32>
__global__ void __launch_bounds__(128) k_eval_poly3(Geometry g, Arrays A, PolyShape sh, const uint64_t* bodies,
                                                    const double4* trial, const double4* trial_q, uint32_t n,
                                                    uint8_t* decisions) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    PairStats st;
    if (i < n) {
        const uint32_t k = A.slot_of_body[bodies[i]];
        const double4 w4 = trial[i];
        double t[3] = {w4.x, w4.y, w4.z};
        wrap_inv<3>(g.L, g.invL, t);
        const double4 q4 = trial_q[i];
        const Q qi{q4.x, q4.y, q4.z, q4.w};
        uint32_t m[3];
        uint8_t dec = 0;
        if (point_to_space<3>(g, t, m)) {
            const FlatStencil fs = flat_stencil<3>(g, A.cell_start, m, lane);
            dec = poly_overlaps<FP32>(g, A, sh, t, qi, fixed_site<3>(g, t), fs, k, lane, st) ? 0 : 1;
        } else if (lane == 0) {
            atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
        }
        if (lane == 0) decisions[i] = dec;
    }
    flush_stats(A.stats, st, 0u);
}

// Overlapping pairs (i < j), FP64 (the overlap check of total_energy).
__global__ void k_overlap_poly3(Geometry g, Arrays A, PolyShape sh, uint32_t n) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t found = 0;
    if (k < n) {
        const uint32_t bi = A.sorted_body[k];
        const double4 s4 = A.sorted_s[k];
        const double t[3] = {s4.x, s4.y, s4.z};
        const double4 q4 = A.sorted_q[k];
        const Q qi{q4.x, q4.y, q4.z, q4.w};
        uint32_t m[3];
        uint32_t c = A.body_cell[bi];
        for (int a = 2; a >= 0; --a) {
            m[a] = c % g.shape[a];
            c /= g.shape[a];
        }
        for_each_neighbor<3>(g, A.cell_start, m, [&](uint32_t q, const float*) -> bool {
            if (A.sorted_body[q] <= bi) return false;
            const double4 o4 = A.sorted_s[q];
            const double sj[3] = {o4.x, o4.y, o4.z};
            if (poly_overlap64(g, A, sh.verts, sh.nv, sh.rcut2, t, qi, sj, q)) found++;
            return false;
        });
    }
    const unsigned tot = __reduce_add_sync(0xffffffffu, found);
    if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&A.stats->overlaps, (unsigned long long)tot);
}

// Trial moves for the move-size tuner (tune_local.rs:21-89): sample j draws a uniformly random
// body, proposes a move of it and its Metropolis uniform from its own counter stream
// Counter(step, substep, seed).index(2^63 | tune_step << 32 | j). The reference draws all samples
// from one sequential stream; per-sample streams make the samples independent of each other
// and of the sweep's streams, with the same distribution.
template <int DIM>
__global__ void k_tune_moves(Geometry g, Arrays A, Launch L, uint32_t tune_step, uint32_t samples, uint32_t rotate,
                             uint64_t* bodies, double4* trial, double4* trial_q, double* uu) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= samples) return;
    Sfc64 rng = make_rng(L.step, L.substep, L.seed, (1ull << 63) | ((uint64_t)tune_step << 32) | (uint64_t)j);
    const uint32_t b = canon_range_u32(rng, L.n_bodies);
    const double4 b4 = A.body_pos[b];
    double x[3] = {b4.x, b4.y, b4.z};
    Q q{1.0, 0.0, 0.0, 0.0};
    if (A.body_ori) {
        const double4 q4 = A.body_ori[b];
        q = Q{q4.x, q4.y, q4.z, q4.w};
    }
    if (rotate && DIM == 2) {
        // Rotate<Angle>::propose (rotate/angle.rs:46-55): theta += Uniform(-a, a); q.s holds theta
        const double u = dsub(as_double(0x3FF0000000000000ULL | (rng.next_u64() >> 12)), 1.0);
        q.s = dadd(q.s, dadd(dmul(u, dsub(L.max_move, -L.max_move)), -L.max_move));
    } else if (rotate) {
        q = versor_move(rng, L.max_move, A.zig_x, A.zig_f, q);
    } else {
        double dv[3];
        ball_sample<DIM>(rng, L.max_move, A.zig_x, A.zig_f, dv);
        for (int a = 0; a < DIM; ++a) x[a] = dadd(x[a], dv[a]);
    }
    wrap_inv<DIM>(g.L, g.invL, x);
    bodies[j] = b;
    trial[j] = make_double4(x[0], x[1], DIM == 3 ? x[2] : 0.0, 0.0);
    trial_q[j] = make_double4(q.s, q.x, q.y, q.z);
    uu[j] = uniform01(rng);
}

// The sequential-stream tuner for hard convex polyhedra (tune_stream_run): Translate or
// Rotate<Versor> proposals, the trial accepted when XenoCollide finds no overlap with any
// candidate of the stencil around its site's space (FP64, the warp 32 candidates at a time).
__global__ void __launch_bounds__(32) k_tune_stream_poly3(TuneJob* jobs, uint32_t n_jobs, PolyShape sh) {
    if (blockIdx.x >= n_jobs) return;
    TuneJob& J = jobs[blockIdx.x];
    const Geometry& g = J.g;
    const Arrays& A = J.a;
    const uint32_t lane = threadIdx.x & 31u;
    PairStats st;
    tune_stream_run(
        J,
        [&](Sfc64& rng, double m, uint32_t b, double* x, double* q) {
            const double4 q4 = A.body_ori[b];
            Q qi{q4.x, q4.y, q4.z, q4.w};
            if (J.rotate) {
                const double4 b4 = A.body_pos[b];
                x[0] = b4.x;
                x[1] = b4.y;
                x[2] = b4.z;
                qi = versor_move(rng, m, A.zig_x, A.zig_f, qi);
                wrap_inv<3>(g.L, g.invL, x);
            } else {
                tune_translate<3>(rng, g, A, m, b, x);
            }
            q[0] = qi.s;
            q[1] = qi.x;
            q[2] = qi.y;
            q[3] = qi.z;
        },
        [&](Sfc64&, uint32_t b, const double* x, const double* q) -> bool {
            double t[3] = {x[0], x[1], x[2]};
            wrap_inv<3>(g.L, g.invL, t);
            uint32_t m[3] = {0, 0, 0};
            if (!point_to_space<3>(g, t, m)) {
                if (lane == 0) atomicOr(&A.stats->error_flags, kErrOutsideCheckerboard);
                return false;
            }
            const FlatStencil fs = flat_stencil<3>(g, A.cell_start, m, lane);
            const Q qi{q[0], q[1], q[2], q[3]};
            return !poly_overlaps<false>(g, A, sh, t, qi, make_int4(0, 0, 0, 0), fs, A.slot_of_body[b], lane, st);
        });
}

// Sweep::apply_with_filter (hoomd-mc/src/sweep.rs:159-224) for hard convex polyhedra: one trial
// per body in index order from the one stream Counter(step, substep, seed).make_rng(), Translate
// or Rotate<Versor>, accepted when no site of the serial grid's stencil overlaps it (dH is 0 or
// infinite: no uniform is drawn); one warp, a lane per stencil cell, as for spheres. The pair
// tests read each body's versor by body index.
__global__ void __launch_bounds__(32) k_serial_poly3(Geometry g, Arrays A, SerialGrid G, PolyShape sh, Launch L,
                                                     uint32_t rotate, const uint8_t* __restrict__ mask) {
    const uint32_t lane = threadIdx.x;
    if (A.stats->error_flags) return;
    Arrays Ab = A;
    Ab.sorted_q = A.body_ori;
    Sfc64 rng = make_rng(L.step, L.substep, L.seed, 0);
    uint64_t accepted = 0;
    for (uint32_t b = 0; b < L.n_bodies; ++b) {
        if (mask && !mask[b]) continue;
        const double4 b4 = A.body_pos[b];
        double x[3] = {b4.x, b4.y, b4.z};
        const double4 q4 = A.body_ori[b];
        Q qi{q4.x, q4.y, q4.z, q4.w};
        if (rotate) {
            qi = versor_move(rng, L.max_move, A.zig_x, A.zig_f, qi);
        } else {
            double dv[3];
            ball_sample<3>(rng, L.max_move, A.zig_x, A.zig_f, dv);
            for (int a = 0; a < 3; ++a) x[a] = dadd(x[a], dv[a]);
        }
        wrap_inv<3>(g.L, g.invL, x);  // W1 = wrap(propose(..))
        double t[3] = {x[0], x[1], x[2]};
        wrap_inv<3>(g.L, g.invL, t);  // the trial site T = wrap(W1)
        uint32_t m[3] = {0, 0, 0}, cell;
        serial_cell<3>(g, G, t, m);
        bool overlap = false;
        if (lane_cell<3>(G, m, lane, &cell)) {
            const uint32_t cnt = G.size[cell];
            for (uint32_t k = 0; k < cnt && !overlap; ++k) {
                const uint32_t j = G.items[(size_t)cell * G.cap + k];
                if (j == b) continue;
                const double4 s4 = G.site[j];
                const double sv[3] = {s4.x, s4.y, s4.z};
                overlap = poly_overlap64(g, Ab, sh.verts, sh.nv, sh.rcut2, t, qi, sv, j);
            }
        }
        if (__any_sync(0xffffffffu, overlap)) continue;
        accepted++;
        if (lane == 0) {
            // update_body_properties: body = wrap(W1) = T, site = wrap(body), versor as proposed
            double sv[3] = {t[0], t[1], t[2]};
            wrap_inv<3>(g.L, g.invL, sv);
            A.body_pos[b] = make_double4(t[0], t[1], t[2], 0.0);
            A.body_ori[b] = make_double4(qi.s, qi.x, qi.y, qi.z);
            G.site[b] = make_double4(sv[0], sv[1], sv[2], 0.0);
            serial_move<3>(g, G, A, b, sv);
        }
        __syncwarp();
        if (A.stats->error_flags) break;
    }
    if (lane == 0) {
        A.stats->accepted = accepted;
        A.stats->rechecks = 0;
    }
}

// Proposals for a body at the origin with the identity orientation, proposal i from
// Counter(step, substep, seed).index(i): kind 0 Translate (the displacement), kind 1 Rotate
// (3-D: the versor; 2-D: the angle), kind 2 one StandardNormal draw.
template <int DIM>
__global__ void k_sample_moves(Launch L, uint32_t kind, uint64_t n, const double* zx, const double* zf, double* out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Sfc64 rng = make_rng(L.step, L.substep, L.seed, i);
    if (kind == 2) {
        out[i] = standard_normal(rng, zx, zf);
    } else if (kind == 0) {
        double dv[3];
        ball_sample<DIM>(rng, L.max_move, zx, zf, dv);
        for (int a = 0; a < DIM; ++a) out[i * DIM + a] = dv[a];
    } else if (DIM == 3) {
        const Q q = versor_move(rng, L.max_move, zx, zf, Q{1.0, 0.0, 0.0, 0.0});
        out[i * 4 + 0] = q.s;
        out[i * 4 + 1] = q.x;
        out[i * 4 + 2] = q.y;
        out[i * 4 + 3] = q.z;
    } else {
        const double u = dsub(as_double(0x3FF0000000000000ULL | (rng.next_u64() >> 12)), 1.0);
        out[i] = dadd(0.0, dadd(dmul(u, dsub(L.max_move, -L.max_move)), -L.max_move));
    }
}

}  // namespace

cudaError_t launch_sample_moves(int dim, uint32_t kind, double maximum, uint64_t step, uint32_t substep,
                                uint32_t seed, uint64_t n, const double* zig, double* out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    Launch l{};
    l.step = step;
    l.substep = substep;
    l.seed = seed;
    l.max_move = maximum;
    const uint32_t blocks = (uint32_t)((n + 127) / 128);
    if (dim == 2)
        k_sample_moves<2><<<blocks, 128, 0, s>>>(l, kind, n, zig, zig + kZigLayers + 1, out);
    else
        k_sample_moves<3><<<blocks, 128, 0, s>>>(l, kind, n, zig, zig + kZigLayers + 1, out);
    return cudaGetLastError();
}

cudaError_t launch_serial_poly(const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv, double rcut2,
                               const Launch& l, bool rotate, const uint32_t* nc, const double* w, uint32_t cap,
                               uint32_t* size, uint32_t* items, uint32_t* cell_of, double4* site, const uint8_t* mask,
                               cudaStream_t s) {
    const SerialGrid G = make_grid(3, nc, w, cap, size, items, cell_of, site);
    cudaError_t e = build_grid(3, g, a, G, l.n_bodies, s);
    if (e != cudaSuccess || l.n_bodies == 0) return e;
    k_serial_poly3<<<1, 32, 0, s>>>(g, a, G, PolyShape{verts, nv, rcut2, 0.f, 0.f, 1.f}, l, rotate ? 1u : 0u, mask);
    return cudaGetLastError();
}

cudaError_t launch_propose_poly(const Geometry& g, const Arrays& a, const Launch& l, bool rotate, cudaStream_t s) {
    const uint64_t n = (uint64_t)g.color_stride * 8u;
    if (n == 0) return cudaSuccess;
    const uint64_t blocks = (n + 127) / 128, wave = (uint64_t)resident_wave((const void*)k_propose_poly3);
    k_propose_poly3<<<(uint32_t)(blocks < wave ? blocks : wave), 128, 0, s>>>(g, a, l, rotate ? 1u : 0u);
    return cudaGetLastError();
}

cudaError_t launch_sweep_poly3_soft(const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                                    const ShapeOverlap& so, const Launch& l, cudaStream_t s) {
    if (l.n_active == 0) return cudaSuccess;
    PolyShape sh{verts, nv, so.rr, 0.f};
    const int wave = resident_wave((const void*)k_sweep_poly3_soft);
    uint32_t blocks = (l.n_active + 3) / 4;  // four warps (trials) per block
    if (blocks > (uint32_t)wave) blocks = (uint32_t)wave;
    PassLaunch pl(blocks, l.overlap_previous != 0 || l.early_wait != 0, s);
    return cudaLaunchKernelEx(&pl.cfg, k_sweep_poly3_soft, g, a, sh, so, l);
}

cudaError_t launch_energy_poly3_soft(const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                                     const ShapeOverlap& so, uint32_t n, double* out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    PolyShape sh{verts, nv, so.rr, 0.f};
    k_energy_poly3_soft<<<(n + 127) / 128, 128, 0, s>>>(g, a, sh, so, n, out);
    return cudaGetLastError();
}

cudaError_t launch_quick_insert_poly3(const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                                      const ShapeOverlap& so, const Launch& l, const QuickInsertArgs& q,
                                      const BodyTags& tags, const uint32_t* nc, const double* w, uint32_t cap,
                                      uint32_t* size, uint32_t* items, uint32_t* cell_of, double4* site,
                                      unsigned long long* out, cudaStream_t s) {
    const SerialGrid G = make_grid(3, nc, w, cap, size, items, cell_of, site);
    cudaError_t e = build_grid(3, g, a, G, q.n0, s);
    if (e != cudaSuccess) return e;
    PolyShape sh{verts, nv, so.rr, 0.f};
    k_quick_insert_poly3<<<1, 32, 0, s>>>(g, a, G, sh, so, l, q, tags, out);
    return cudaGetLastError();
}

cudaError_t launch_tune_stream_poly(TuneJob* jobs, uint32_t n_jobs, const double4* verts, uint32_t nv, double rcut2,
                                    cudaStream_t s) {
    if (n_jobs == 0) return cudaSuccess;
    k_tune_stream_poly3<<<n_jobs, 32, 0, s>>>(jobs, n_jobs, PolyShape{verts, nv, rcut2, 0.f, 0.f, 1.f});
    return cudaGetLastError();
}

namespace {
// Fixed-point sites (fixed_site): half a unit of L / 2^32 each, and FP64's own (a relative 2^-49 of L).
float site_error(const Geometry& g) {
    const double L = fmax(g.L[0], fmax(g.L[1], g.L[2]));
    return (float)(1.2 * L / 4294967296.0);
}
using PolyKernel = void (*)(Geometry, Arrays, PolyShape, Launch, uint32_t, Injected);
}  // namespace

cudaError_t launch_flow_poly(bool fp32, const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                             double rcut2, float rcut2_hi32, float bound_scale, const Launch& l, bool rotate,
                             cudaStream_t s, uint32_t variant) {
    if (l.n_active == 0) return cudaSuccess;
    const uint32_t rot = rotate ? 1u : 0u;
    const uint64_t entries = (uint64_t)g.color_stride * 8u * 4u;
    uint64_t blocks = (entries + 127) / 128;
    const uint64_t wave_d = (uint64_t)resident_wave((const void*)k_draw_poly3);
    PassLaunch pd((uint32_t)(blocks < wave_d ? blocks : wave_d), l.overlap_previous != 0, s);
    cudaError_t e = cudaLaunchKernelEx(&pd.cfg, k_draw_poly3, g, a, l, rot);
    if (e != cudaSuccess) return e;
    // the compiled launch variants, in the order of kPolyShapes
    static const PolyKernel kernels[2][2] = {{k_flow_poly3<false, false, 4>, k_flow_poly3<false, false, 3>},
                                             {k_flow_poly3<true, false, 4>, k_flow_poly3<true, false, 3>}};
    static_assert(n_shapes(kPolyShapes) == 2, "one compiled kernel per polyhedron variant");
    const PolyKernel k = kernels[fp32][variant < 2 ? variant : 0];
    const uint64_t wave = (uint64_t)resident_wave((const void*)k, 32 * kWarps);
    blocks = ((uint64_t)g.color_stride * 2 + kWarps * kGroup - 1) / (kWarps * kGroup);  // warps for two colours' units
    PassLaunch pl((uint32_t)(blocks < wave ? blocks : wave), l.overlap_previous != 0, s, 32 * kWarps);
    return cudaLaunchKernelEx(&pl.cfg, k, g, a, PolyShape{verts, nv, rcut2, rcut2_hi32, site_error(g), bound_scale}, l, rot,
                              Injected{});
}

cudaError_t launch_trials_poly(bool fp32, const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                               double rcut2, float rcut2_hi32, float bound_scale, const Injected& j, cudaStream_t s) {
    if (j.n == 0) return cudaSuccess;
    const PolyKernel k = fp32 ? k_flow_poly3<true, true, 1> : k_flow_poly3<false, true, 1>;
    const uint32_t wave = (uint32_t)resident_wave((const void*)k), n = (j.n + 4 * kGroup - 1) / (4 * kGroup);
    k<<<n < wave ? n : wave, 128, 0, s>>>(
        g, a, PolyShape{verts, nv, rcut2, rcut2_hi32, site_error(g), bound_scale}, Launch{}, 0u, j);
    return cudaGetLastError();
}

cudaError_t launch_eval_poly(bool fp32, const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv,
                             double rcut2, float rcut2_hi32, const uint64_t* bodies, const double4* trial,
                             const double4* trial_q, uint32_t n, uint8_t* decisions, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    PolyShape sh{verts, nv, rcut2, rcut2_hi32, 0.f, 1.f};
    const uint32_t blocks = (n + 3) / 4;
    if (fp32)
        k_eval_poly3<true><<<blocks, 128, 0, s>>>(g, a, sh, bodies, trial, trial_q, n, decisions);
    else
        k_eval_poly3<false><<<blocks, 128, 0, s>>>(g, a, sh, bodies, trial, trial_q, n, decisions);
    return cudaGetLastError();
}

cudaError_t launch_overlap_poly(const Geometry& g, const Arrays& a, const double4* verts, uint32_t nv, double rcut2,
                                uint32_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    PolyShape sh{verts, nv, rcut2, 0.f};
    k_overlap_poly3<<<(n + 127) / 128, 128, 0, s>>>(g, a, sh, n);
    return cudaGetLastError();
}

}  // namespace hmc

namespace hmc {
cudaError_t launch_tune_moves(int dim, const Geometry& g, const Arrays& a, const Launch& l, uint32_t tune_step,
                              uint32_t samples, bool rotate, uint64_t* bodies, double4* trial, double4* trial_q,
                              double* u, cudaStream_t s) {
    if (samples == 0) return cudaSuccess;
    const uint32_t blocks = (samples + 127) / 128;
    if (dim == 2)
        k_tune_moves<2><<<blocks, 128, 0, s>>>(g, a, l, tune_step, samples, rotate ? 1u : 0u, bodies, trial, trial_q, u);
    else
        k_tune_moves<3><<<blocks, 128, 0, s>>>(g, a, l, tune_step, samples, rotate ? 1u : 0u, bodies, trial, trial_q, u);
    return cudaGetLastError();
}
}  // namespace hmc
