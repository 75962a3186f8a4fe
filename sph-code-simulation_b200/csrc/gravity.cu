// gravity.cu — GravityForce::calculation (Barnes–Hut tree walk and the
// exhaustive direct sum).
//
// Reference: src/gravity_force.cpp:52-89, BHNode::calc_force
// (src/bhtree.cpp:347-393) and the Hernquist & Katz softening kernels f, g
// (src/bhtree.cpp:318-345).
//
// Per-lane stackless walk over the preorder node array: each lane (one
// particle; a warp holds 32 octree-consecutive particles) either accepts its
// current node as an (unsoftened) monopole and jumps over the subtree (skip
// pointer), or opens it — a leaf is then summed pairwise with spline-softened
// f and g and skipped, an internal node is descended into (index + 1).  Lanes
// follow their own paths, so a warp runs as many iterations as its longest
// walk rather than the union of its lanes' walks (1.5x faster on the Evrard
// sphere than a warp-synchronous union walk).  Each lane meets its nodes in
// exactly the order of the reference's recursion and adds into acc (starting
// from the fluid acceleration) in that order, so in the plain form with
// unfused FP64 (-fmad=false for this file) the result is bit-identical to the
// reference's on the same tree.  The mixed-precision walk is in
// gravity_mixed.cu (compiled with FMA contraction).
//
// What bounds it: issue slots and the FP64 pipe (0.56 M sphere: 66 % of the
// issue slots, FP64 pipe 58 %, 17 of 32 lanes per instruction).  An accepted
// node needs 1 / sqrt(d2) with both operations rounded as the reference's, an
// opened leaf a pair of spline kernels with ten quotients, on the few lanes
// that open one while the warp waits.  The roots and quotients are taken with
// Markstein's correction (rounded.cuh): no branch to a special-case path, so
// the chains of one term overlap, and quotients by h / 2 and its cube share
// one reciprocal per particle (k_half).  Measured (fixed state, one box, the
// general operations -> these): 17 K sphere 0.945 -> 0.52 ms, 137 K 2.00 ->
// 1.38, 1.1 M 13.2 -> 9.9, 4.2 M 47.7 -> 37.5; then 1 - 3 % more (1.1 M 10.1) for the
// divisors of all ones; without the softened pairs' arithmetic 7.3 ms on the 1.1 M
// sphere (timing-only copy).
// Measured and not kept (1.1 M sphere, against 9.9 ms): each lane's
// interactions queued in shared memory and summed a queue at a time, walk test
// in FP32 (13.2 ms; the queueing costs as many instructions as it aligns);
// sums and walk steps interleaved over a short ring with the softened pairs
// formed a warp at a time (14.5 ms); a union walk of the warp over blocks of
// siblings with per-lane queues (18.4 ms: 59 % of the lanes' slots used); the
// nodes laid out in sibling blocks (L1 hits 56 -> 84 %, same time: the walk
// does not wait on its loads); lanes that wait at an opened leaf for those
// behind them (12.7 ms).  With the general operations: pairs recorded and
// replayed in order (190 against 116 ms, 8.8 M sphere), lanes parked on opened
// leaves (169 ms and more), an accepted node's terms formed one iteration
// later (134 ms).  Kept from before: the squared edge of each level from a
// table, the next node's records loaded as soon as the test has chosen it.
#include <cuda_runtime.h>

#include "context.cuh"
#include "rounded.cuh"
#include "softening.cuh"

namespace sphgpu {

namespace {

// One warp per block.  Resident blocks per SM cap the registers: 20 (96
// registers) is best where they fill the chip (1.1 M sphere 9.9 ms; 16: 10.4,
// 24: 12.0, spilling), 16 (128 registers, more of a term's chains in flight)
// where a block's own latency counts: 17 K sphere 0.60 -> 0.52 ms, 137 K 1.45 ->
// 1.38.  The line is at four rounds of 16 blocks (148 x 16 x 32 x 4 particles).
constexpr int GBLK = 32;
constexpr int GFEW = 148 * 16 * GBLK * 4;

// Softened pair of the particles at distance rr = sqrt(r2): the sums
// f(rr, hi) + f(rr, hq) and g(rr, hi) + g(rr, hq) of hk_f and hk_g
// (softening.cuh), every operation and its order as there, the quotients taken
// as rounded products with reciprocals the terms share (rounded.cuh).
// k = {h / 2, (h / 2)^3 and their rounded reciprocals} (k_half).
__device__ __forceinline__ void hk_fg_rn(double r, double rinv, double r3, double r3i, const double4& k, double& f,
                                         double& g)
{
    const double u = quot_rn(r, k.x, k.z);
    const double u3 = u * u * u;
    const bool near = u < 1.0;
    // every branch's operations in their own order, selected at the end: no
    // branch in between, so the chains of both smoothing lengths overlap
    const double t = (near ? 3.0 / 20 : 0.3) * u * u;
    const double w = quot_rn(u3, near ? 20.0 : 30.0, near ? 1.0 / 20.0 : 1.0 / 30.0);
    const double p = near ? (1.0 / 3.0 - t) + w : (4.0 / 3.0 - u + t) - w;
    const double fe = quot_rn((near ? -0.5 : -1.0) * u * u * p + (near ? 1.4 : 1.6), k.x, k.z);
    const double r15 = 15 * r;
    const double fm = -recip_any(r15, rinv * (1.0 / 15.0)) + fe;
    const double gn = 4.0 / 3.0 - 1.2 * u * u + 0.5 * u * u * u;
    const double gm = -1.0 / 15 + 8.0 / 3 * u * u * u - 3.0 * u * u * u * u + 1.2 * u * u * u * u * u
        - quot_rn(u3 * u * u * u, 6.0, 1.0 / 6.0);
    const double gq = quot_rn(near ? gn : gm, near ? k.y : r3, near ? k.w : r3i);
    f = near ? fe : (u < 2.0 ? fm : rinv);
    g = u < 2.0 ? gq : r3i;
}
// Smoothing lengths, and squared distances, for which no operation above
// leaves the middle of the exponent range.
__device__ __forceinline__ bool pair_range(double x) { return x > 0x1p-80 && x < 0x1p80; }

// {e, e^3, 1 / e, 1 / e^3}, e = h / 2, of every particle
__global__ void k_half(DevState S, int n, double4* __restrict__ half)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const double h = S.vel[i].w, e = h * 0.5, e3 = e * e * e;
    half[i] = pair_range(h) && !all_ones(e) && !all_ones(e3) ? make_double4(e, e3, recip_rn(e), recip_rn(e3))
                                                             : make_double4(-1.0, 0.0, 0.0, 0.0);
}

// subset != null: only the listed particles (the mixed form's FP64
// re-evaluation); those launches add to no work counter.
template <bool PER, int RES>
__global__ void __launch_bounds__(GBLK, RES) k_gravity(DevParams P, DevState S, DevTree Tr,
                                                        const double4* __restrict__ half, int n,
                                                        DevStatus* __restrict__ st, const int* __restrict__ subset,
                                                        int nsub)
{
    const int slot = blockIdx.x * GBLK + threadIdx.x;
    const bool valid = slot < (subset ? nsub : n);
    const int i = subset ? (valid ? subset[slot] : n) : slot;
    double xi = 0, yi = 0, zi = 0;
    double4 acc = make_double4(0, 0, 0, 0);
    if(valid) {
        const double4 p = S.pos[i];
        xi = p.x;
        yi = p.y;
        zi = p.z;
        acc = S.acc[i];
    }
    double ax = acc.x, ay = acc.y, az = acc.z, phi = 0.0;
    const double G = P.G;
    const int nnodes = *Tr.nnodes;
    // node edges halve exactly per level: edge(L) = root edge * 2^(1 - L);
    // the squared edge of every level (at most 22), as the opening test forms it
    __shared__ double s_l2[32];
    {
        const double e = ldexp(ldg4(&Tr.geo[0]).w, 1 - (int)threadIdx.x);
        s_l2[threadIdx.x] = e * e;
        __syncwarp();
    }
    auto offset = [&](const double4& c) {
        Vec3d d{xsub(xi, c.x), xsub(yi, c.y), xsub(zi, c.z)};
        if(PER) {
            d.x = min_image(d.x, P.range[0]);
            d.y = min_image(d.y, P.range[1]);
            d.z = min_image(d.z, P.range[2]);
        }
        return d;
    };
    int nd = valid ? 0 : nnodes, steps = 0;
    unsigned n_mono = 0, n_leaf = 0;  // work counters of this lane (steps = nodes met)
    // the records of the node in hand; the next node's are loaded as soon as
    // the opening test has chosen it, before this node's terms are formed
    int4 lk = make_int4(0, 0, nnodes, 0);
    double4 mc = make_double4(0, 0, 0, 0);
    if(nd < nnodes) {
        lk = __ldg(&Tr.link[nd]);
        mc = ldg4(&Tr.mass[nd]);
    }
    while(nd < nnodes) {
        if(++steps > nnodes) {  // corrupt node table: report, never loop
            atomicOr(&st->pass_guard, PASS_GUARD_GRAVITY);
            break;
        }
        const bool leaf = (lk.w >> 8) != 0;
        const Vec3d d = offset(mc);
        const double l2 = s_l2[lk.w & 31];
        const double d2 = d.x * d.x + d.y * d.y + d.z * d.z;
        const bool open = (l2 > P.theta2 * d2) || (d2 < l2);
        const int next = (open && !leaf) ? nd + 1 : lk.z;
        int4 lk_n = lk;
        double4 mc_n = mc;
        if(next < nnodes) {
            lk_n = __ldg(&Tr.link[next]);
            mc_n = ldg4(&Tr.mass[next]);
        }
        if(!open) {
            ++n_mono;
            double rinv;
            if(mid_range(d2) && root_not_ones(d2)) {
                const double y = rsqrt_near(d2);
                rinv = recip_rn(root_rn(d2, y), y);
            } else {
                rinv = 1.0 / sqrt(d2);
            }
            phi -= G * mc.w * rinv;
            const double s = G * mc.w * (rinv * rinv * rinv);
            ax -= d.x * s;
            ay -= d.y * s;
            az -= d.z * s;
        }
        if(open && leaf) {
            for(int q = lk.x; q < lk.y; ++q) {
                if(q == i) continue;
                ++n_leaf;
                const double4 pq = ldg4(&S.pos[q]);
                const double4 kq = ldg4(&half[q]), ki = ldg4(&half[i]);
                const Vec3d r = offset(pq);
                const double r2 = r.x * r.x + r.y * r.y + r.z * r.z;
                double f1, f2, g1, g2;
                if(pair_range(r2) && root_not_ones(r2) && ki.x > 0.0 && kq.x > 0.0) {
                    const double y = rsqrt_near(r2);
                    const double rr = root_rn(r2, y);
                    const double rinv = recip_rn(rr, y);
                    const double r3 = rr * rr * rr;
                    const double r3i = recip_any(r3, y * y * y);
                    hk_fg_rn(rr, rinv, r3, r3i, ki, f1, g1);
                    hk_fg_rn(rr, rinv, r3, r3i, kq, f2, g2);
                } else {
                    const double rr = sqrt(r2), hi = S.vel[i].w, hq = __ldg(&S.vel[q].w);
                    f1 = hk_f<double>(rr, hi);
                    f2 = hk_f<double>(rr, hq);
                    g1 = hk_g<double>(rr, hi);
                    g2 = hk_g<double>(rr, hq);
                }
                phi -= G * pq.w * (f1 + f2) * 0.5;
                const double c = G * pq.w * (g1 + g2) * 0.5;
                ax -= r.x * c;
                ay -= r.y * c;
                az -= r.z * c;
            }
        }
        nd = next;
        lk = lk_n;
        mc = mc_n;
    }
    if(valid) {
        S.acc[i] = make_double4(ax, ay, az, acc.w);
        S.visc[i].w = phi;
    }
    if(subset) return;
    block_count(&st->grav_nodes, (unsigned)min(steps, nnodes));
    block_count(&st->grav_mono, n_mono);
    block_count(&st->grav_leaf_pairs, n_leaf);
}

// -DEXHAUSTIVE_SEARCH direct summation (src/gravity_force.cpp:70-84): every j
// in caller-index order, self included.
__global__ void k_gravity_direct(DevParams P, DevState S, int n, const int* __restrict__ inv)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const double4 p = S.pos[i];
    const double hi = S.vel[i].w;
    const double G = P.G;
    double phi = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
    for(int jid = 0; jid < n; ++jid) {
        const int j = inv[jid];
        const double4 pj = S.pos[j];
        const double hj = S.vel[j].w;
        const Vec3d r = rij(P, p.x, p.y, p.z, pj.x, pj.y, pj.z);
        const double rr = sqrt(r.x * r.x + r.y * r.y + r.z * r.z);
        phi -= G * pj.w * (hk_f<double>(rr, hi) + hk_f<double>(rr, hj)) * 0.5;
        const double c = G * pj.w * (hk_g<double>(rr, hi) + hk_g<double>(rr, hj)) * 0.5;
        fx -= r.x * c;
        fy -= r.y * c;
        fz -= r.z * c;
    }
    double4 a = S.acc[i];
    a.x += fx;
    a.y += fy;
    a.z += fz;
    S.acc[i] = a;
    S.visc[i].w = phi;
}

}  // namespace

// The particles' half kernels (of the smoothing lengths as they are now).
static int gravity_half(sphgpu_ctx* c)
{
    k_half<<<grid_for(c->n, 256), 256, 0, c->stream>>>(c->s, c->n, c->d_half);
    SPHGPU_LAUNCH_CHECK(c, "gravity half kernels");
    return SPHGPU_OK;
}

static void launch_gravity(sphgpu_ctx* c, const int* subset, int count)
{
    const bool few = count <= GFEW;
    auto* k = c->prm.periodic ? (few ? k_gravity<true, 16> : k_gravity<true, 20>)
                              : (few ? k_gravity<false, 16> : k_gravity<false, 20>);
    k<<<grid_for(count, GBLK), GBLK, 0, c->stream>>>(c->dp, c->s, c->t, c->d_half, c->n, c->d_status, subset,
                                                     subset ? count : 0);
}

int gravity(sphgpu_ctx* c, bool direct)
{
    // the mixed form's FP64 re-evaluation follows the last module that
    // writes acc (recheck.cu); GravityForce runs every step, with gravity off too
    if(!c->prm.use_gravity) return direct ? SPHGPU_OK : mixed_recheck(c);
    if(!direct && !c->have_tree) return fail(c, SPHGPU_ERR_STATE, "GravityForce before tree make");
    if(!direct && c->prm.precision == SPHGPU_MIXED) {
        // the walk's FP32 node records: tree data, timed with the tree
        stage_begin(c, SPHGPU_T_TREE);
        const int rc = gravity_nodes_mixed(c);
        if(rc < 0) return rc;
        stage_end(c, SPHGPU_T_TREE, 1);
    } else if(!direct) {
        stage_begin(c, SPHGPU_T_TREE);
        const int rc = gravity_half(c);
        if(rc < 0) return rc;
        stage_end(c, SPHGPU_T_TREE, 1);
    }
    stage_begin(c, SPHGPU_T_GRAVITY);
    if(direct) {
        k_gravity_direct<<<grid_for(c->n, 128), 128, 0, c->stream>>>(c->dp, c->s, c->n, c->d_inv);
    } else if(c->prm.precision == SPHGPU_MIXED) {
        const int rc = gravity_walk_mixed(c);
        if(rc < 0) return rc;
    } else {
        launch_gravity(c, nullptr, c->n);
    }
    SPHGPU_LAUNCH_CHECK(c, "GravityForce");
    stage_end(c, SPHGPU_T_GRAVITY, 1);
    return direct ? SPHGPU_OK : mixed_recheck(c);
}

int gravity_subset64(sphgpu_ctx* c, const int* idx, int nsub)
{
    if(!c->prm.use_gravity || nsub <= 0) return SPHGPU_OK;
    const int rc = gravity_half(c);
    if(rc < 0) return rc;
    launch_gravity(c, idx, nsub);
    SPHGPU_LAUNCH_CHECK(c, "GravityForce (FP64 re-evaluation)");
    return SPHGPU_OK;
}

}  // namespace sphgpu
