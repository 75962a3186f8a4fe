// pre.cu — PreInteraction::calculation for ssph, disph, gsph and gdisph.
//
// Reference: src/pre_interaction.cpp:39-283 (ssph, initial_smoothing,
// newton_raphson), src/disph/d_pre_interaction.cpp:21-230 (disph),
// src/gsph/g_pre_interaction.cpp:27-144 (gsph), src/gdisph/gd_pre_interaction.cpp:
// 29-280 (gdisph: the disph smoothing length, density and pressure, the gsph
// MUSCL gradients, a mass-weighted Balsara switch normalised by density, and
// without it the implicit alpha update weighted by mass x energy).
//
// A group of G lanes owns one particle and strides over its gather list
// (ELL row, coalesced index loads; neighbour state as 32-byte double4 loads
// that mostly hit L1/L2 because neighbours are close in octree order).
//   1. Newton-Raphson on h (<= 10 iterations, |dh| < 1e-4 (h + h_b)) over the
//      candidates with r < h, group-reduced each iteration;
//   2. one fused pass at the final h (disph: over the candidates the last
//      sweep kept, within (1 + 4e-4) of its h): density (and the DISPH number/pressure
//      sums), grad-h sums, max signal speed, neighbour count, the Balsara
//      div/curl sums and the GSPH MUSCL gradients — every quantity the
//      reference computes in separate loops over the same set {r < h};
//   3. per-particle epilogue (P, grad-h, Balsara, time-dependent alpha) and
//      the block-reduced minimum of h / v_sig.
// The set predicates (r computed from the unfused FP64 r^2, r < h) match the
// reference exactly; sums are taken in a different order than the
// reference's distance-sorted loop, so results agree to rounding.
// k_pre: plain FP64 form.  k_pre_mixed: pair arithmetic and sums in FP32; h,
// its Newton update and the predicates stay FP64.
// What bounds it: issue slots and the FP64 pipe with 16 warps per SM in flight,
// waiting on the neighbour loads and the FP64 chains (1.1 M disph sphere, FP64,
// before: 43 % of the issue slots, FP64 pipe 38 %, 14 % of the stalls on
// instruction fetch).  The kernel function and the periodic box are compile-
// time (three kernels' code in one loop missed the instruction cache), two
// candidates are evaluated and masked per iteration instead of branched on one
// after the other, 1 / r comes from a branch-free refinement, and the factors
// that depend on h alone leave the sums.  Measured (before -> now): disph FP64
// 1.1 M sphere 3.79 -> 2.69 ms, 1 M shear layer 4.22 -> 2.83,
// 2 M gsph tube 3.50 -> 2.61, 244 K gdisph tube 0.551 -> 0.458, 17 K ssph sphere
// 0.052 -> 0.033.  Loading the next positions one iteration ahead as well (not
// only their indices) was slower before: the extra live records spill.
#include <cfloat>
#include <cuda_runtime.h>

#include "context.cuh"
#include "rounded.cuh"

namespace sphgpu {

namespace {

constexpr double AREA3 = 4.0 * 3.14159265358979323846 / 3.0;  // A for DIM = 3
constexpr int PBLK = 256;

__device__ __forceinline__ double exact_r(const DevParams& P, double xi, double yi, double zi, double4 pj,
                                          Vec3d& d)
{
    d = rij(P, xi, yi, zi, pj.x, pj.y, pj.z);
    return sqrt(abs2x(d));
}

// Minimum image without a branch: the candidate min_image takes (d while
// |d| <= L / 2; beyond, d - L or d + L by the sign of d).
__device__ __forceinline__ double image_of(double d, double L)
{
    const double b = d > 0.0 ? xsub(d, L) : xadd(d, L);
    return fabs(d) <= 0.5 * L ? d : b;
}

// x_i - x_j with the periodic form decided at compile time
template <bool PER>
__device__ __forceinline__ Vec3d offset_of(const DevParams& P, const double4& pi, const double4& pj)
{
    Vec3d d{xsub(pi.x, pj.x), xsub(pi.y, pj.y), xsub(pi.z, pj.z)};
    if constexpr(PER) {
        d.x = image_of(d.x, P.range[0]);
        d.y = image_of(d.y, P.range[1]);
        d.z = image_of(d.z, P.range[2]);
    }
    return d;
}

// r and 1 / r of a pair from one reciprocal square root good to an ulp
// (rounded.cuh); both 0 for r = 0 (and below 2^-500, where the kernels cannot
// tell r from 0).
__device__ __forceinline__ void pair_distance(double r2, double& r, double& rinv)
{
    const double y = rsqrt_near(r2);
    const bool some = r2 >= 0x1p-1000;
    rinv = some ? y : 0.0;
    r = some ? r2 * y : 0.0;
}

// The pair predicate r < h of one smoothing length on r^2 (root_lt): sure
// outside the band lo .. hi around h^2.
struct Within {
    double h, lo, hi;
    __device__ __forceinline__ explicit Within(double h_) : h(h_), lo(h_ * h_ * (1.0 - 0x1p-40)), hi(h_ * h_ * (1.0 + 0x1p-40)) {}
    __device__ __forceinline__ bool sure(double r2) const { return r2 < lo; }
    __device__ __forceinline__ bool unsure(double r2) const { return !(r2 < lo) && r2 <= hi; }
};

// A pair sum times the factor of h left out of its terms; no pairs, no sum (h of
// 0 or NaN, from a mass of zero or a bad density guess, has no finite factor).
__device__ __forceinline__ double scaled(bool some, double sum, double factor) { return some ? sum * factor : 0.0; }

// Two resident blocks per SM (128 registers a thread): with two candidates in
// flight fewer registers spill (4 blocks of 128 threads: 2.69 -> 2.74 ms on the
// 1.1 M sphere; 5: 2.81).
constexpr int PRE_BLOCKS = 2;

// skin_delta > 0: the lists are skin lists (supersets of the gather lists);
// a particle whose h reaches R - skin_delta (R = its gather radius, the sml
// the walk left) takes only exact members (gather_member).
// KER, PER: the kernel function and the periodic box at compile time.
template <int G, int TYPE, int KER, bool PER>
__global__ void __launch_bounds__(PBLK, PRE_BLOCKS) k_pre(DevParams P, DevState S, int n, const int* __restrict__ list,
                                              const int* __restrict__ count, int cap, const double* __restrict__ dtp,
                                              double* __restrict__ hvs, DevStatus* __restrict__ st, DevTree Tr,
                                              double skin_delta, int* __restrict__ scratch, int scap)
{
    constexpr int GPW = 32 / G;
    const int lane = threadIdx.x & (G - 1);
    const long long warp = ((long long)blockIdx.x * PBLK + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * PBLK) >> 5;
    const double dt = *dtp;
    constexpr bool gdisph = TYPE == SPHGPU_GDISPH;
    const bool disph = TYPE == SPHGPU_DISPH || gdisph, gsph = TYPE == SPHGPU_GSPH;
    // AV switch sums weighted by m_j u_j and normalised by (gamma - 1) / P
    // (disph; gdisph without the Balsara switch), else by m_j and 1 / rho
    const bool av_energy = disph && !(gdisph && P.balsara);
    double hv_min = DBL_MAX;
    unsigned nonconv = 0;
    unsigned n_cand = 0, n_newton = 0, n_pairs = 0, n_list = 0;  // work counters of this lane

    for(long long wb = warp * GPW; wb < n; wb += nwarps * GPW) {
        const int i = (int)(wb + ((threadIdx.x & 31) / G));
        const bool valid = i < n;
        const int cnt = valid ? min(count[i], cap) : 0;
        const int* li = list + (size_t)(valid ? i : 0) * (size_t)cap;
        const double4 pi = valid ? S.pos[i] : make_double4(0, 0, 0, 0);
        const double4 vi = valid ? S.vel[i] : make_double4(0, 0, 0, 1);
        const double4 ti = valid ? S.thermo[i] : make_double4(1, 0, 0, 0);
        const double sml0 = vi.w;

        // ---- 1. smoothing length (src/pre_interaction.cpp:227-283,
        //         src/disph/d_pre_interaction.cpp:174-230)
        double h = sml0;
        // disph: each sweep also keeps, per lane and in the lane's own order,
        // the candidates within (1 + 4e-4) h in a scratch row; after a
        // converged sweep (|h_new - h| < 1e-4 (h_new + h), so h_new <
        // (1 + 2.0003e-4) h) they hold every pair of the fused pass, which
        // then reads them instead of the whole list (8.78 M sphere: pre 31.8
        // -> 30.8 ms FP64, 27.4 -> 24.1 ms FP32 when it came; the gsph and
        // gdisph bodies spilled with it and ran slower)
        constexpr bool keep = TYPE == SPHGPU_DISPH;
        int* srow = scratch + (size_t)(valid ? i : 0) * (size_t)scap;
        int nk = 0;
        bool conv = false;
        if(P.iterative) {
            h = sml0 / P.ratio;
            const double b = disph ? P.nngb / AREA3 : pi.w * P.nngb / AREA3;
            for(int it = 0; it < 10; ++it) {
                const double hb = h;
                double d = 0, dd = 0;
                const KernH<double> kh(KER, h);
                const Within in(h);
                const bool exact = skin_delta > 0.0 && !(h < sml0 - skin_delta);
                const double hk = h * (1.0 + 4e-4), keep2 = hk * hk;
                nk = 0;
                // Two candidates per iteration, both evaluated and masked: some
                // lane of a warp is nearly always inside, so a branch would
                // save nothing, and the two chains overlap.  Their indices are
                // fetched an iteration ahead.
                int ja = lane < cnt ? __ldg(&li[lane]) : 0;
                int jb = lane + G < cnt ? __ldg(&li[lane + G]) : 0;
                n_cand += lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u;
                for(int k = lane; k < cnt; k += 2 * G) {
                    const int ca = ja, cb = jb;  // cb is a valid index even past the list end
                    const bool two = k + G < cnt;
                    if(k + 2 * G < cnt) ja = __ldg(&li[k + 2 * G]);
                    if(k + 3 * G < cnt) jb = __ldg(&li[k + 3 * G]);
                    const double4 pa = ldg4(&S.pos[ca]);
                    const double4 pb = ldg4(&S.pos[cb]);
                    const double r2a = abs2x(offset_of<PER>(P, pi, pa)), r2b = abs2x(offset_of<PER>(P, pi, pb));
                    if constexpr(keep) {
                        if(r2a < keep2) srow[lane + G * nk++] = ca;
                        if(two && r2b < keep2) srow[lane + G * nk++] = cb;
                    }
                    bool ia = in.sure(r2a), ib = two && in.sure(r2b);
                    const bool ua = in.unsure(r2a), ub = two && in.unsure(r2b);
                    if(ua || ub || (exact && (ia || ib))) {  // rare
                        if(ua) ia = sqrt(r2a) < h;
                        if(ub) ib = sqrt(r2b) < h;
                        if(exact && ia) ia = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, ca, r2a);
                        if(exact && ib) ib = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, cb, r2b);
                    }
                    double ra, rb, ya, yb;
                    pair_distance(r2a, ra, ya);
                    pair_distance(r2b, rb, yb);
                    n_newton += (ia ? 1u : 0u) + (ib ? 1u : 0u);
                    const Shape<double, KER> sa(ra * kh.inv, ia), sb(rb * kh.inv, ib);
                    if(disph) {
                        d += sa.w();
                        dd += sa.dh();
                        d += sb.w();
                        dd += sb.dh();
                    } else {
                        const double ma = ia ? pa.w : 0.0, mb = ib ? pb.w : 0.0;
                        d += ma * sa.w();
                        dd += ma * sa.dh();
                        d += mb * sb.w();
                        dd += mb * sb.dh();
                    }
                }
                const double d0 = group_sum<G>(d);
                const double ds = scaled(d0 != 0.0, d0, kh.wn), dds = scaled(d0 != 0.0, group_sum<G>(dd), kh.dhn);
                const double h3 = h * h * h;
                const double f = ds * h3 - b;
                const double df = dds * h3 + 3 * ds * (h * h);
                h -= f / df;
                if(fabs(h - hb) < (h + hb) * 1e-4) {
                    conv = true;
                    break;
                }
            }
            if(!conv) {
                h = sml0 / P.ratio;
                if(valid && lane == 0) ++nonconv;
            }
        }

        // ---- 2. fused pass over {r < h}
        const KernH<double> kh(KER, h);
        const Within in(h);
        double dens = 0, dhd = 0, ni = 0, pres = 0, dhp = 0, dhn = 0;
        double divv = 0, rx = 0, ry = 0, rz = 0;
        double gd[3] = {0, 0, 0}, gu[3] = {0, 0, 0}, gv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        double vsig = ti.w * 2.0;
        int nn = 0;
        const bool need_av = !gsph && (P.balsara || P.td_av);
        const bool need_grad = (gsph || gdisph) && P.gsph2;
        const bool exact = skin_delta > 0.0 && !(h < sml0 - skin_delta);
        n_list += lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u;
        const bool kept = keep && conv;
        n_cand += kept ? (unsigned)nk : (lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u);
        // one candidate, evaluated and masked (`use`: it is in the list): what
        // is outside adds zeros
        struct Pair {
            Vec3d dv;
            double r2;
            bool in;
            double4 v, t;
        };
        auto load = [&](const double4& pj, int j, bool use) {
            Pair q;
            q.dv = offset_of<PER>(P, pi, pj);
            q.r2 = abs2x(q.dv);
            q.in = use && in.sure(q.r2);
            const bool unsure = use && in.unsure(q.r2);
            if(unsure || (exact && q.in)) {  // rare
                if(unsure) q.in = sqrt(q.r2) < h;
                if(exact && q.in) q.in = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, j, q.r2);
            }
            // coherent loads: this kernel writes vel.w and thermo.x, .y of every
            // particle (the components read here, velocity, u and c_s, it
            // does not change)
            q.v = q.t = make_double4(0, 0, 0, 0);
            if(q.in) {
                q.v = S.vel[j];
                q.t = S.thermo[j];
            }
            return q;
        };
        auto add = [&](const double4& pj, int j, const Pair& q) {
            double rT, rinvT;
            pair_distance(q.r2, rT, rinvT);
            if(q.r2 < 0x1p-1000 && q.r2 > 0.0) {  // rare: v_sig needs v . r / r of these too
                rinvT = rsqrt(q.r2);
                rT = q.r2 * rinvT;
            }
            nn += q.in ? 1 : 0;
            const Shape<double, KER> sh(rT * kh.inv, q.in);
            const double w = sh.w();
            const double mj = q.in ? pj.w : 0.0;  // (a mass that is no number stays outside too)
            if(disph) {
                const double dh = sh.dh();
                const double uj = q.t.z;
                dens += mj * w;
                ni += w;
                pres += mj * uj * w;
                dhp += mj * uj * dh;
                dhn += dh;
            } else {
                dens += mj * w;
                if(!gsph) dhd += mj * sh.dh();
            }
            {
                const double vr = q.dv.x * (vi.x - q.v.x) + q.dv.y * (vi.y - q.v.y) + q.dv.z * (vi.z - q.v.z);
                // coincident particles (r = 0): the reference's vr / r is
                // 0 / 0, a NaN that never raises v_sig (+-inf if r underflowed)
                const double v = rT > 0.0 ? ti.w + q.t.w - 3.0 * vr * (double)rinvT
                                           : (vr < 0.0 ? (double)INFINITY : -(double)INFINITY);
                if(q.in && i != j && v > vsig) vsig = v;
            }
            if(need_av || need_grad) {
                const double c = sh.dw(rinvT);
                const double dwx = q.dv.x * c, dwy = q.dv.y * c, dwz = q.dv.z * c;
                const double vx = (vi.x - q.v.x), vy = (vi.y - q.v.y), vz = (vi.z - q.v.z);
                if(need_av) {
                    const double wgt = av_energy ? mj * q.t.z : mj;
                    divv -= wgt * (vx * dwx + vy * dwy + vz * dwz);
                    rx += (vy * dwz - vz * dwy) * wgt;
                    ry += (vz * dwx - vx * dwz) * wgt;
                    rz += (vx * dwy - vy * dwx) * wgt;
                }
                if(need_grad) {
                    const double du = mj * (q.t.z - ti.z);
                    gd[0] += dwx * mj;
                    gd[1] += dwy * mj;
                    gd[2] += dwz * mj;
                    gu[0] += dwx * du;
                    gu[1] += dwy * du;
                    gu[2] += dwz * du;
                    // dv[k] += dw * (m_j (v_j[k] - v_i[k]))
                    const double m0 = -mj * vx, m1 = -mj * vy, m2 = -mj * vz;
                    gv[0] += dwx * m0;
                    gv[1] += dwy * m0;
                    gv[2] += dwz * m0;
                    gv[3] += dwx * m1;
                    gv[4] += dwy * m1;
                    gv[5] += dwz * m1;
                    gv[6] += dwx * m2;
                    gv[7] += dwy * m2;
                    gv[8] += dwz * m2;
                }
            }
        };
        if(kept) {
            // the lane's kept candidates, in its own order (the same sums)
            for(int m = 0; m < nk; m += 2) {
                const bool two = m + 1 < nk;
                const int ca = srow[lane + G * m], cb = two ? srow[lane + G * (m + 1)] : ca;
                const double4 pa = ldg4(&S.pos[ca]), pb = ldg4(&S.pos[cb]);
                const Pair qa = load(pa, ca, true), qb = load(pb, cb, two);
                add(pa, ca, qa);
                add(pb, cb, qb);
            }
        } else {
            int ja = lane < cnt ? __ldg(&li[lane]) : 0;
            int jb = lane + G < cnt ? __ldg(&li[lane + G]) : 0;
            for(int k = lane; k < cnt; k += 2 * G) {
                const int ca = ja, cb = jb;  // cb is a valid index even past the list end
                const bool two = k + G < cnt;
                if(k + 2 * G < cnt) ja = __ldg(&li[k + 2 * G]);
                if(k + 3 * G < cnt) jb = __ldg(&li[k + 3 * G]);
                const double4 pa = ldg4(&S.pos[ca]), pb = ldg4(&S.pos[cb]);
                const Pair qa = load(pa, ca, true), qb = load(pb, cb, two);
                add(pa, ca, qa);
                add(pb, cb, qb);
            }
        }
        n_pairs += (unsigned)nn;
        nn = group_sum<G>(nn);
        const bool some = nn > 0;
        const double densS = scaled(some, group_sum<G>(dens), kh.wn);
        vsig = group_max<G>(vsig);
        double dhdS = 0, niS = 0, presS = 0, dhpS = 0, dhnS = 0;
        if(disph) {
            niS = scaled(some, group_sum<G>(ni), kh.wn);
            presS = scaled(some, group_sum<G>(pres), kh.wn);
            dhpS = scaled(some, group_sum<G>(dhp), kh.dhn);
            dhnS = scaled(some, group_sum<G>(dhn), kh.dhn);
        } else if(!gsph) {
            dhdS = scaled(some, group_sum<G>(dhd), kh.dhn);
        }
        double divS = 0, rxS = 0, ryS = 0, rzS = 0;
        if(need_av) {
            divS = scaled(some, group_sum<G>(divv), kh.dwn);
            rxS = scaled(some, group_sum<G>(rx), kh.dwn);
            ryS = scaled(some, group_sum<G>(ry), kh.dwn);
            rzS = scaled(some, group_sum<G>(rz), kh.dwn);
        }
        double gdS[3], guS[3], gvS[9];
        if(need_grad) {
#pragma unroll
            for(int k = 0; k < 3; ++k) {
                gdS[k] = scaled(some, group_sum<G>(gd[k]), kh.dwn);
                guS[k] = scaled(some, group_sum<G>(gu[k]), kh.dwn);
            }
#pragma unroll
            for(int k = 0; k < 9; ++k) gvS[k] = scaled(some, group_sum<G>(gv[k]), kh.dwn);
        }

        // ---- 3. epilogue (lane 0 of the group writes)
        if(!valid || lane != 0) continue;
        const double gamma = P.gamma;
        const double ui = ti.z, ci = ti.w;
        double pres_i;
        double4 vs = S.visc[i];
        if(disph) {
            pres_i = (gamma - 1.0) * presS;
            vs.z = h / (3 * niS) * dhpS / (1.0 + h / (3 * niS) * dhnS);
        } else {
            pres_i = (gamma - 1.0) * densS * ui;
            if(!gsph) vs.z = 1.0 / (1.0 + h / (3 * densS) * dhdS);
        }
        S.thermo[i] = make_double4(densS, pres_i, ui, ci);
        S.vel[i].w = h;
        S.nbr[i] = nn;
        const double hv = h / vsig;
        if(hv < hv_min) hv_min = hv;
        if(need_av) {
            // Balsara switch and time-dependent alpha (src/pre_interaction.cpp:115-161,
            // src/disph/d_pre_interaction.cpp:106-154)
            double dv_ = divS, r0 = rxS, r1 = ryS, r2 = rzS;
            if(av_energy) {
                const double pinv = (gamma - 1.0) / pres_i;
                dv_ *= pinv;
                r0 *= pinv;
                r1 *= pinv;
                r2 *= pinv;
            } else {
                dv_ /= densS;
                r0 /= densS;
                r1 /= densS;
                r2 /= densS;
            }
            if(P.balsara) {
                const double rot = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
                vs.y = fabs(dv_) / (fabs(dv_) + rot + 1e-4 * ci / h);
                if(P.td_av) {
                    const double tau = P.eps_av * ci / h;
                    const double da = (-(vs.x - P.alpha_min) * tau + fmax(-dv_, 0.0) * (P.alpha_max - vs.x)) * dt;
                    vs.x += da;
                }
            } else {
                const double tau = P.eps_av * ci / h;
                const double s = fmax(-dv_, 0.0);
                vs.x = (vs.x + dt * tau * P.alpha_min + s * dt * P.alpha_max) / (1.0 + dt * tau + s * dt);
            }
        }
        S.visc[i] = vs;
        if(need_grad) {
            // MUSCL gradients (src/gsph/g_pre_interaction.cpp:112-136)
            const double gm1 = gamma - 1.0, rinv = 1.0 / densS;
            const double g15[15] = {gdS[0],
                                    gdS[1],
                                    gdS[2],
                                    (gdS[0] * ui + guS[0]) * gm1,
                                    (gdS[1] * ui + guS[1]) * gm1,
                                    (gdS[2] * ui + guS[2]) * gm1,
                                    gvS[0] * rinv,
                                    gvS[1] * rinv,
                                    gvS[2] * rinv,
                                    gvS[3] * rinv,
                                    gvS[4] * rinv,
                                    gvS[5] * rinv,
                                    gvS[6] * rinv,
                                    gvS[7] * rinv,
                                    gvS[8] * rinv};
            S.grad[i] = make_double4(g15[0], g15[1], g15[2], g15[3]);
            S.grad[(size_t)n + i] = make_double4(g15[4], g15[5], g15[6], g15[7]);
            S.grad[2 * (size_t)n + i] = make_double4(g15[8], g15[9], g15[10], g15[11]);
            S.grad[3 * (size_t)n + i] = make_double4(g15[12], g15[13], g15[14], 0.0);
        }
    }
    // block reductions: min h / v_sig, Newton fallbacks
    __shared__ double s_min[PBLK / 32];
    __shared__ unsigned s_nc[PBLK / 32];
    hv_min = warp_min(hv_min);
    for(int o = 16; o > 0; o >>= 1) nonconv += __shfl_xor_sync(FULL_MASK, nonconv, o);
    if((threadIdx.x & 31) == 0) {
        s_min[threadIdx.x >> 5] = hv_min;
        s_nc[threadIdx.x >> 5] = nonconv;
    }
    __syncthreads();
    if(threadIdx.x == 0) {
        double m = s_min[0];
        unsigned c = s_nc[0];
        for(int w = 1; w < PBLK / 32; ++w) {
            m = fmin(m, s_min[w]);
            c += s_nc[w];
        }
        if(m < DBL_MAX) atomic_min_pos(hvs, m);
        if(c) atomicAdd(&st->newton_nonconv, (unsigned long long)c);
    }
    block_count(&st->pre_cand, n_cand);
    block_count(&st->pre_newton_pairs, n_newton);
    block_count(&st->pre_pairs, n_pairs);
    block_count(&st->pre_list, n_list);
}

// The mixed form: pair arithmetic and sums in FP32.  A kernel of its own: the
// smoothing length follows the rounding of the FP32 sums, and with it which
// pairs lie inside (a move of h by 1e-7 takes a handful of pairs in a million
// particles across the kernel's edge), so its operations and their fusing are
// spelt out and stay as they are.  What changed around them: two candidates are
// evaluated and masked per iteration, the box and the kernel function are
// compile-time, and two resident blocks leave registers for both candidates
// (1.1 M disph sphere 3.00 -> 2.75 ms, 131 K shear layer 0.477 -> 0.398, 493 K
// ssph sphere 0.69 -> 0.59, 1 M gsph tube 1.54 -> 1.30, gdisph 1.92 -> 1.47).
template <int G, int TYPE, int KER, bool PER>
__global__ void __launch_bounds__(PBLK, PRE_BLOCKS) k_pre_mixed(DevParams P, DevState S, int n, const int* __restrict__ list,
                                              const int* __restrict__ count, int cap, const double* __restrict__ dtp,
                                              double* __restrict__ hvs, DevStatus* __restrict__ st, DevTree Tr,
                                              double skin_delta, int* __restrict__ scratch, int scap)
{
    using T = float;
    constexpr int GPW = 32 / G;
    const int lane = threadIdx.x & (G - 1);
    const long long warp = ((long long)blockIdx.x * PBLK + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * PBLK) >> 5;
    const double dt = *dtp;
    constexpr bool gdisph = TYPE == SPHGPU_GDISPH;
    const bool disph = TYPE == SPHGPU_DISPH || gdisph, gsph = TYPE == SPHGPU_GSPH;
    // AV switch sums weighted by m_j u_j and normalised by (gamma - 1) / P
    // (disph; gdisph without the Balsara switch), else by m_j and 1 / rho
    const bool av_energy = disph && !(gdisph && P.balsara);
    double hv_min = DBL_MAX;
    unsigned nonconv = 0;
    unsigned n_cand = 0, n_newton = 0, n_pairs = 0, n_list = 0;  // work counters of this lane

    for(long long wb = warp * GPW; wb < n; wb += nwarps * GPW) {
        const int i = (int)(wb + ((threadIdx.x & 31) / G));
        const bool valid = i < n;
        const int cnt = valid ? min(count[i], cap) : 0;
        const int* li = list + (size_t)(valid ? i : 0) * (size_t)cap;
        const double4 pi = valid ? S.pos[i] : make_double4(0, 0, 0, 0);
        const double4 vi = valid ? S.vel[i] : make_double4(0, 0, 0, 1);
        const double4 ti = valid ? S.thermo[i] : make_double4(1, 0, 0, 0);
        const double sml0 = vi.w;

        // ---- 1. smoothing length (src/pre_interaction.cpp:227-283,
        //         src/disph/d_pre_interaction.cpp:174-230)
        double h = sml0;
        // disph: each sweep also keeps, per lane and in the lane's own order,
        // the candidates within (1 + 4e-4) h in a scratch row; after a
        // converged sweep (|h_new - h| < 1e-4 (h_new + h), so h_new <
        // (1 + 2.0003e-4) h) they hold every pair of the fused pass, which
        // then reads them instead of the whole list (8.78 M sphere, when it
        // came: 27.4 -> 24.1 ms, now 22.1; the gsph and gdisph bodies spilled
        // with it and ran slower)
        constexpr bool keep = TYPE == SPHGPU_DISPH;
        int* srow = scratch + (size_t)(valid ? i : 0) * (size_t)scap;
        int nk = 0;
        bool conv = false;
        if(P.iterative) {
            h = sml0 / P.ratio;
            const double b = disph ? P.nngb / AREA3 : pi.w * P.nngb / AREA3;
            for(int it = 0; it < 10; ++it) {
                const double hb = h;
                T d = 0, dd = 0;
                const KernF<KER> kh((T)h);
                const Within in(h);
                const bool exact = skin_delta > 0.0 && !(h < sml0 - skin_delta);
                const double hk = h * (1.0 + 4e-4), keep2 = hk * hk;
                nk = 0;
                // two candidates per iteration (the same per-lane order), both
                // evaluated; a sum keeps its value where the mask is off
                int ja = lane < cnt ? __ldg(&li[lane]) : 0;
                int jb = lane + G < cnt ? __ldg(&li[lane + G]) : 0;
                n_cand += lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u;
                for(int k = lane; k < cnt; k += 2 * G) {
                    const int ca = ja, cb = jb;  // cb is a valid index even past the list end
                    const bool two = k + G < cnt;
                    if(k + 2 * G < cnt) ja = __ldg(&li[k + 2 * G]);
                    if(k + 3 * G < cnt) jb = __ldg(&li[k + 3 * G]);
                    const double4 pa = ldg4(&S.pos[ca]);
                    const double4 pb = ldg4(&S.pos[cb]);
                    const double r2a = abs2x(offset_of<PER>(P, pi, pa)), r2b = abs2x(offset_of<PER>(P, pi, pb));
                    if constexpr(keep) {
                        if(r2a < keep2) srow[lane + G * nk++] = ca;
                        if(two && r2b < keep2) srow[lane + G * nk++] = cb;
                    }
                    bool ia = in.sure(r2a), ib = two && in.sure(r2b);
                    const bool ua = in.unsure(r2a), ub = two && in.unsure(r2b);
                    if(ua || ub || (exact && (ia || ib))) {  // rare
                        if(ua) ia = sqrt(r2a) < h;
                        if(ub) ib = sqrt(r2b) < h;
                        if(exact && ia) ia = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, ca, r2a);
                        if(exact && ib) ib = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, cb, r2b);
                    }
                    n_newton += (ia ? 1u : 0u) + (ib ? 1u : 0u);
                    auto add = [&](double r2, bool inside, T mj) {
                        const float r2f = (float)r2;
                        const T rT = r2f > 0.f ? r2f * rsqrtf(r2f) : 0.f;
                        const T w = kh.w(rT);
                        const T dh = kh.dhw(rT);
                        const T dn = disph ? __fadd_rn(d, w) : fmaf(mj, w, d);
                        const T ddn = disph ? __fadd_rn(dd, dh) : fmaf(mj, dh, dd);
                        d = inside ? dn : d;
                        dd = inside ? ddn : dd;
                    };
                    add(r2a, ia, (T)pa.w);
                    add(r2b, ib, (T)pb.w);
                }
                const double ds = (double)group_sum<G>(d), dds = (double)group_sum<G>(dd);
                const double h3 = h * h * h;
                const double f = ds * h3 - b;
                const double df = dds * h3 + 3 * ds * (h * h);
                h -= f / df;
                if(fabs(h - hb) < (h + hb) * 1e-4) {
                    conv = true;
                    break;
                }
            }
            if(!conv) {
                h = sml0 / P.ratio;
                if(valid && lane == 0) ++nonconv;
            }
        }

        // ---- 2. fused pass over {r < h}
        const KernF<KER> kh((T)h);
        const Within in(h);
        T dens = 0, dhd = 0, ni = 0, pres = 0, dhp = 0, dhn = 0;
        T divv = 0, rx = 0, ry = 0, rz = 0;
        T gd[3] = {0, 0, 0}, gu[3] = {0, 0, 0}, gv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        double vsig = ti.w * 2.0;
        int nn = 0;
        const bool need_av = !gsph && (P.balsara || P.td_av);
        const bool need_grad = (gsph || gdisph) && P.gsph2;
        const bool exact = skin_delta > 0.0 && !(h < sml0 - skin_delta);
        n_list += lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u;
        const bool kept = keep && conv;
        n_cand += kept ? (unsigned)nk : (lane < cnt ? (unsigned)((cnt - lane + G - 1) / G) : 0u);
        // one candidate, evaluated and masked (`use`: it is in the list): a sum
        // keeps its value where the mask is off
        struct Pair {
            Vec3d dv;
            double r2;
            bool in;
            double4 v, t;
        };
        auto load = [&](const double4& pj, int j, bool use) {
            Pair q;
            q.dv = offset_of<PER>(P, pi, pj);
            q.r2 = abs2x(q.dv);
            // the set predicate in FP64, the distance in FP32
            q.in = use && in.sure(q.r2);
            const bool unsure = use && in.unsure(q.r2);
            if(unsure || (exact && q.in)) {  // rare
                if(unsure) q.in = sqrt(q.r2) < h;
                if(exact && q.in) q.in = gather_member(P, Tr, pi.x, pi.y, pi.z, sml0, skin_delta, j, q.r2);
            }
            // coherent loads: this kernel writes vel.w and thermo.x, .y of every
            // particle (the components read here, velocity, u and c_s, it
            // does not change)
            q.v = q.t = make_double4(0, 0, 0, 0);
            if(q.in) {
                q.v = S.vel[j];
                q.t = S.thermo[j];
            }
            return q;
        };
        auto add = [&](const double4& pj, int j, const Pair& q) {
            const float r2f = (float)q.r2;
            const float rif = r2f > 0.f ? rsqrtf(r2f) : 0.f;
            const double r = (double)(r2f * rif), rinv = (double)rif;
            auto put = [&](T& sum, T with) { sum = q.in ? with : sum; };
            nn += q.in ? 1 : 0;
            const T rT = (T)r;
            const T w = kh.w(rT);
            const T mj = (T)pj.w;
            if(disph) {
                const T dh = kh.dhw(rT);
                const T uj = (T)q.t.z;
                put(dens, fmaf(mj, w, dens));
                put(ni, ni + w);
                put(pres, fmaf(mj * uj, w, pres));
                put(dhp, fmaf(mj * uj, dh, dhp));
                put(dhn, dhn + dh);
            } else {
                put(dens, TYPE == SPHGPU_SSPH ? __fadd_rn(dens, __fmul_rn(mj, w)) : fmaf(mj, w, dens));
                if(!gsph) put(dhd, fmaf(mj, kh.dhw(rT), dhd));
            }
            {
                const double vr = q.dv.x * (vi.x - q.v.x) + q.dv.y * (vi.y - q.v.y) + q.dv.z * (vi.z - q.v.z);
                // coincident particles (r = 0): the reference's vr / r is
                // 0 / 0, a NaN that never raises v_sig (+-inf if r underflowed)
                const double v = r > 0.0 ? ti.w + q.t.w - 3.0 * vr * rinv
                                         : (vr < 0.0 ? (double)INFINITY : -(double)INFINITY);
                if(q.in && i != j && v > vsig) vsig = v;
            }
            if(need_av || need_grad) {
                const T c = TYPE == SPHGPU_DISPH ? kh.k.dwc(rT, (T)rinv) : kh.dwc(rT, (T)rinv);
                const T dwx = (T)q.dv.x * c, dwy = (T)q.dv.y * c, dwz = (T)q.dv.z * c;
                const T vx = (T)(vi.x - q.v.x), vy = (T)(vi.y - q.v.y), vz = (T)(vi.z - q.v.z);
                if(need_av) {
                    const T wgt = av_energy ? mj * (T)q.t.z : mj;
                    put(divv, fmaf(-wgt, vx * dwx + vy * dwy + vz * dwz, divv));
                    put(rx, fmaf(vy * dwz - vz * dwy, wgt, rx));
                    put(ry, fmaf(vz * dwx - vx * dwz, wgt, ry));
                    put(rz, fmaf(vx * dwy - vy * dwx, wgt, rz));
                }
                if(need_grad) {
                    const T du = mj * (T)(q.t.z - ti.z);
                    put(gd[0], fmaf(dwx, mj, gd[0]));
                    put(gd[1], fmaf(dwy, mj, gd[1]));
                    put(gd[2], fmaf(dwz, mj, gd[2]));
                    put(gu[0], fmaf(dwx, du, gu[0]));
                    put(gu[1], fmaf(dwy, du, gu[1]));
                    put(gu[2], fmaf(dwz, du, gu[2]));
                    // dv[k] += dw * (m_j (v_j[k] - v_i[k]))
                    const T m0 = -mj * vx, m1 = -mj * vy, m2 = -mj * vz;
                    put(gv[0], fmaf(dwx, m0, gv[0]));
                    put(gv[1], fmaf(dwy, m0, gv[1]));
                    put(gv[2], fmaf(dwz, m0, gv[2]));
                    put(gv[3], fmaf(dwx, m1, gv[3]));
                    put(gv[4], fmaf(dwy, m1, gv[4]));
                    put(gv[5], fmaf(dwz, m1, gv[5]));
                    put(gv[6], fmaf(dwx, m2, gv[6]));
                    put(gv[7], fmaf(dwy, m2, gv[7]));
                    put(gv[8], fmaf(dwz, m2, gv[8]));
                }
            }
        };
        if(kept) {
            // the lane's kept candidates, in its own order (the same sums)
            for(int m = 0; m < nk; m += 2) {
                const bool two = m + 1 < nk;
                const int ca = srow[lane + G * m], cb = two ? srow[lane + G * (m + 1)] : ca;
                const double4 pa = ldg4(&S.pos[ca]);
                const double4 pb = ldg4(&S.pos[cb]);
                const Pair qa = load(pa, ca, true), qb = load(pb, cb, two);
                add(pa, ca, qa);
                add(pb, cb, qb);
            }
        } else {
            // the next candidates' indices are fetched one iteration ahead
            int ja = lane < cnt ? __ldg(&li[lane]) : 0;
            int jb = lane + G < cnt ? __ldg(&li[lane + G]) : 0;
            for(int k = lane; k < cnt; k += 2 * G) {
                const int ca = ja, cb = jb;
                const bool two = k + G < cnt;
                if(k + 2 * G < cnt) ja = __ldg(&li[k + 2 * G]);
                if(k + 3 * G < cnt) jb = __ldg(&li[k + 3 * G]);
                const double4 pa = ldg4(&S.pos[ca]);
                const double4 pb = ldg4(&S.pos[cb]);
                const Pair qa = load(pa, ca, true), qb = load(pb, cb, two);
                add(pa, ca, qa);
                add(pb, cb, qb);
            }
        }
        n_pairs += (unsigned)nn;
        const double densS = (double)group_sum<G>(dens);
        nn = group_sum<G>(nn);
        vsig = group_max<G>(vsig);
        double dhdS = 0, niS = 0, presS = 0, dhpS = 0, dhnS = 0;
        if(disph) {
            niS = (double)group_sum<G>(ni);
            presS = (double)group_sum<G>(pres);
            dhpS = (double)group_sum<G>(dhp);
            dhnS = (double)group_sum<G>(dhn);
        } else if(!gsph) {
            dhdS = (double)group_sum<G>(dhd);
        }
        double divS = 0, rxS = 0, ryS = 0, rzS = 0;
        if(need_av) {
            divS = (double)group_sum<G>(divv);
            rxS = (double)group_sum<G>(rx);
            ryS = (double)group_sum<G>(ry);
            rzS = (double)group_sum<G>(rz);
        }
        double gdS[3], guS[3], gvS[9];
        if(need_grad) {
#pragma unroll
            for(int k = 0; k < 3; ++k) {
                gdS[k] = (double)group_sum<G>(gd[k]);
                guS[k] = (double)group_sum<G>(gu[k]);
            }
#pragma unroll
            for(int k = 0; k < 9; ++k) gvS[k] = (double)group_sum<G>(gv[k]);
        }

        // ---- 3. epilogue (lane 0 of the group writes)
        if(!valid || lane != 0) continue;
        const double gamma = P.gamma;
        const double ui = ti.z, ci = ti.w;
        double pres_i;
        double4 vs = S.visc[i];
        if(disph) {
            pres_i = (gamma - 1.0) * presS;
            vs.z = h / (3 * niS) * dhpS / (1.0 + h / (3 * niS) * dhnS);
        } else {
            pres_i = (gamma - 1.0) * densS * ui;
            if(!gsph) vs.z = 1.0 / (1.0 + h / (3 * densS) * dhdS);
        }
        S.thermo[i] = make_double4(densS, pres_i, ui, ci);
        S.vel[i].w = h;
        S.nbr[i] = nn;
        const double hv = h / vsig;
        if(hv < hv_min) hv_min = hv;
        if(need_av) {
            // Balsara switch and time-dependent alpha (src/pre_interaction.cpp:115-161,
            // src/disph/d_pre_interaction.cpp:106-154)
            double dv_ = divS, r0 = rxS, r1 = ryS, r2 = rzS;
            if(av_energy) {
                const double pinv = (gamma - 1.0) / pres_i;
                dv_ *= pinv;
                r0 *= pinv;
                r1 *= pinv;
                r2 *= pinv;
            } else {
                dv_ /= densS;
                r0 /= densS;
                r1 /= densS;
                r2 /= densS;
            }
            if(P.balsara) {
                const double rot = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
                vs.y = fabs(dv_) / (fabs(dv_) + rot + 1e-4 * ci / h);
                if(P.td_av) {
                    const double tau = P.eps_av * ci / h;
                    const double da = (-(vs.x - P.alpha_min) * tau + fmax(-dv_, 0.0) * (P.alpha_max - vs.x)) * dt;
                    vs.x += da;
                }
            } else {
                const double tau = P.eps_av * ci / h;
                const double s = fmax(-dv_, 0.0);
                vs.x = (vs.x + dt * tau * P.alpha_min + s * dt * P.alpha_max) / (1.0 + dt * tau + s * dt);
            }
        }
        S.visc[i] = vs;
        if(need_grad) {
            // MUSCL gradients (src/gsph/g_pre_interaction.cpp:112-136)
            const double gm1 = gamma - 1.0, rinv = 1.0 / densS;
            const double g15[15] = {gdS[0],
                                    gdS[1],
                                    gdS[2],
                                    (gdS[0] * ui + guS[0]) * gm1,
                                    (gdS[1] * ui + guS[1]) * gm1,
                                    (gdS[2] * ui + guS[2]) * gm1,
                                    gvS[0] * rinv,
                                    gvS[1] * rinv,
                                    gvS[2] * rinv,
                                    gvS[3] * rinv,
                                    gvS[4] * rinv,
                                    gvS[5] * rinv,
                                    gvS[6] * rinv,
                                    gvS[7] * rinv,
                                    gvS[8] * rinv};
            S.grad[i] = make_double4(g15[0], g15[1], g15[2], g15[3]);
            S.grad[(size_t)n + i] = make_double4(g15[4], g15[5], g15[6], g15[7]);
            S.grad[2 * (size_t)n + i] = make_double4(g15[8], g15[9], g15[10], g15[11]);
            S.grad[3 * (size_t)n + i] = make_double4(g15[12], g15[13], g15[14], 0.0);
        }
    }
    // block reductions: min h / v_sig, Newton fallbacks
    __shared__ double s_min[PBLK / 32];
    __shared__ unsigned s_nc[PBLK / 32];
    hv_min = warp_min(hv_min);
    for(int o = 16; o > 0; o >>= 1) nonconv += __shfl_xor_sync(FULL_MASK, nonconv, o);
    if((threadIdx.x & 31) == 0) {
        s_min[threadIdx.x >> 5] = hv_min;
        s_nc[threadIdx.x >> 5] = nonconv;
    }
    __syncthreads();
    if(threadIdx.x == 0) {
        double m = s_min[0];
        unsigned c = s_nc[0];
        for(int w = 1; w < PBLK / 32; ++w) {
            m = fmin(m, s_min[w]);
            c += s_nc[w];
        }
        if(m < DBL_MAX) atomic_min_pos(hvs, m);
        if(c) atomicAdd(&st->newton_nonconv, (unsigned long long)c);
    }
    block_count(&st->pre_cand, n_cand);
    block_count(&st->pre_newton_pairs, n_newton);
    block_count(&st->pre_pairs, n_pairs);
    block_count(&st->pre_list, n_list);
}

// PreInteraction::initial_smoothing (src/pre_interaction.cpp:171-215):
// density at the guessed h over {r < h}.
template <typename T, int G>
__global__ void __launch_bounds__(PBLK) k_initial_density(DevParams P, DevState S, int n,
                                                          const int* __restrict__ list,
                                                          const int* __restrict__ count, int cap)
{
    constexpr int GPW = 32 / G;
    const int lane = threadIdx.x & (G - 1);
    const long long warp = ((long long)blockIdx.x * PBLK + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * PBLK) >> 5;
    for(long long wb = warp * GPW; wb < n; wb += nwarps * GPW) {
        const int i = (int)(wb + ((threadIdx.x & 31) / G));
        const bool valid = i < n;
        const int cnt = valid ? min(count[i], cap) : 0;
        const int* li = list + (size_t)(valid ? i : 0) * (size_t)cap;
        const double4 pi = valid ? S.pos[i] : make_double4(0, 0, 0, 0);
        const double h = valid ? S.vel[i].w : 1.0;
        const KernH<T> kh(P.kernel, (T)h);
        T d = 0;
        for(int k = lane; k < cnt; k += G) {
            const double4 pj = S.pos[li[k]];
            Vec3d dv;
            const double r = exact_r(P, pi.x, pi.y, pi.z, pj, dv);
            if(r < h) d += (T)pj.w * kh.w((T)r);
        }
        const double ds = (double)group_sum<G>(d);
        if(valid && lane == 0) S.thermo[i].x = ds;
    }
}

constexpr int GROUP = 4;

unsigned pre_grid(int n)
{
    const long long groups_per_block = PBLK / GROUP;
    long long blocks = (n + groups_per_block - 1) / groups_per_block;
    const long long cap = 148LL * 8 * 4;
    return (unsigned)std::max<long long>(1, std::min(blocks, cap));
}

template <typename K>
void launch_pre_kernel(sphgpu_ctx* c, K* k)
{
    k<<<pre_grid(c->n), PBLK, 0, c->stream>>>(c->dp, c->s, c->n, c->d_glist, c->d_gcount, (int)c->gcap, c->d_dt,
                                              c->d_hvs, c->d_status, c->t,
                                              c->skin_valid ? c->skin_delta_now : 0.0, c->d_plist, (int)c->pcap);
}

template <int TYPE, int KER>
void launch_pre_form(sphgpu_ctx* c)
{
    if(c->prm.precision == SPHGPU_MIXED) {
        launch_pre_kernel(c, c->prm.periodic ? k_pre_mixed<GROUP, TYPE, KER, true> : k_pre_mixed<GROUP, TYPE, KER, false>);
    } else {
        launch_pre_kernel(c, c->prm.periodic ? k_pre<GROUP, TYPE, KER, true> : k_pre<GROUP, TYPE, KER, false>);
    }
}

template <int TYPE>
void launch_pre(sphgpu_ctx* c)
{
    if(c->prm.kernel == SPHGPU_WENDLAND) launch_pre_form<TYPE, SPHGPU_WENDLAND>(c);
    else if(c->prm.kernel == SPHGPU_GAUSSIAN) launch_pre_form<TYPE, SPHGPU_GAUSSIAN>(c);
    else launch_pre_form<TYPE, SPHGPU_CUBIC_SPLINE>(c);
}

}  // namespace

int pre_interaction(sphgpu_ctx* c)
{
    if(!c->have_tree) return fail(c, SPHGPU_ERR_STATE, "PreInteraction before tree make");
    if(c->prm.sph_type == SPHGPU_SRGSPH) return sr_pre_interaction(c);
    int rc_walk = SPHGPU_OK;
    const bool mixed = c->prm.precision == SPHGPU_MIXED;
    if(c->first_pre) {
        // initial_smoothing: h from the initial density, no kernel ratio
        int rc = gather_walk(c, true, 1.0);
        if(rc < 0) return rc;
        stage_begin(c, SPHGPU_T_PRE);
        if(mixed) {
            k_initial_density<float, GROUP><<<pre_grid(c->n), PBLK, 0, c->stream>>>(c->dp, c->s, c->n, c->d_glist,
                                                                                    c->d_gcount, (int)c->gcap);
        } else {
            k_initial_density<double, GROUP><<<pre_grid(c->n), PBLK, 0, c->stream>>>(c->dp, c->s, c->n, c->d_glist,
                                                                                     c->d_gcount, (int)c->gcap);
        }
        SPHGPU_LAUNCH_CHECK(c, "initial_smoothing");
        stage_end(c, SPHGPU_T_PRE, 1);
        c->first_pre = false;
    }
    rc_walk = gather_lists(c, c->dp.ratio);
    if(rc_walk < 0) return rc_walk;
    int rcs = save_gather_radius(c);
    if(rcs < 0) return rcs;
    // the pair-list buffer is the sweeps' scratch (the pair lists are built after)
    if(c->pcap < c->gcap && (rcs = ensure_list_capacity(c, 1, c->gcap)) < 0) return rcs;
    stage_begin(c, SPHGPU_T_PRE);
    const double big = DBL_MAX;
    SPHGPU_CUDA(c, cudaMemcpyAsync(c->d_hvs, &big, sizeof(double), cudaMemcpyHostToDevice, c->stream));
    const int type = c->prm.sph_type;
    if(type == SPHGPU_DISPH) launch_pre<SPHGPU_DISPH>(c);
    else if(type == SPHGPU_GSPH) launch_pre<SPHGPU_GSPH>(c);
    else if(type == SPHGPU_GDISPH) launch_pre<SPHGPU_GDISPH>(c);
    else launch_pre<SPHGPU_SSPH>(c);
    SPHGPU_LAUNCH_CHECK(c, "PreInteraction");
    stage_end(c, SPHGPU_T_PRE, 1);
    int rc = tree_set_kernel(c);
    if(rc < 0) return rc;
    rc = build_force_lists(c);
    if(rc < 0) return rc;
    return rc_walk;
}

}  // namespace sphgpu
