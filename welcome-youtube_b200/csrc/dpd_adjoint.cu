// dpd_adjoint.cu -- reverse mode through the DPD step (sm_100a).
//
// k_force_vjp    vector-Jacobian product of the pair + bond forces of one
//                configuration: given the cotangent g of the forces, the
//                gradients with respect to positions, predicted velocities,
//                the repulsions a_ij, gamma and the bond constant.  The pair
//                noise theta is replayed from its key (frozen noise).
// k_rdf          Gaussian-smoothed pair distribution of two bead types
//                (the structural target of a fit) and its gradient (VJP).
// adj_update     the adjoint of the Groot-Warren update, applied by the VJP
//                kernel itself.  The adjoint state lies in the slots of the
//                configuration it belongs to and moves from step to step
//                through the steps' stored sorts, so that its accesses are as
//                local as the sort is (in gid order every access was a sector
//                of its own: 82 us a step on 24 boxes of 65,536 beads, and 11
//                for the gather of the force cotangents).
//
// Pair term (w = 1 - r, A = a - gamma w rv + s theta, s = sigma / sqrt(dt)):
//   f = fm d,  fm = w A / r,  rv = d . dv / r
//   d(c.f)/dd  = (c.d) [dfm/dr dhat + dfm/drv (dv - rv dhat) / r] + fm c
//   d(c.f)/ddv = (c.d) dfm/drv dhat
//   dfm/dr  = (-A + w gamma rv) / r - w A / r^2,   dfm/drv = -gamma w^2 / r
//   d(c.f)/da_ij = (c.d) w / r,  d(c.f)/dgamma = (c.d) w (-w rv + s theta / (2 gamma)) / r
// with c = g_i - g_j for the pair (i, j).  Every bead sums over its 3x3 cells
// (each pair from both ends; the two halves are exact negatives), the
// parameter gradients count each pair once.  s follows the temperature cycle
// (s(step) = sqrt(2 gamma kT(t) / dt)), as the forward forces do.
//
// Angle terms (U = K (1 - cos), or K (cos - c0)^2 at the junctions of the
// branched shapes, per triplet i-j-k, a = x_j - x_i, c = x_k - x_j): with
// F = -grad U the VJP on bead m is -d phi / d x_m, phi = sum over beads of
// g . dU/dx = D U(a, c)[da, dc], da = g_j - g_i, dc = g_k - g_j.  dphi/da and
// dphi/dc are Hessian-vector products of U, written out in angle_hvp; then
// d/dx_i = -d/da, d/dx_j = d/da - d/dc, d/dx_k = d/dc.  Linear chains: each
// bead gathers the triplets it is part of (as middle, as last of its prev's,
// as first of its next's), so no two threads write one bead.  Branched
// shapes: k_mol_vjp, one thread per molecule.
//
// Stirring (f_x,i = A sin(2 pi k y_i) minus its replica mean): the VJP on y_m
// is A 2 pi k cos(2 pi k y_m) (g_x,m - mean of g_x), the mean from k_gsum.
#include <algorithm>

#include "dpd_device.cuh"

#define NGRAD DPD_NGRAD

__device__ __forceinline__ float dot2(float2 u, float2 v) { return u.x * v.x + u.y * v.y; }

// dphi/da (pa) and dphi/dc (pc) of phi = D U(a, c)[da, dc] for an angle term
// U(cos) of kind 0, U = K (1 - cos) (U' = -K, U'' = 0), or kind 1,
// U = K (cos - c0)^2 (U' = 2 K (cos - c0), U'' = 2 K):
//   cos = (a.c) / (|a| |c|),  Dcos = q / AC - cos (a.da) / A2 - cos (c.dc) / C2,  q = da.c + a.dc
//   dDcos/da = dc / AC - q a / (AC A2) - gca ((a.da) / A2 + (c.dc) / C2) - cos (da / A2 - 2 (a.da) a / A2^2)
//   dDcos/dc = da / AC - q c / (AC C2) - gcc ((a.da) / A2 + (c.dc) / C2) - cos (dc / C2 - 2 (c.dc) c / C2^2)
// with gca = dcos/da = c / AC - cos a / A2, gcc = dcos/dc = a / AC - cos c / C2;
// phi = U' Dcos, so dphi/da = U'' Dcos gca + U' dDcos/da (and likewise for c)
__device__ __forceinline__ void angle_hvp(float2 a, float2 c, float2 da, float2 dc, int kind, float K, float c0,
                                          float2 &pa, float2 &pc) {
    const float A2 = dot2(a, a), C2 = dot2(c, c);
    const float iac = rsqrtf(A2 * C2), iA2 = 1.0f / A2, iC2 = 1.0f / C2;
    const float cs = dot2(a, c) * iac;
    const float q = dot2(da, c) + dot2(a, dc), ada = dot2(a, da), cdc = dot2(c, dc);
    const float m = ada * iA2 + cdc * iC2;
    const float2 gca = make_float2(c.x * iac - cs * a.x * iA2, c.y * iac - cs * a.y * iA2);
    const float2 gcc = make_float2(a.x * iac - cs * c.x * iC2, a.y * iac - cs * c.y * iC2);
    const float ta = q * iac * iA2, tc = q * iac * iC2;
    const float ka2 = 2.0f * ada * iA2 * iA2, kc2 = 2.0f * cdc * iC2 * iC2;
    const float u1 = kind == 0 ? -K : 2.0f * K * (cs - c0), u2 = kind == 0 ? 0.0f : 2.0f * K;
    const float dcos = q * iac - cs * m;
    pa = make_float2(u2 * dcos * gca.x + u1 * (dc.x * iac - ta * a.x - gca.x * m - cs * (da.x * iA2 - ka2 * a.x)),
                     u2 * dcos * gca.y + u1 * (dc.y * iac - ta * a.y - gca.y * m - cs * (da.y * iA2 - ka2 * a.y)));
    pc = make_float2(u2 * dcos * gcc.x + u1 * (da.x * iac - tc * c.x - gcc.x * m - cs * (dc.x * iC2 - kc2 * c.x)),
                     u2 * dcos * gcc.y + u1 * (da.y * iac - tc * c.y - gcc.y * m - cs * (dc.y * iC2 - kc2 * c.y)));
}

// the angle-term VJP of a bead of a linear chain at pi with cotangent gi and
// links lk (x_bar increment): the triplets (p, d, n), (pp, p, d) and
// (d, n, nn) of its chain, where they exist
__device__ __forceinline__ float2 angle_vjp(const StateView &sv, const float2 *__restrict__ g, const RepDev &R, float2 pi,
                                           float2 gi, int2 lk) {
    const float L = R.L, h = R.halfL, ka = R.ka;
    float2 out = make_float2(0.0f, 0.0f);
    auto vec = [&](float2 u, float2 v) {  // v - u, minimum image
        return make_float2(minimg(v.x - u.x, L, h), minimg(v.y - u.y, L, h));
    };
    auto dif = [](float2 u, float2 v) { return make_float2(v.x - u.x, v.y - u.y); };
    float2 pp_ = pi, pn = pi, gp = gi, gn = gi;
    if (lk.x >= 0) {
        pp_ = sv.pos[lk.x];
        gp = g[lk.x];
    }
    if (lk.y >= 0) {
        pn = sv.pos[lk.y];
        gn = g[lk.y];
    }
    float2 pa, pc;
    if (lk.x >= 0 && lk.y >= 0) {  // the bead in the middle: -(dphi/da - dphi/dc)
        angle_hvp(vec(pp_, pi), vec(pi, pn), dif(gp, gi), dif(gi, gn), 0, ka, 0.0f, pa, pc);
        out.x -= pa.x - pc.x;
        out.y -= pa.y - pc.y;
    }
    if (lk.x >= 0) {
        const int q = sv.link[lk.x].x;
        if (q >= 0) {  // (q, p, d): the bead last, -dphi/dc
            const float2 pq = sv.pos[q], gq = g[q];
            angle_hvp(vec(pq, pp_), vec(pp_, pi), dif(gq, gp), dif(gp, gi), 0, ka, 0.0f, pa, pc);
            out.x -= pc.x;
            out.y -= pc.y;
        }
    }
    if (lk.y >= 0) {
        const int q = sv.link[lk.y].y;
        if (q >= 0) {  // (d, n, q): the bead first, +dphi/da
            const float2 pq = sv.pos[q], gq = g[q];
            angle_hvp(vec(pi, pn), vec(pn, pq), dif(gi, gn), dif(gn, gq), 0, ka, 0.0f, pa, pc);
            out.x += pa.x;
            out.y += pa.y;
        }
    }
    return out;
}

// per replica, the sum of the x cotangents (the stirring term's mean)
__global__ void __launch_bounds__(BEAD_TPB) k_gsum(const RepDev *__restrict__ reps, const Chunk *__restrict__ ch,
                                                   const float2 *__restrict__ g, double *__restrict__ gsum) {
    const Chunk c = ch[blockIdx.x];
    if (reps[c.rep].stir_A == 0.0f) return;
    const int d = c.begin + (int)threadIdx.x;
    double v = d < c.end ? (double)g[d].x : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane_id() == 0 && v != 0.0) atomicAdd(gsum + c.rep, v);
}

#define VJP_TPB 256
#define VJP_LIST 32         // pairs a bead lists at a time
#define VJP_TYPES 4         // types whose pairs have lane-private gradient sums
#define VJP_COMBOS (VJP_TYPES * (VJP_TYPES + 1) / 2)

//   x_bar(n)  = x_bar(n+1) + J_x^T F_bar
//   vh_bar(n) = dt x_bar(n) + vh_bar(n+1) + J_v^T F_bar
//   F_bar(n)  = dt^2 x_bar(n) + dt vh_bar(n+1) + cvt J_v^T F_bar
// of bead d (type t) of the configuration n+1; xf = J_x^T F_bar, vf = J_v^T F_bar
__device__ __forceinline__ void adj_update(const AdjUpdate &u, const RepDev &R, int d, int t, float2 xf, float2 vf) {
    float2 x0 = u.X[d];
    const float2 v0 = u.V[d];
    if (u.G && (t == u.ta || t == u.tb)) {
        const float2 g = u.G[d];
        x0.x += g.x;
        x0.y += g.y;
    }
    const int o = u.src[d];
    const float2 x = make_float2(x0.x + xf.x, x0.y + xf.y);
    u.X2[o] = x;
    u.V2[o] = make_float2(R.dt * x.x + v0.x + vf.x, R.dt * x.y + v0.y + vf.y);
    u.F2[o] = make_float2(R.dt2 * x.x + R.dt * v0.x + R.cvt * vf.x, R.dt2 * x.y + R.dt * v0.y + R.cvt * vf.y);
}

// LPB lanes share a bead: each takes its part of the bead's 3 x 3 cells' slots
// (cells are column-major: three contiguous ranges, six where the rows wrap)
// and marks the ones inside the cutoff in a word; the bead's hits are listed in
// the order of its cells and slots and evaluated by its lanes in turn, so that
// the noise and the derivative run on lanes that have a pair.  Each pair is
// evaluated by both of its beads: no atomics on floats, and a bead's terms are
// added in its list's order: as a thread per bead would add them (the same
// bits) where a lane's part of the slots is at most the 32 of its word, which is
// up to 64 candidates with two lanes and 128 with four; beyond that, the lanes'
// next words follow the first.  The sums of the parameters' gradient are FP64: per lane and pair of
// types in shared memory for the first four types (no two lanes on one word),
// through an atomic for the others.
// A CTA takes a run of consecutive tasks (256 / LPB beads of a chunk) and hands
// its gradient sums over when the replica changes and at its end.  UPDATE: the
// adjoint of the step's update is applied at once (adj_update); else the
// products go to xbar and vbar.
// What bounds it: about 180 warp instructions a bead at density 4, half of them
// the 12.6 evaluations (40 of whose 140 instructions are the noise), issued at
// 2.2 of 4 a cycle: the chains of loads and arithmetic of a few warps.  So a
// lane evaluates two pairs at a time: 24 boxes of 65,536 beads 403 us, 429 with
// one.  And the fullest list of a warp is 1.6 times the mean.  The same boxes
// took 939 us (and 82 for the update) with a thread per bead and an FP64 shared
// atomic per pair; one box 31 against 68, of 16,384: 14 against 60, of 4,096: 10
// against 61.  Tried: one queue of pairs per warp evaluated by full rounds, its
// terms summed through shared memory, 504 us (more shared memory, 16 warps an
// SM); the order of the sum left to the lanes, 397 us.
template <int LPB, int MINB, bool UPDATE>
__global__ void __launch_bounds__(VJP_TPB, MINB) k_force_vjp(StateView sv, long long step, const RepDev *__restrict__ reps,
                                                       const Chunk *__restrict__ ch, int ntask,
                                                       const float2 *__restrict__ g, float2 *__restrict__ xbar,
                                                       float2 *__restrict__ vbar, AdjUpdate up,
                                                       double *__restrict__ grad, const double *__restrict__ gsum,
                                                       const long long *__restrict__ step_base) {
    constexpr int BEADS = VJP_TPB / LPB;
    __shared__ int list[BEADS][VJP_LIST + 1];
    __shared__ double acc[VJP_COMBOS][VJP_TPB];
    __shared__ double sgrad[NGRAD];
    __shared__ float a_sh[DPD_MAXT * DPD_MAXT];
    const int tid = (int)threadIdx.x, lane = (int)lane_id(), sub = tid % LPB, bead = tid / LPB;
    for (int k = tid; k < NGRAD; k += VJP_TPB) sgrad[k] = 0.0;
#pragma unroll
    for (int k = 0; k < VJP_COMBOS; k++) acc[k][tid] = 0.0;
    double ggam = 0.0, gkb = 0.0;
    if (step_base) step += *step_base;  // the step relative to a step number kept on the device
    const int t0 = (int)((long long)ntask * blockIdx.x / gridDim.x);
    const int t1 = (int)((long long)ntask * (blockIdx.x + 1) / gridDim.x);
    int rep = -1;
    float gam = 0.0f, s = 0.0f;
    NoiseKey nk;
    // the CTA's gradient sums of replica `rep`, added to the global ones
    auto hand_over = [&]() {
        auto add = [&](double v, int slot) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0 && v != 0.0) atomicAdd(&sgrad[slot], v);
        };
        int k = 0;
#pragma unroll 1
        for (int i = 0; i < VJP_TYPES; i++)
#pragma unroll 1
            for (int j = i; j < VJP_TYPES; j++, k++) {
                add(acc[k][tid], i * DPD_MAXT + j);
                acc[k][tid] = 0.0;
            }
        add(ggam, DPD_MAXT * DPD_MAXT);
        add(gkb, DPD_MAXT * DPD_MAXT + 1);
        ggam = gkb = 0.0;
        __syncthreads();
        for (int q = tid; q < NGRAD; q += VJP_TPB)
            if (sgrad[q] != 0.0) {
                atomicAdd(&grad[(size_t)rep * NGRAD + q], sgrad[q]);
                sgrad[q] = 0.0;
            }
        __syncthreads();
    };
    for (int task = t0; task < t1; task++) {
        const Chunk c = ch[task / LPB];
        const RepDev &R = reps[c.rep];
        if (c.rep != rep) {  // uniform over the CTA
            if (rep >= 0) hand_over();
            rep = c.rep;
            if (tid < DPD_MAXT * DPD_MAXT) a_sh[tid] = R.a[tid];
            gam = R.gamma;
            s = sdt_at(R, step);
            nk = make_noise_key(R, step);
            __syncthreads();
        }
        const int d = c.begin + task % LPB * BEADS + bead;
        const bool act = d < c.end;
        const float L = R.L, h = R.halfL;
        const int ncx = R.ncx, ncy = R.ncy;
        const int32_t *__restrict__ cs = sv.cstart + R.c0;
        float2 pi = make_float2(0.f, 0.f), vi = pi, gi2 = pi;
        uint32_t tgi = 0;
        int cx = 0, cy = 0;
        if (act) {
            pi = sv.pos[d];
            vi = sv.vt[d];
            gi2 = g[d];
            tgi = sv.tg[d];
            cell_xy(R, pi.x, pi.y, cx, cy);
        }
        const int d0 = act ? d : c.begin;  // (a slot to read for lanes without a pair)
        const uint32_t gi = tgi & GID_MASK;
        const int ti = (int)(tgi >> TYPE_SHIFT);
        const bool low = act && cy == 0, high = act && cy == ncy - 1;  // ncy >= 3: the rows wrap at one end
        // does some bead of the warp sit in an edge cell (its neighbours' images matter), or in one of an edge row
        const bool rows = __any_sync(0xffffffffu, low || high);
        const bool wrap = rows || __any_sync(0xffffffffu, act && (cx == 0 || cx == ncx - 1));
        // the slots of the bead's columns in order: three ranges, or six; l: ends of the ranges counted together,
        // b: what leads from that count to the slot
        int l0 = 0, l1 = 0, l2 = 0, l3 = 0, l4 = 0, l5 = 0, b0 = 0, b1 = 0, b2 = 0, b3 = 0, b4 = 0, b5 = 0;
        if (act) {
            const int32_t *c0 = cs + (cx > 0 ? cx - 1 : ncx - 1) * ncy, *c1 = cs + cx * ncy;
            const int32_t *c2 = cs + (cx + 1 < ncx ? cx + 1 : 0) * ncy;
            if (!rows) {
                b0 = c0[cy - 1];
                b1 = c1[cy - 1];
                b2 = c2[cy - 1];
                l0 = c0[cy + 2] - b0;
                l1 = l0 + (c1[cy + 2] - b1);
                l2 = l1 + (c2[cy + 2] - b2);
                b1 -= l0;
                b2 -= l1;
                l3 = l4 = l5 = l2;
            } else {
                // the rows before the wrap [ra, rb) and after it [rc, rd): row ncy - 1 then 0, 1; or ncy - 2, ncy - 1
                // then 0; or cy - 1 .. cy + 1 and none
                const int ra = low ? ncy - 1 : cy - 1, rb = low || high ? ncy : cy + 2;
                const int rc = 0, rd = low ? 2 : (high ? 1 : 0);
                b0 = c0[ra];
                l0 = c0[rb] - b0;
                b1 = c0[rc];
                l1 = l0 + (c0[rd] - b1);
                b2 = c1[ra];
                l2 = l1 + (c1[rb] - b2);
                b3 = c1[rc];
                l3 = l2 + (c1[rd] - b3);
                b4 = c2[ra];
                l4 = l3 + (c2[rb] - b4);
                b5 = c2[rc];
                l5 = l4 + (c2[rd] - b5);
                b1 -= l0;
                b2 -= l1;
                b3 -= l2;
                b4 -= l3;
                b5 -= l4;
            }
        }
        auto slot = [&](int k) {
            if (!rows) return k + (k < l0 ? b0 : (k < l1 ? b1 : b2));
            return k + (k < l0 ? b0 : (k < l1 ? b1 : (k < l2 ? b2 : (k < l3 ? b3 : (k < l4 ? b4 : b5)))));
        };
        float xbx = 0.f, xby = 0.f, vbx = 0.f, vby = 0.f;  // x_bar in the bead's first lane, v_bar in its second
        // The pair of the lane's bead with entry k of its list (some entry if there are only n: then nothing counts);
        // its terms, and the parameter gradients.
        struct Terms {
            float tx, ty, u, hx, hy;
        };
        auto pair = [&](int k, int n) {
            Terms t;
            const int j = n > 0 ? list[bead][min(k, n - 1)] : d0;
            const float2 pj = sv.pos[j], vj = sv.vt[j], gj = g[j];
            const uint32_t tgj = sv.tg[j];
            const int tj = (int)(tgj >> TYPE_SHIFT);
            float dx = __fsub_rn(pi.x, pj.x), dy = __fsub_rn(pi.y, pj.y);
            if (wrap) {
                dx = minimg(dx, L, h);
                dy = minimg(dy, L, h);
            }
            const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
            float r, ir;
            r_and_ir(r2, r, ir);
            const float w = 1.0f - r;
            const float dvx = vi.x - vj.x, dvy = vi.y - vj.y;
            const float rv = (dx * dvx + dy * dvy) * ir;
            const float th = pair_theta(nk, gi, tgj & GID_MASK);
            const float a = a_sh[ti * DPD_MAXT + tj];
            const float A = a - gam * w * rv + s * th;
            const float fm = w * A * ir;
            const float cxv = gi2.x - gj.x, cyv = gi2.y - gj.y;
            const float cd = cxv * dx + cyv * dy;
            const float dfr = (-A + w * gam * rv) * ir - w * A * ir * ir;
            const float dfv = -gam * w * w * ir;
            t.hx = dx * ir;
            t.hy = dy * ir;
            t.tx = __fmaf_rn(fm, cxv, __fmul_rn(cd, dfr * t.hx + dfv * (dvx - rv * t.hx) * ir));
            t.ty = __fmaf_rn(fm, cyv, __fmul_rn(cd, dfr * t.hy + dfv * (dvy - rv * t.hy) * ir));
            t.u = cd * dfv;
            if (k < n && gi < (tgj & GID_MASK)) {  // parameter gradients: each pair once
                const int lo = min(ti, tj), hi = max(ti, tj);
                const double da = (double)(cd * w * ir);
                if (hi < VJP_TYPES) acc[lo * (2 * VJP_TYPES - 1 - lo) / 2 + hi][tid] += da;
                else atomicAdd(&sgrad[lo * DPD_MAXT + hi], da);
                ggam += (double)(cd * w * (-w * rv + (gam > 0.0f ? s * th / (2.0f * gam) : 0.0f)) * ir);
            }
            return t;
        };
        // the terms of round q's pairs added in the list's order
        auto add = [&](const Terms &t, int q, int n) {
            if (LPB == 2) {  // each lane hands the other what it sums
                const float o1 = __shfl_xor_sync(0xffffffffu, sub ? t.tx : t.u, 1);
                const float o2 = __shfl_xor_sync(0xffffffffu, sub ? t.ty : t.hx, 1);
                const float o3 = __shfl_xor_sync(0xffffffffu, t.hy, 1);
                const int left = n - q * LPB;
                if (sub == 0) {
                    if (left > 0) {
                        xbx += t.tx;
                        xby += t.ty;
                    }
                    if (left > 1) {
                        xbx += o1;
                        xby += o2;
                    }
                } else {
                    if (left > 0) {
                        vbx = __fmaf_rn(o1, o2, vbx);
                        vby = __fmaf_rn(o1, o3, vby);
                    }
                    if (left > 1) {
                        vbx = __fmaf_rn(t.u, t.hx, vbx);
                        vby = __fmaf_rn(t.u, t.hy, vby);
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < LPB; i++) {
                    const float ax = __shfl_sync(0xffffffffu, t.tx, i, LPB), ay = __shfl_sync(0xffffffffu, t.ty, i, LPB);
                    const float au = __shfl_sync(0xffffffffu, t.u, i, LPB), ahx = __shfl_sync(0xffffffffu, t.hx, i, LPB);
                    const float ahy = __shfl_sync(0xffffffffu, t.hy, i, LPB);
                    if (q * LPB + i < n) {
                        xbx += ax;
                        xby += ay;
                        vbx = __fmaf_rn(au, ahx, vbx);
                        vby = __fmaf_rn(au, ahy, vby);
                    }
                }
            }
        };
        // the listed pairs [0, n) of every bead, two rounds of its lanes at a time (two independent chains a lane)
        auto evaluate = [&](int n) {
            __syncwarp();
            const int rounds = (__reduce_max_sync(0xffffffffu, n) + LPB - 1) / LPB;
            int q = 0;
            for (; q + 1 < rounds; q += 2) {
                const Terms t0 = pair(q * LPB + sub, n), t1 = pair((q + 1) * LPB + sub, n);
                add(t0, q, n);
                add(t1, q + 1, n);
            }
            if (q < rounds) add(pair(q * LPB + sub, n), q, n);
            __syncwarp();
        };
        // each lane marks the hits of its part of the slots in a word; then the bead's hits are listed in order
        const int per = (l5 + LPB - 1) / LPB, k0 = sub * per, k1 = min(k0 + per, l5);
        const int most = __reduce_max_sync(0xffffffffu, per);
        for (int kb = 0; kb < most; kb += 32) {
            uint32_t mark = 0;
            const int rounds = min(32, most - kb);
#pragma unroll 4
            for (int u = 0; u < rounds; u++) {
                const int k = k0 + kb + u, j = slot(k);
                const bool in = k < k1;
                const float2 pj = sv.pos[in ? j : 0];
                float dx = __fsub_rn(pi.x, pj.x), dy = __fsub_rn(pi.y, pj.y);
                if (wrap) {
                    dx = minimg(dx, L, h);
                    dy = minimg(dy, L, h);
                }
                const float r2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
                mark |= (in && r2 < 1.0f && r2 > 1e-24f && j != d ? 1u : 0u) << u;
            }
            int at = __popc(mark);  // the place of this lane's first hit among its bead's
            const int own = at;
#pragma unroll
            for (int o = 1; o < LPB; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, at, o, LPB);
                if (sub >= o) at += t;
            }
            const int n = __shfl_sync(0xffffffffu, at, LPB - 1, LPB);
            at -= own;
            for (int first = 0; __any_sync(0xffffffffu, first < n); first += VJP_LIST) {  // once, unless crowded
                int to = at - first;
                for (uint32_t m = mark; m; m &= m - 1, to++)
                    if (to >= 0 && to < VJP_LIST) list[bead][to] = slot(k0 + kb + __ffs(m) - 1);
                evaluate(max(0, min(n - first, VJP_LIST)));
            }
        }
        if (LPB == 2) {
            vbx = __shfl_down_sync(0xffffffffu, vbx, 1);
            vby = __shfl_down_sync(0xffffffffu, vby, 1);
        }
        if (act && sub == 0) {
            // bonds: f_i = kb (1 - r0/r) d with d = x_p - x_i (linear chains; the
            // branched shapes' bonds and angles are k_mol_vjp's)
            const int2 lk = R.arch == 0 ? sv.link[d] : make_int2(-1, -1);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int p = q ? lk.y : lk.x;
                if (p < 0) continue;
                const float2 pp = sv.pos[p], gp = g[p];
                const float dx = minimg(pp.x - pi.x, L, h), dy = minimg(pp.y - pi.y, L, h);
                const float r = sqrtf(dx * dx + dy * dy);
                const float cxv = gi2.x - gp.x, cyv = gi2.y - gp.y;
                const float cd = cxv * dx + cyv * dy;
                const float u = 1.0f - R.r0 / r;
                const float kr = R.kb * R.r0 / (r * r) * cd / r;
                xbx -= kr * dx + R.kb * u * cxv;
                xby -= kr * dy + R.kb * u * cyv;
                if (q == 1) gkb += (double)(u * cd);  // each bond once, from its prev end
            }
            if (R.ka != 0.0f && (lk.x >= 0 || lk.y >= 0)) {
                const float2 t = angle_vjp(sv, g, R, pi, gi2, lk);
                xbx += t.x;
                xby += t.y;
            }
            if (R.stir_A != 0.0f) {
                const double w2 = 2.0 * R.stir_k;
                const double dfy = (double)R.stir_A * M_PI * w2 * cospi(w2 * (double)pi.y);
                xby += (float)(dfy * ((double)gi2.x - gsum[c.rep] / (double)R.n));
            }
        }
        if (act && sub == 0) {
            if (UPDATE) {
                adj_update(up, R, d, ti, make_float2(xbx, xby), make_float2(vbx, vby));
            } else {
                xbar[d] = make_float2(xbx, xby);
                vbar[d] = make_float2(vbx, vby);
            }
        }
    }
    if (rep >= 0) hand_over();
}

// Gaussian-smoothed distribution of (ta, tb) pairs: h_b += K(r - r_b) dr for
// each unordered pair with r < rmax + 4 sigma, K the unit Gaussian of width sigma
struct RdfConst {
    int ta, tb, nbin;
    float rmax, sigma;
};

__device__ __forceinline__ bool rdf_types(const RdfConst &q, int ti, int tj) {
    return (ti == q.ta && tj == q.tb) || (ti == q.tb && tj == q.ta);
}

// One pair inside the loss's reach, queued by the lane that found it: the
// minimum-image distance and the bins within 4 sigma of it, b0 | b1 << 16.
struct RdfPair {
    float dx, dy, r;
    uint32_t bins;
};

#define RDF_WARPS (BEAD_TPB / 32)
#define RDF_QCAP 64  // per warp: fewer than 32 wait, at most 32 arrive per round

// The CTA's part of its chunk (1 / split of it), its beads of the loss's types
// listed in shared memory and handed to the warps one at a time: the beads of
// a cluster, with their many neighbours, spread over the CTA.  A warp reads the
// types of its bead's window 32 slots a round (each column of cells one
// contiguous slot range, two where it wraps, the ranges found by a lane each)
// and keeps the slots of the types; takes the distances of those 32 at a time
// and queues the pairs inside the reach; and evaluates the queue:
//   VJP == false  half a warp per pair, a lane per bin of its reach: FP64 sums
//                 in shared memory, a copy per half warp, so no two lanes meet
//                 (of the nsum bins from blockIdx.y nsum on); each pair once
//                 (j > d)
//   VJP == true   lane = pair: the derivative of its bins' Gaussians against
//                 the bin weights; the bead's sum is taken in the order of the
//                 window's cells and slots
// blockIdx.z: the configuration.
// What bounds it: the issue of the scan (about 200 slots around each bead of
// the types, most of another type) and of 13 Gaussians per pair and side.
// 24 boxes of 65,536 beads: 186 us (VJP: 272) against 766 (783) with a thread
// per bead and an FP64 shared atomic per pair and bin; one box of 16,384: 10
// (13) against 100 (87), or 1.7 (2.2) in a launch with 31 others (rdf_batch).
template <bool VJP>
__global__ void __launch_bounds__(BEAD_TPB) k_rdf(const __grid_constant__ RdfViews views,
                                                  const RepDev *__restrict__ reps, const Chunk *__restrict__ ch,
                                                  int split, RdfConst q, int nsum, double *__restrict__ hist,
                                                  const double *__restrict__ wgt, float2 *__restrict__ G, size_t N) {
    const StateView sv = views.v[blockIdx.z];
    if (VJP) G += blockIdx.z * N;
    __shared__ int list[BEAD_TPB];
    __shared__ int nlist, next;
    __shared__ RdfPair queue[RDF_WARPS][RDF_QCAP];
    __shared__ int cand[RDF_WARPS][RDF_QCAP];
    __shared__ __align__(16) float part_xy[VJP ? RDF_WARPS : 1][2][VJP ? 36 : 1];
    extern __shared__ __align__(16) double rdf_sh[];
    float *wsh = reinterpret_cast<float *>(rdf_sh);  // VJP: the bins' weights
    const Chunk c = ch[blockIdx.x / split];
    const RepDev &R = reps[c.rep];
    const int tid = (int)threadIdx.x, lane = (int)lane_id(), w = tid >> 5;
    if (tid == 0) {
        nlist = 0;
        next = RDF_WARPS;
    }
    if (VJP)
        for (int k = tid; k < q.nbin; k += BEAD_TPB) wsh[k] = (float)wgt[(size_t)c.rep * q.nbin + k];
    else
        for (int k = tid; k < 2 * RDF_WARPS * nsum; k += BEAD_TPB) rdf_sh[k] = 0.0;
    __syncthreads();
    const int part = BEAD_TPB / split;
    if (tid < part) {
        const int d = c.begin + (int)(blockIdx.x % split) * part + tid;
        if (d < c.end) {
            const int t = (int)(sv.tg[d] >> TYPE_SHIFT);
            if (t == q.ta || t == q.tb) list[atomicAdd(&nlist, 1)] = d;
        }
    }
    __syncthreads();
    const int n = nlist;
    if (n == 0) return;
    const float L = R.L, h = R.halfL;
    const float rc = q.rmax + 4.0f * q.sigma, dr = q.rmax / q.nbin;
    const float inv2s2 = 0.5f / (q.sigma * q.sigma), kn = dr * 0.3989422804f / q.sigma;
    const int ncx = R.ncx, ncy = R.ncy;
    const int rcell = min((int)ceilf(rc * (float)R.icsx), (min(ncx, ncy) - 1) / 2);
    const int32_t *__restrict__ cs = sv.cstart + R.c0;
    const int bin0 = VJP ? 0 : (int)blockIdx.y * nsum, bin1 = min(bin0 + nsum, q.nbin);
    double *acc = rdf_sh + (tid >> 4) * nsum;  // !VJP: this half warp's sums
    float gx = 0.0f;
    int waiting = 0, ncand = 0;
    const uint32_t below = (1u << lane) - 1u;
    // the queued pairs [0, cnt)
    auto evaluate = [&](int cnt) {
        __syncwarp();
        if (VJP) {
            if (lane < cnt) {
                const RdfPair p = queue[w][lane];
                const int b0 = (int)(p.bins & 0xFFFFu), b1 = (int)(p.bins >> 16);
                float dldr = 0.f;
                for (int b = b0; b <= b1; b++) {
                    const float rb = (b + 0.5f) * dr, e = p.r - rb;
                    const float k = kn * __expf(-e * e * inv2s2);
                    dldr += wsh[b] * k * (-e * 2.0f * inv2s2);
                }
                part_xy[w][0][lane] = dldr * p.dx / p.r;
                part_xy[w][1][lane] = dldr * p.dy / p.r;
            } else if (lane < ((cnt + 3) & ~3)) {
                part_xy[w][0][lane] = part_xy[w][1][lane] = 0.0f;
            }
            __syncwarp();
            if (lane < 2) {  // lane 0 sums x, lane 1 sums y, in order
                const float4 *v = reinterpret_cast<const float4 *>(part_xy[w][lane]);
                for (int u = 0; 4 * u < cnt; u++) {
                    const float4 t = v[u];
                    gx += t.x;
                    gx += t.y;
                    gx += t.z;
                    gx += t.w;
                }
            }
        } else {
            for (int u = 0; u < cnt; u += 2) {
                const int e = u + (lane >> 4);
                if (e < cnt) {
                    const float r = queue[w][e].r;
                    const uint32_t bins = queue[w][e].bins;
                    const int b1 = min((int)(bins >> 16), bin1 - 1);
                    for (int b = max((int)(bins & 0xFFFFu), bin0) + (lane & 15); b <= b1; b += 16) {
                        const float rb = (b + 0.5f) * dr, e2 = r - rb;
                        const float k = kn * __expf(-e2 * e2 * inv2s2);
                        acc[b - bin0] += (double)k;
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    };
    for (int it = w; it < n;) {
        const int d = list[it];
        const int ti = (int)(sv.tg[d] >> TYPE_SHIFT);
        const float2 pi = sv.pos[d];
        int cx, cy;
        cell_xy(R, pi.x, pi.y, cx, cy);
        // the distances of candidates [0, cnt), the pairs inside the reach queued
        auto distances = [&](int cnt) {
            __syncwarp();
            RdfPair p;
            bool keep = false;
            if (lane < cnt) {
                const float2 pj = sv.pos[cand[w][lane]];
                p.dx = minimg(pi.x - pj.x, L, h);
                p.dy = minimg(pi.y - pj.y, L, h);
                p.r = sqrtf(p.dx * p.dx + p.dy * p.dy);
                keep = p.r < rc && p.r != 0.0f;
            }
            if (keep) {
                const int b0 = max(0, (int)floorf((p.r - 4.0f * q.sigma) / dr));
                const int b1 = min(q.nbin - 1, (int)floorf((p.r + 4.0f * q.sigma) / dr));
                keep = b0 <= b1 && (VJP || (b1 >= bin0 && b0 < bin1));
                p.bins = (uint32_t)b0 | (uint32_t)b1 << 16;
            }
            const uint32_t m = __ballot_sync(0xffffffffu, keep);
            if (keep) queue[w][waiting + __popc(m & below)] = p;
            waiting += __popc(m);
            if (waiting >= 32) {  // a full round now, the rest to the front
                evaluate(32);
                waiting -= 32;
                RdfPair t;
                if (lane < waiting) t = queue[w][32 + lane];
                __syncwarp();
                if (lane < waiting) queue[w][lane] = t;
            }
        };
        const int lo = cy - rcell, hi = cy + rcell;  // 2 rcell + 1 <= ncy: the rows wrap at one end at most
        for (int g0 = -rcell; g0 <= rcell; g0 += 16) {
            // a lane's range: column g0 + lane / 2, its first rows or, where they wrap, the others
            const int ox = g0 + (lane >> 1);
            int js = 0, je = 0;
            if (ox <= rcell) {
                const int nx = cx + ox < 0 ? cx + ox + ncx : (cx + ox >= ncx ? cx + ox - ncx : cx + ox);
                const int32_t *col = cs + nx * ncy;
                int r0 = max(lo, 0), r1 = min(hi, ncy - 1);  // the rows inside: first unless rows below 0 come before
                const bool other = (lane & 1) != (lo < 0 ? 1 : 0);
                if (other) {
                    r0 = lo < 0 ? lo + ncy : 0;
                    r1 = lo < 0 ? ncy - 1 : hi - ncy;
                }
                if (r0 <= r1) {
                    js = col[r0];
                    je = col[r1 + 1];
                    if (!VJP) js = max(js, d + 1);  // the histogram counts each pair once
                }
            }
            for (uint32_t m = __ballot_sync(0xffffffffu, js < je); m; m &= m - 1) {
                const int from = __ffs(m) - 1;
                const int s = __shfl_sync(0xffffffffu, js, from), e = __shfl_sync(0xffffffffu, je, from);
                for (int base = s; base < e; base += 32) {
                    const int j = base + lane;
                    const bool ok = j < e && j != d && rdf_types(q, ti, (int)(sv.tg[j] >> TYPE_SHIFT));
                    const uint32_t t = __ballot_sync(0xffffffffu, ok);
                    if (ok) cand[w][ncand + __popc(t & below)] = j;
                    ncand += __popc(t);
                    if (ncand >= 32) {
                        distances(32);
                        ncand -= 32;
                        const int c1 = lane < ncand ? cand[w][32 + lane] : 0;
                        __syncwarp();
                        if (lane < ncand) cand[w][lane] = c1;
                    }
                }
            }
        }
        distances(ncand);
        ncand = 0;
        if (VJP) {
            evaluate(waiting);
            waiting = 0;
            const float gy = __shfl_sync(0xffffffffu, gx, 1);
            if (lane == 0) G[d] = make_float2(gx, gy);
            gx = 0.0f;
        }
        int nxt = 0;
        if (lane == 0) nxt = atomicAdd(&next, 1);
        it = __shfl_sync(0xffffffffu, nxt, 0);
    }
    if (!VJP) {
        evaluate(waiting);
        __syncthreads();
        for (int k = tid; bin0 + k < bin1; k += BEAD_TPB) {
            double sum = 0.0;
            for (int u = 0; u < 2 * RDF_WARPS; u++) sum += rdf_sh[u * nsum + k];
            if (sum != 0.0) atomicAdd(&hist[(size_t)c.rep * q.nbin + bin0 + k], sum);
        }
    }
}

// the adjoint of the update alone, after the branched shapes' k_mol_vjp has added its share to xb
__global__ void __launch_bounds__(BEAD_TPB) k_adj_update(const uint32_t *__restrict__ tg,
                                                         const RepDev *__restrict__ reps, const Chunk *__restrict__ ch,
                                                         const float2 *__restrict__ xb, const float2 *__restrict__ vb,
                                                         AdjUpdate up) {
    const Chunk c = ch[blockIdx.x];
    const int d = c.begin + (int)threadIdx.x;
    if (d < c.end) adj_update(up, reps[c.rep], d, (int)(tg[d] >> TYPE_SHIFT), xb[d], vb[d]);
}

// cotangents of the window's start state into gid order: x_bar(0) gains the part
// that flows through the start forces (xb = J_x^T F_bar(0)), and the predicted
// velocity's cotangent is that force VJP's vb; vh_bar(0) is V as it stands
__global__ void __launch_bounds__(BEAD_TPB) k_adj_state(const uint32_t *__restrict__ tg, const RepDev *__restrict__ reps,
                                                        const Chunk *__restrict__ ch, const float2 *__restrict__ X,
                                                        const float2 *__restrict__ V, const float2 *__restrict__ xb,
                                                        const float2 *__restrict__ vb, float2 *__restrict__ oX,
                                                        float2 *__restrict__ oV, float2 *__restrict__ oVT) {
    const Chunk c = ch[blockIdx.x];
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end) return;
    const uint32_t g = (tg[d] & GID_MASK) + (uint32_t)reps[c.rep].b0;
    const float2 x = X[d], a = xb[d];
    oX[g] = make_float2(x.x + a.x, x.y + a.y);
    oV[g] = V[d];
    oVT[g] = vb[d];
}

// The bonded terms of the branched shapes (the template terms of
// k_mol_forces): one thread per molecule (its first bead) adds each of its
// beads' share to x_bar after k_force_vjp, so no two threads write one bead.
// Bond (i, j), d = x_j - x_i, F_i = kb (1 - r0/r) d = -F_j, c = g_i - g_j:
//   d(c.F_i)/dd = kb ((1 - r0/r) c + r0 (c.d) d / r^3),  d(c.F_i)/dkb = (1 - r0/r) (c.d)
// Angle (i, j, k): x_bar_i += dphi/da, x_bar_j -= dphi/da - dphi/dc, x_bar_k -= dphi/dc.
__global__ void __launch_bounds__(BEAD_TPB) k_mol_vjp(StateView sv, const RepDev *__restrict__ reps,
                                                      const Chunk *__restrict__ ch, const dpd_template *__restrict__ mol,
                                                      const float2 *__restrict__ g, float2 *__restrict__ xbar,
                                                      double *__restrict__ grad) {
    const Chunk c = ch[blockIdx.x];
    const RepDev &R = reps[c.rep];
    if (R.arch == 0) return;
    const int d = c.begin + (int)threadIdx.x;
    double gkb = 0.0;
    if (d < c.end) {
        const int2 lk0 = sv.link[d];
        if (lk0.x < 0 && lk0.y >= 0) {
            const dpd_template &M = mol[c.rep];
            const int ml = M.mlen;
            int sl[DPD_MAXML];
            float2 p[DPD_MAXML], gg[DPD_MAXML], xb[DPD_MAXML];
            int n = 0;
            for (int q = d; q >= 0 && n < ml; q = sv.link[q].y) {
                sl[n] = q;
                p[n] = sv.pos[q];
                gg[n] = g[q];
                xb[n] = make_float2(0.0f, 0.0f);
                n++;
            }
            if (n == ml) {  // (an incomplete molecule raised DPD_F_CHAIN in the forward pass)
                const float L = R.L, h = R.halfL, kb = R.kb;
                for (int q = 0; q < M.nb; q++) {
                    const int i = M.bi[q], j = M.bj[q];
                    const float dx = minimg(p[j].x - p[i].x, L, h), dy = minimg(p[j].y - p[i].y, L, h);
                    const float r = sqrtf(dx * dx + dy * dy), r0 = (float)M.br0[q];
                    const float cx = gg[i].x - gg[j].x, cy = gg[i].y - gg[j].y, cd = cx * dx + cy * dy;
                    const float u = 1.0f - r0 / r, k3 = kb * r0 * cd / (r * r * r);
                    const float tx = kb * u * cx + k3 * dx, ty = kb * u * cy + k3 * dy;  // d(c.F_i)/dd
                    xb[i].x -= tx;
                    xb[i].y -= ty;
                    xb[j].x += tx;
                    xb[j].y += ty;
                    gkb += (double)(u * cd);
                }
                for (int q = 0; q < M.na; q++) {
                    const int i = M.ai[q], j = M.aj[q], k = M.ak[q];
                    const float2 a = make_float2(minimg(p[j].x - p[i].x, L, h), minimg(p[j].y - p[i].y, L, h));
                    const float2 cc = make_float2(minimg(p[k].x - p[j].x, L, h), minimg(p[k].y - p[j].y, L, h));
                    const float2 da = make_float2(gg[j].x - gg[i].x, gg[j].y - gg[i].y);
                    const float2 dc = make_float2(gg[k].x - gg[j].x, gg[k].y - gg[j].y);
                    float2 pa, pc;
                    angle_hvp(a, cc, da, dc, M.akind[q], (float)M.aK[q], (float)M.ac0[q], pa, pc);
                    xb[i].x += pa.x;
                    xb[i].y += pa.y;
                    xb[j].x -= pa.x - pc.x;
                    xb[j].y -= pa.y - pc.y;
                    xb[k].x -= pc.x;
                    xb[k].y -= pc.y;
                }
                for (int e = 0; e < ml; e++) {
                    const float2 o = xbar[sl[e]];
                    xbar[sl[e]] = make_float2(o.x + xb[e].x, o.y + xb[e].y);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gkb += __shfl_down_sync(0xffffffffu, gkb, o);
    if (lane_id() == 0 && gkb != 0.0) atomicAdd(&grad[(size_t)c.rep * NGRAD + DPD_MAXT * DPD_MAXT + 1], gkb);
}

void launch_force_vjp(const StateView &sv, long long step, const RepDev *rep, const Chunk *bch, int nbch,
                      const float2 *g, float2 *xbar, float2 *vbar, double *grad, double *gsum, int nrep, bool stir,
                      const dpd_template *mol, cudaStream_t s, const long long *step_base, const AdjUpdate *up) {
    if (stir) {
        cudaMemsetAsync(gsum, 0, (size_t)nrep * sizeof(double), s);
        k_gsum<<<nbch, BEAD_TPB, 0, s>>>(rep, bch, g, gsum);
    }
    // Lanes per bead and CTAs an SM: as many lanes as keep all tasks on the GPU at once (a small box is latency).  A
    // larger box is rounds of tasks, of 444 with (4, 3) and of 592 with (2, 4), and one of the latter takes 2.5 of the
    // former: two lanes where that is less in all, and past six rounds of four.  us a launch with (lanes, CTAs an SM),
    // density 4:
    //   beads      (8, 2)  (4, 2)  (4, 3)  (2, 2)  (2, 4)
    //   4,096         9.6    12.3    12.7    18.8    20.0
    //   16,384       15.2    14.0    14.6    19.4    21.0
    //   25,600       20.3    21.4    16.8    22.2    23.6
    //   36,864       24.2    20.9    25.5    21.3    22.8
    //   50,176       32.2    26.8    25.1    30.5    24.2
    //   65,536       37.0    33.6    32.7    32.5    30.5
    //   82,944       46.8    42.1    35.1    45.2    49.2
    //   102,400      55.2    46.3    41.7    43.4    52.0
    //   131,044      67.2    53.3    53.2    53.5    50.6
    //   144,400      74.0    60.4    57.8    56.1    53.8
    //   160,000      83.0    70.1    64.0    70.3    65.4
    //   179,776      89.2    70.1    67.3    65.9    66.1
    //   204,304     100.8    78.6    75.3    75.1    70.2
    //   1,048,576   484     375     339     335     287
    const bool update = up && !mol;  // the branched shapes add their share first
    const AdjUpdate none{};
    auto go = [&](auto kern, int lpb, int per_sm) {
        const int ntask = nbch * lpb;
        kern<<<std::min(ntask, per_sm * 148), VJP_TPB, 0, s>>>(sv, step, rep, bch, ntask, g, xbar, vbar,
                                                             update ? *up : none, grad, gsum, step_base);
    };
    if (nbch * 8 <= 2 * 148) go(update ? k_force_vjp<8, 2, true> : k_force_vjp<8, 2, false>, 8, 2);
    else if (nbch * 4 <= 2 * 148) go(update ? k_force_vjp<4, 2, true> : k_force_vjp<4, 2, false>, 4, 2);
    else if (nbch * 4 > 3 * 148 && nbch * 2 <= 2 * 148)
        go(update ? k_force_vjp<2, 2, true> : k_force_vjp<2, 2, false>, 2, 2);
    else if (nbch <= 666 && 5 * ((nbch * 2 + 591) / 592) > 2 * ((nbch * 4 + 443) / 444))
        go(update ? k_force_vjp<4, 3, true> : k_force_vjp<4, 3, false>, 4, 3);
    else go(update ? k_force_vjp<2, 4, true> : k_force_vjp<2, 4, false>, 2, 4);
    if (mol) {
        k_mol_vjp<<<nbch, BEAD_TPB, 0, s>>>(sv, rep, bch, mol, g, xbar, grad);
        if (up) k_adj_update<<<nbch, BEAD_TPB, 0, s>>>(sv.tg, rep, bch, xbar, vbar, *up);
    }
}

// CTAs per chunk of beads: the whole chunk, or halves, quarters or eighths of
// it while that leaves the GPU short of eight CTAs per SM
static int rdf_split(int nbch) {
    int split = 1;
    while (split < 8 && nbch * split < 8 * 148) split *= 2;
    return split;
}

// A configuration of a small box is a fraction of a wave, its time that of the
// slowest warp: one of 16,384 beads alone takes 10 us (VJP: 13), 32 together 1.7
// (2.2) each.  So as many are taken together as make two waves of whole chunks;
// a box with that many chunks alone gains nothing by it.
int rdf_batch(int nbch) { return std::max(1, std::min(RDF_VIEWS, 2 * 8 * 148 / nbch)); }

void launch_rdf(const RdfViews &views, int nv, const RepDev *rep, const Chunk *bch, int nbch, int ta, int tb, int nbin,
                float rmax, float sigma, double *hist, cudaStream_t s) {
    RdfConst q{ta, tb, nbin, rmax, sigma};
    const int split = rdf_split(nbch * nv);
    // up to 256 bins (32 KB of sums a CTA) in one pass over the pairs, more in blocks of 256
    const int nsum = std::min(nbin, 256);
    k_rdf<false><<<dim3(nbch * split, (nbin + nsum - 1) / nsum, nv), BEAD_TPB, 2 * RDF_WARPS * nsum * sizeof(double),
                   s>>>(views, rep, bch, split, q, nsum, hist, nullptr, nullptr, 0);
}

void launch_rdf_vjp(const RdfViews &views, int nv, const RepDev *rep, const Chunk *bch, int nbch, int ta, int tb,
                    int nbin, float rmax, float sigma, const double *wgt, float2 *G, size_t N, cudaStream_t s) {
    RdfConst q{ta, tb, nbin, rmax, sigma};
    const int split = rdf_split(nbch * nv);
    k_rdf<true><<<dim3(nbch * split, 1, nv), BEAD_TPB, nbin * sizeof(float), s>>>(views, rep, bch, split, q, 0, nullptr,
                                                                                wgt, G, N);
}

void launch_adj_state(const uint32_t *tg, const RepDev *rep, const Chunk *bch, int nbch, const float2 *X,
                      const float2 *V, const float2 *xb, const float2 *vb, float2 *oX, float2 *oV, float2 *oVT,
                      cudaStream_t s) {
    k_adj_state<<<nbch, BEAD_TPB, 0, s>>>(tg, rep, bch, X, V, xb, vb, oX, oV, oVT);
}

// the device's step number, on the stream and without a copy or a wait
__global__ void k_set_step(long long *__restrict__ step, long long v) { *step = v; }

void launch_set_step(long long *step, long long v, cudaStream_t s) { k_set_step<<<1, 1, 0, s>>>(step, v); }

// ---------------------------------------------------------------- a fit iteration without the host
//
// dpd_fit_graph captures one optimizer iteration (the window, its adjoint, the
// loss and the parameter update) as a CUDA graph and replays it: every value
// that changes from one iteration to the next lives on the device (FitDev).

__global__ void k_fit_begin(const long long *__restrict__ step, FitDev *__restrict__ fd) { fd->base = *step; }

__global__ void k_set_step_rel(long long *__restrict__ step, const FitDev *__restrict__ fd, long long off) {
    *step = fd->base + off;
}

// The smoothed-RDF loss of each replica (one block each) and the weights dL/dh
// of its bins, as the host computes them for dpd_window_adjoint:
// g = h / last_steps * L^2 / (npairs 2 pi r_b dr), loss = mean over bins of
// (g - target)^2, w = 2 (g - target) / nbin * L^2 / (npairs 2 pi r_b dr) / last_steps.
// The loss goes to loss_out[iter * nrep + replica].
__global__ void k_rdf_loss(const RepDev *__restrict__ reps, const double *__restrict__ hist,
                           const long long *__restrict__ npairs, const double *__restrict__ target, int nbin,
                           double rmax, int last_steps, double *__restrict__ loss_out, double *__restrict__ wgt,
                           const FitDev *__restrict__ fd) {
    __shared__ double red[32];
    const int r = (int)blockIdx.x, nrep = (int)gridDim.x;
    const double L = (double)reps[r].L, area = L * L, dr = rmax / nbin;
    const long long np = npairs[r];
    double sum = 0.0;
    for (int b = (int)threadIdx.x; b < nbin; b += (int)blockDim.x) {
        const double rb = (b + 0.5) * dr;
        const double norm = np > 0 ? area / ((double)np * 2.0 * M_PI * rb * dr) : 0.0;
        const double g = hist[(size_t)r * nbin + b] / last_steps * norm;
        const double e = g - target[(size_t)r * nbin + b];
        sum += e * e;
        wgt[(size_t)r * nbin + b] = 2.0 * e / nbin * norm / last_steps;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane_id() == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
        loss_out[(size_t)fd->iter * nrep + r] = t / nbin;
    }
}

// The optimizer step of the shared a_ij (one thread per fitted slot): the
// gradient summed over the replicas in replica order, then Adam as
// torch.optim.Adam takes it (no weight decay): m += (1 - b1)(g - m),
// v = b2 v + (1 - b2) g^2, a -= lr / (1 - b1^t) m / (sqrt(v) / sqrt(1 - b2^t) + eps).
// The new value goes into a_ij and a_ji of every replica; the gradient and the
// value the window ran with go to grad_out / value_out[iter * nfit + k].
__global__ void k_fit_update(RepDev *__restrict__ reps, int nrep, const double *__restrict__ grad,
                             FitDev *__restrict__ fd, double *__restrict__ grad_out, double *__restrict__ value_out) {
    const int k = (int)threadIdx.x, it = fd->iter;
    if (k < fd->nfit) {
        const int slot = fd->slot[k];
        double g = 0.0;
        for (int r = 0; r < nrep; r++) g += grad[(size_t)r * NGRAD + slot];
        const double t = (double)(it + 1);
        const double m = fd->m[k] + (1.0 - fd->beta1) * (g - fd->m[k]);
        const double v = fd->beta2 * fd->v[k] + (1.0 - fd->beta2) * g * g;
        fd->m[k] = m;
        fd->v[k] = v;
        const double bc1 = 1.0 - pow(fd->beta1, t), bc2 = 1.0 - pow(fd->beta2, t);
        const double denom = sqrt(v) / sqrt(bc2) + fd->eps;
        const double val = fd->value[k] - fd->lr / bc1 * m / denom;
        grad_out[(size_t)it * fd->nfit + k] = g;
        value_out[(size_t)it * fd->nfit + k] = fd->value[k];
        fd->value[k] = val;
        const int i = slot / DPD_MAXT, j = slot % DPD_MAXT;
        for (int r = 0; r < nrep; r++) {
            reps[r].a[i * DPD_MAXT + j] = (float)val;
            reps[r].a[j * DPD_MAXT + i] = (float)val;
        }
    }
    __syncthreads();
    if (k == 0) fd->iter = it + 1;
}

void launch_fit_begin(long long *step, FitDev *fd, cudaStream_t s) { k_fit_begin<<<1, 1, 0, s>>>(step, fd); }

void launch_set_step_rel(long long *step, const FitDev *fd, long long off, cudaStream_t s) {
    k_set_step_rel<<<1, 1, 0, s>>>(step, fd, off);
}

void launch_rdf_loss(const RepDev *rep, int nrep, const double *hist, const long long *npairs, const double *target,
                     int nbin, double rmax, int last_steps, double *loss_out, double *wgt, const FitDev *fd,
                     cudaStream_t s) {
    k_rdf_loss<<<nrep, 256, 0, s>>>(rep, hist, npairs, target, nbin, rmax, last_steps, loss_out, wgt, fd);
}

void launch_fit_update(RepDev *rep, int nrep, const double *grad, FitDev *fd, double *grad_out, double *value_out,
                       cudaStream_t s) {
    k_fit_update<<<1, DPD_MAXT * DPD_MAXT, 0, s>>>(rep, nrep, grad, fd, grad_out, value_out);
}
