// dpd_chem.cu -- the lipid chemistry pass (sm_100a).
//
// Three stages per chemistry step, each decided on the state the previous
// stage left (kernel boundaries), every decision a keyed Philox draw of
// (seed, step, salt, gid) -- the reference's counter-based mechanism
// (cel/engine/oercel.c:819-826) -- and every conflict resolved by the lowest
// requesting gid (atomicMin claim, then a check by each requester; the
// reference GPU port resolves its lock rounds the same way, lowest rank wins,
// cel/engine_gpu/oercel_gpu.cu:1746-1757).  The draws do not depend on the
// state, so one pass over the beads (fused into the permute kernel of the step,
// or k_chem_scan for the phase entry point) applies the breaks and lists the
// few beads whose growth or bonding draw succeeded; the later stages run over
// those lists only.
//   1 brk : an H whose next bead is T breaks the bond with p_break;
//   2 grow: a P with >= n_t_min T beads within r_grow, with p_grow, becomes a
//           T bonded behind its nearest growable H-terminated chain end
//           (the tail of a chain headed by H and shorter than max_chain, or a
//           lone H) within r_grow;
//   3 bond: a free T, with p_bond, bonds to its nearest free H within r_bond.
// Nearest = smallest squared FP32 distance, ties to the lower gid
// (oercel.c:1387-1396).
#include "dpd_chem.cuh"

// stage 1 on a sorted state in place (the phase entry point dpd_chemistry)
__global__ void __launch_bounds__(BEAD_TPB) k_chem_scan(Bufs b, int cur, const RepDev *__restrict__ reps,
                                                        const Chunk *__restrict__ ch) {
    const Chunk c = ch[blockIdx.x];
    const RepDev &R = reps[c.rep];
    const long long step = *b.step;
    if (!chem_due(R, step)) return;
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end) return;
    const uint32_t *tg = b.tg[cur];
    int2 *link = b.link[cur];
    const uint32_t t0 = tg[d];
    const int t = link[d].y;
    if (type_of(t0) == T_H && t >= 0 && h_breaks(R, step, t0, tg[t])) {
        link[d].y = -1;
        link[t].x = -1;
        const float2 p = b.pos[cur][d];
        push_event(b, step, 1, t0 & GID_MASK, tg[t] & GID_MASK, p.x, p.y, c.rep);
    }
    chem_candidate(b, R, step, c.rep, d, t0);
}

#define LIST_GRID 148

// Stages 2 and 3 over the step's candidate lists.  Every request is made at
// once, a warp per listed P (growth) or T (bonding); the last CTA then applies
// the growth claims, makes the bonding claims and applies those.  A bonding
// request made before the growth is the one made after it unless its H went to
// a growing chain: growth links a P to the tail of a chain or to a lone H, so it
// takes free H beads away and touches no other bead that bonding looks at.  Such
// a request is made again.
// What bounds it: latency, a chain of about a dozen dependent loads a stage for
// a few dozen list entries.  1,048,576 beads with a check every step: 144.6 us a
// step against 147.2 with a kernel for each stage.
__global__ void __launch_bounds__(BEAD_TPB) k_chem_lists(Bufs b, int cur, const RepDev *__restrict__ reps) {
    pdl_begin();
    const int ng = (int)b.status->n_grow, nb = (int)b.status->n_bond;
    if (ng + nb == 0) return;  // (the same in every CTA: the counter of last_cta stays at rest)
    const int nw = (int)(gridDim.x * blockDim.x) >> 5, lane = (int)lane_id();
    int32_t *found = b.req + ng;  // the bonding requests behind the growth requests (a bead is in one list)
    for (int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); k < ng + nb; k += nw) {
        if (k < ng) {
            chem_grow_req_one(b, cur, reps, k, lane);
        } else {
            const int e = chem_bond_find(b, cur, reps, b.bond_list[k - ng], lane);
            if (lane == 0) found[k - ng] = e;
        }
    }
    if (!last_cta(&b.status->done)) return;
    const long long step = *b.step;
    for (int k = (int)threadIdx.x; k < ng; k += (int)blockDim.x) chem_grow_apply_one(b, cur, k, step);
    __syncthreads();
    const int rounds = (nb + (int)blockDim.x - 1) / (int)blockDim.x;
    for (int r = 0; r < rounds; r++) {
        const int k = r * (int)blockDim.x + (int)threadIdx.x;
        int2 it = make_int2(0, 0);
        int e = -1;
        if (k < nb) {
            it = b.bond_list[k];
            e = __ldcg(found + k);
        }
        const int2 le = e >= 0 ? b.link[cur][e] : make_int2(-1, -1);
        for (unsigned m = __ballot_sync(0xffffffffu, le.x >= 0 || le.y >= 0); m; m &= m - 1) {
            const int from = __ffs(m) - 1;
            const int2 w = make_int2(__shfl_sync(0xffffffffu, it.x, from), __shfl_sync(0xffffffffu, it.y, from));
            const int again = chem_bond_find(b, cur, reps, w, lane);
            if (lane == from) {
                e = again;
                found[k] = again;
            }
        }
        if (e >= 0) atomicMin(b.claim + e, b.tg[cur][it.x] & GID_MASK);
    }
    __syncthreads();
    for (int k = (int)threadIdx.x; k < nb; k += (int)blockDim.x) {
        const int e = __ldcg(found + k);
        if (e >= 0) chem_bond_apply_one(b, cur, b.bond_list[k], e, step);
    }
}

int chem_kernel_count() { return 1; }

void launch_chem_scan(const Bufs &b, int cur, const RepDev *rep, const Chunk *bch, int nbch, cudaStream_t s) {
    k_chem_scan<<<nbch, BEAD_TPB, 0, s>>>(b, cur, rep, bch);
}

void launch_chem_lists(const Bufs &b, int cur, const RepDev *rep, cudaStream_t s) {
    launch_pdl(k_chem_lists, LIST_GRID, BEAD_TPB, 0, s, b, cur, rep);
}
