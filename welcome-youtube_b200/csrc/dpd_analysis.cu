// dpd_analysis.cu -- analysis of a replica's configuration on the GPU: clusters
// of beads of one type and their neighbour fraction (the reference's
// `snapcheck.py tclust`, cel/engine/tests/snapcheck.py:122-144).
//
// Two beads of type t are joined when their distance is <= rcut (rcut <= 1,
// so the 3 x 3 cells around a bead hold every partner); the clusters are the
// connected components.  A lock-free union-find over the bead slots links the
// larger root under the smaller one with a compare-and-swap, so every cluster
// ends with its lowest slot as root whatever the order of the links; full
// path compression then gives each bead its root.  The neighbour counts are
// those of the reference: for every bead of type t, the beads of any type and
// of type t within 1.0 (self excluded).  Comparisons are those of FP64 distances
// from the FP32 positions with the minimum image, as the reference computes them
// from its snapshot.
#include "dpd_device.cuh"

namespace {

__device__ __forceinline__ int uf_find(int *parent, int i) {
    // path halving; parents only ever decrease, so the walk ends at the root
    // within as many steps as there are beads (GID_MASK bounds that)
    for (int it = 0; it <= (int)GID_MASK; it++) {
        const int p = __ldcg(parent + i);
        if (p == i) return i;
        const int g = __ldcg(parent + p);
        if (g != p) atomicCAS(parent + i, p, g);
        i = g;
    }
    return i;
}

__device__ __forceinline__ void uf_union(int *parent, int a, int b, DevStatus *status) {
    for (int it = 0; it < 4096; it++) {
        a = uf_find(parent, a);
        b = uf_find(parent, b);
        if (a == b) return;
        const int lo = a < b ? a : b, hi = a < b ? b : a;
        if (atomicCAS(parent + hi, hi, lo) == hi) return;  // hi was still a root: linked
        a = lo;                                            // someone moved hi first: find again
        b = hi;
    }
    raise_flag(status, DPD_F_ANALYSIS);
}

__device__ __forceinline__ double min_image(double d, double L) { return d - L * rint(d / L); }

__device__ __forceinline__ double exact_r2(float2 pi, float2 pj, double L) {
    const double dx = min_image((double)pj.x - (double)pi.x, L), dy = min_image((double)pj.y - (double)pi.y, L);
    return dx * dx + dy * dy;
}

// Contact searches.  One bead in five or fewer is of the type, so a CTA lists
// its beads of the type in shared memory and NEAR_LANES lanes share each: they
// take the slots of its 3 x 3 cells in turn (cells are column-major: three
// contiguous ranges, two each where the rows wrap).  Squared distances are
// FP32; one within near_eps of a threshold is taken again in FP64 with the
// reference's minimum image, so every comparison is the FP64 one.  786,432
// beads: k_uf_link 115 us against 168, k_agg_link 105 against 128, with a thread
// per bead and two FP64 divisions per candidate (what is left is the union-find's
// own chains).
constexpr int NEAR_LANES = 8;

// Bound of the FP32 error of a squared distance up to about 1: a coordinate
// difference across the box edge is off by half an ulp of L at most (6e-8 L),
// others are exact, so 2 sqrt(2) of that, and a few roundings near 1.
__device__ __forceinline__ float near_eps(float L) { return 2e-6f + 2e-7f * L; }

// calls near(j, squared distance) for the slots j != d of bead d's cells within
// the FP32 reach of lim, from this lane's share of them; same as exact_r2 where
// it could matter for lim or lim2
template <class F>
__device__ __forceinline__ void each_near(const float2 *__restrict__ pos, const RepDev &R,
                                          const int32_t *__restrict__ cs, int d, int sub, double lim, double lim2,
                                          F near) {
    const float2 pi = pos[d];
    const float L = R.L, h = R.halfL, f1 = (float)lim, f2 = (float)lim2, eps = near_eps(L);
    const int ncx = R.ncx, ncy = R.ncy;
    int cx, cy;
    cell_xy(R, pi.x, pi.y, cx, cy);
    for (int ox = -1; ox <= 1; ox++) {
        const int nx = cx + ox < 0 ? ncx - 1 : (cx + ox >= ncx ? 0 : cx + ox);
        const int32_t *col = cs + nx * ncy;
        for (int seg = -1; seg <= 1; seg++) {  // the rows below 0, inside, and past the top
            const int r0 = max(cy - 1, seg * ncy), r1 = min(cy + 1, seg * ncy + ncy - 1);
            if (r0 > r1) continue;
            const int je = col[r1 - seg * ncy + 1];
            for (int j = col[r0 - seg * ncy] + sub; j < je; j += NEAR_LANES) {
                if (j == d) continue;
                const float2 pj = pos[j];
                const float dx = minimg(pj.x - pi.x, L, h), dy = minimg(pj.y - pi.y, L, h);
                const float q = dx * dx + dy * dy;
                if (q > f1 + eps) continue;
                double r2 = (double)q;
                if (fabsf(q - f1) <= eps || fabsf(q - f2) <= eps) r2 = exact_r2(pi, pj, (double)L);
                if (r2 <= lim) near(j, r2);
            }
        }
    }
}

// the CTA's beads d for which mine is true, listed in shared memory; returns their number
__device__ __forceinline__ int list_beads(bool mine, int d, int *list, int *n) {
    if (threadIdx.x == 0) *n = 0;
    __syncthreads();
    if (mine) list[atomicAdd(n, 1)] = d;
    __syncthreads();
    return *n;
}

// sums over the CTA of up to five values and a maximum, one atomic each
__device__ __forceinline__ void cta_sums(const long long *v, int nv, unsigned mx, unsigned long long *const *dst,
                                         unsigned long long *dst_max) {
    __shared__ long long red[BEAD_TPB / 32][6];
    const int w = (int)threadIdx.x >> 5;
    for (int k = 0; k < nv; k++) {
        const long long t = warp_sum_ll(v[k]);
        if (lane_id() == 0) red[w][k] = t;
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane_id() == 0) red[w][5] = mx;
    __syncthreads();
    const int k = (int)threadIdx.x;
    if (k < nv) {
        long long t = 0;
        for (int q = 0; q < BEAD_TPB / 32; q++) t += red[q][k];
        if (t) atomicAdd(dst[k], (unsigned long long)t);
    }
    if (k == 5 && dst_max) {
        long long t = 0;
        for (int q = 0; q < BEAD_TPB / 32; q++) t = max(t, red[q][5]);
        if (t) atomicMax(dst_max, (unsigned long long)t);
    }
}

}  // namespace

// parent[i] = i for the beads of type t of the replica, -1 for the others
__global__ void __launch_bounds__(BEAD_TPB) k_uf_init(Bufs b, int cur, const RepDev *__restrict__ reps,
                                                      const Chunk *__restrict__ ch, int rep_index, int t,
                                                      int *__restrict__ parent, int *__restrict__ size) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end) return;
    parent[d] = (int)(b.tg[cur][d] >> TYPE_SHIFT) == t ? d : -1;
    size[d] = 0;
}

// joins each bead of type t with the type-t beads of higher slot within rcut,
// and counts its neighbours within 1.0 (all types; type t)
__global__ void __launch_bounds__(BEAD_TPB) k_uf_link(Bufs b, int cur, const RepDev *__restrict__ reps,
                                                      const Chunk *__restrict__ ch, int rep_index, int t, double rcut,
                                                      int *__restrict__ parent, unsigned long long *__restrict__ acc) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    __shared__ int list[BEAD_TPB], nlist;
    const RepDev &R = reps[c.rep];
    const int d0 = c.begin + (int)threadIdx.x;
    const int n = list_beads(d0 < c.end && parent[d0] >= 0, d0, list, &nlist);
    const uint32_t *__restrict__ tg = b.tg[cur];
    const int sub = (int)threadIdx.x % NEAR_LANES;
    const double r2c = rcut * rcut;
    long long cnt[2] = {0, 0};
    for (int k = (int)threadIdx.x / NEAR_LANES; k < n; k += BEAD_TPB / NEAR_LANES) {
        const int d = list[k];
        each_near(b.pos[cur], R, b.cstart + R.c0, d, sub, 1.0, r2c, [&](int j, double r2) {
            const bool same = (int)(tg[j] >> TYPE_SHIFT) == t;
            cnt[0]++;
            cnt[1] += same;
            if (same && j > d && r2 <= r2c) uf_union(parent, d, j, b.status);
        });
    }
    unsigned long long *const dst[2] = {acc + 0, acc + 1};
    cta_sums(cnt, 2, 0u, dst, nullptr);
}

// each bead's root, and the bead counted in its cluster's size
__global__ void __launch_bounds__(BEAD_TPB) k_uf_label(const Chunk *__restrict__ ch, int rep_index,
                                                       int *__restrict__ parent, int *__restrict__ size) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end || parent[d] < 0) return;
    const int r = uf_find(parent, d);
    atomicAdd(size + r, 1);
}

// per cluster root: the cluster count, the largest size and the sum of squared sizes
__global__ void __launch_bounds__(BEAD_TPB) k_uf_stats(const Chunk *__restrict__ ch, int rep_index,
                                                       const int *__restrict__ parent, const int *__restrict__ size,
                                                       unsigned long long *__restrict__ acc) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    long long nc = 0, sq = 0, nb = 0;
    unsigned mx = 0;
    if (d < c.end && parent[d] == d) {
        const long long s = size[d];
        nc = 1;
        sq = s * s;
        nb = s;
        mx = (unsigned)s;
    }
    const long long v[3] = {nc, sq, nb};
    unsigned long long *const dst[3] = {acc + 2, acc + 3, acc + 4};
    cta_sums(v, 3, mx, dst, acc + 5);
}

// ---------------------------------------------------------------- membrane aggregates

// The first two stages of the reference's cell detection (cel/tools/cells.py:
// lipid_molecules 68-86, detect 345-366): molecules are the components of the
// bonds between lipid beads (H, T), aggregates the components of the molecules
// joined by tail-tail contacts (T-T distance <= r_tail).  One union-find over
// the lipid beads takes both kinds of edges: the prev/next links (every bead of
// a molecule is linked in template order) and the T-T contacts.

__global__ void __launch_bounds__(BEAD_TPB) k_agg_init(Bufs b, int cur, const Chunk *__restrict__ ch, int rep_index,
                                                       int *__restrict__ parent, int *__restrict__ size,
                                                       int *__restrict__ minlab) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end) return;
    const int t = (int)(b.tg[cur][d] >> TYPE_SHIFT);
    parent[d] = (t == 1 || t == 2) ? d : -1;
    size[d] = 0;
    minlab[d] = 0x7fffffff;
}

__global__ void __launch_bounds__(BEAD_TPB) k_agg_link(Bufs b, int cur, const RepDev *__restrict__ reps,
                                                       const Chunk *__restrict__ ch, int rep_index, double r_tail,
                                                       int *__restrict__ parent) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    __shared__ int list[BEAD_TPB], nlist;
    const RepDev &R = reps[c.rep];
    const uint32_t *__restrict__ tg = b.tg[cur];
    const int d0 = c.begin + (int)threadIdx.x;
    const bool lipid = d0 < c.end && parent[d0] >= 0;
    if (lipid) {
        const int nx = b.link[cur][d0].y;
        if (nx >= 0 && parent[nx] >= 0) uf_union(parent, d0, nx, b.status);
    }
    const int n = list_beads(lipid && (int)(tg[d0] >> TYPE_SHIFT) == 2, d0, list, &nlist);
    const int sub = (int)threadIdx.x % NEAR_LANES;
    const double r2c = r_tail * r_tail;
    for (int k = (int)threadIdx.x / NEAR_LANES; k < n; k += BEAD_TPB / NEAR_LANES) {
        const int d = list[k];
        each_near(b.pos[cur], R, b.cstart + R.c0, d, sub, r2c, r2c, [&](int j, double) {
            if (j > d && (int)(tg[j] >> TYPE_SHIFT) == 2) uf_union(parent, d, j, b.status);
        });
    }
}

// per lipid bead: its root; molecules (beads without prev) counted per aggregate;
// the aggregate's smallest gid
__global__ void __launch_bounds__(BEAD_TPB) k_agg_label(Bufs b, int cur, const Chunk *__restrict__ ch, int rep_index,
                                                        int *__restrict__ parent, int *__restrict__ size,
                                                        int *__restrict__ minlab) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    if (d >= c.end || parent[d] < 0) return;
    const int r = uf_find(parent, d);
    if (b.link[cur][d].x < 0) atomicAdd(size + r, 1);
    atomicMin(minlab + r, (int)(b.tg[cur][d] & GID_MASK));
}

// per aggregate root: counts (acc[2] aggregates, [3] membranes, [4] molecules,
// [5] largest, [6] molecules in small aggregates); per bead (gid order) its
// aggregate's smallest gid, -1 for other beads
__global__ void __launch_bounds__(BEAD_TPB) k_agg_stats(Bufs b, int cur, const Chunk *__restrict__ ch, int rep_index,
                                                        int nrep_beads, int min_lipids, const int *__restrict__ parent,
                                                        const int *__restrict__ size, const int *__restrict__ minlab,
                                                        unsigned long long *__restrict__ acc, int32_t *out_label) {
    const Chunk c = ch[blockIdx.x];
    if (c.rep != rep_index) return;
    const int d = c.begin + (int)threadIdx.x;
    long long na = 0, nm = 0, nmol = 0, small = 0;
    unsigned mx = 0;
    if (d < c.end) {
        const int p = parent[d];
        const int g = (int)(b.tg[cur][d] & GID_MASK);
        if (out_label && g < nrep_beads) out_label[g] = p >= 0 ? __ldcg(minlab + uf_find((int *)parent, d)) : -1;
        if (p == d) {
            const int s = size[d];
            na = 1;
            nm = s >= min_lipids;
            nmol = s;
            small = s < min_lipids ? s : 0;
            mx = (unsigned)s;
        }
    }
    const long long v[4] = {na, nm, nmol, small};
    unsigned long long *const dst[4] = {acc + 2, acc + 3, acc + 4, acc + 6};
    cta_sums(v, 4, mx, dst, acc + 5);
}

void launch_aggregates(const Bufs &b, int cur, const RepDev *rep, const Chunk *bch, int nbch, int rep_index, int n,
                       double r_tail, int min_lipids, int *parent, int *size, int *minlab, unsigned long long *acc,
                       int32_t *out_label, cudaStream_t s) {
    cudaMemsetAsync(acc, 0, 8 * sizeof(unsigned long long), s);
    k_agg_init<<<nbch, BEAD_TPB, 0, s>>>(b, cur, bch, rep_index, parent, size, minlab);
    k_agg_link<<<nbch, BEAD_TPB, 0, s>>>(b, cur, rep, bch, rep_index, r_tail, parent);
    k_agg_label<<<nbch, BEAD_TPB, 0, s>>>(b, cur, bch, rep_index, parent, size, minlab);
    k_agg_stats<<<nbch, BEAD_TPB, 0, s>>>(b, cur, bch, rep_index, n, min_lipids, parent, size, minlab, acc,
                                          out_label);
}

void launch_type_clusters(const Bufs &b, int cur, const RepDev *rep, const Chunk *bch, int nbch, int rep_index, int t,
                          double rcut, int *parent, int *size, unsigned long long *acc, cudaStream_t s) {
    cudaMemsetAsync(acc, 0, 8 * sizeof(unsigned long long), s);
    k_uf_init<<<nbch, BEAD_TPB, 0, s>>>(b, cur, rep, bch, rep_index, t, parent, size);
    k_uf_link<<<nbch, BEAD_TPB, 0, s>>>(b, cur, rep, bch, rep_index, t, rcut, parent, acc);
    k_uf_label<<<nbch, BEAD_TPB, 0, s>>>(bch, rep_index, parent, size);
    k_uf_stats<<<nbch, BEAD_TPB, 0, s>>>(bch, rep_index, parent, size, acc);
}
