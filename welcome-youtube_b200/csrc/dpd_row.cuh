// dpd_row.cuh -- the stats row of a step, summed in the epilogue of a force kernel.
#pragma once
#include "dpd_device.cuh"

// The stats-row terms of a thread's owned beads, as k_observables sums them:
// momentum and kinetic energy of v = vh + dt/2 F in fixed point, the bead
// count of each type (16-bit fields, two types per word) and the molecule
// heads.  flush() adds the warp's sums into its slot of the CTA's sums in
// shared memory (all lanes of the warp call it; the slot starts at zero).
struct RowAcc {
    long long sx = 0, sy = 0, s2 = 0;
    uint32_t c[DPD_MAXT / 2] = {0, 0, 0, 0};
    uint32_t heads = 0;
    __device__ __forceinline__ void add(const RepDev &R, float2 v, float2 f, uint32_t tg, int2 lk) {
        const double vx = (double)v.x + (double)R.hdt * (double)f.x;
        const double vy = (double)v.y + (double)R.hdt * (double)f.y;
        sx += __double2ll_rn(vx * OBS_FIX);
        sy += __double2ll_rn(vy * OBS_FIX);
        s2 += __double2ll_rn((vx * vx + vy * vy) * OBS_FIX);
        const int ty = (int)(tg >> TYPE_SHIFT);
#pragma unroll
        for (int w = 0; w < DPD_MAXT / 2; w++)
            c[w] += ty == 2 * w ? 1u : (ty == 2 * w + 1 ? 0x10000u : 0u);
        heads += (lk.x < 0 && lk.y >= 0) ? 1u : 0u;
    }
    __device__ __forceinline__ void flush(long long (*rs)[3], uint32_t (*rc)[DPD_MAXT / 2 + 1]) {
        const long long a = warp_sum_ll(sx), bb = warp_sum_ll(sy), d = warp_sum_ll(s2);
        uint32_t cw[DPD_MAXT / 2 + 1];
#pragma unroll
        for (int w = 0; w < DPD_MAXT / 2; w++) cw[w] = __reduce_add_sync(0xffffffffu, c[w]);
        cw[DPD_MAXT / 2] = __reduce_add_sync(0xffffffffu, heads);
        if (lane_id() == 0) {  // the warp's own slot: no other thread writes it
            const int w = (int)threadIdx.x >> 5;
            rs[w][0] += a;
            rs[w][1] += bb;
            rs[w][2] += d;
#pragma unroll
            for (int k = 0; k < DPD_MAXT / 2 + 1; k++) rc[w][k] += cw[k];
        }
    }
};

// The end of a force kernel that assembles a stats row: the CTA's sums of its
// tile's owned beads into the tile's place of rowpart (plain stores; mine: the
// tile belongs to the row's replica).  The first tile marks the row as pending.
__device__ __forceinline__ void row_partial(const Bufs &b, const RowOut &row, const long long (*rs)[3],
                                            const uint32_t (*rc)[DPD_MAXT / 2 + 1], bool mine) {
    __syncthreads();
    const int tid = (int)threadIdx.x, nw = (int)blockDim.x >> 5;
    if (!mine || tid > ROW_WORDS) return;
    if (tid == ROW_WORDS) {
        if ((int)blockIdx.x == row.tile0) *b.row_pending = *b.step + 1;
        return;
    }
    // the warps' sums: 3 fixed-point sums, the type counts, the heads
    long long v = 0;
    if (tid < 3) {
        for (int w = 0; w < nw; w++) v += rs[w][tid];
    } else if (tid < 3 + DPD_MAXT) {
        const int t = tid - 3;
        for (int w = 0; w < nw; w++) v += (rc[w][t >> 1] >> (16 * (t & 1))) & 0xFFFFu;
    } else {
        for (int w = 0; w < nw; w++) v += rc[w][DPD_MAXT / 2];
    }
    b.rowpart[(size_t)((int)blockIdx.x - row.tile0) * ROW_WORDS + tid] = v;
}

// The pending row of the last force kernel, by one CTA of 256 threads: the
// tiles' sums added up, the row in k_observables' slots (0, 1 momentum, 2
// kinetic, 4 max bond, 5 heads, 8 + t type counts) into obs_out and the host
// ring.  It rides along as an extra CTA of a kernel of the next step's sort
// (launch_sort_bins, launch_sort_pfx), or runs alone at the end of a call.  As
// a hand-over by the last CTA of the force kernel (a fence and a counter in
// every CTA, then a dependent pass) a step of 4,096 beads took 17.1 us, now
// 15.5; the 31,029-bead one, whose stirring sums are now cleared on the way
// too, 28.5 and 20.9.
__device__ __forceinline__ void row_collect(const Bufs &b, const RowOut &row) {
    __shared__ long long part[8][ROW_WORDS];
    const long long pending = *b.row_pending;
    if (pending == 0) return;
    const int tid = (int)threadIdx.x, w = tid >> 5;
    // a thread takes whole tiles, 16 bytes a load, all of a tile's in flight
    long long v[ROW_WORDS];
#pragma unroll
    for (int k = 0; k < ROW_WORDS; k++) v[k] = 0;
    for (int t = tid; t < row.ntile; t += 256) {
        const longlong2 *q = reinterpret_cast<const longlong2 *>(b.rowpart + (size_t)t * ROW_WORDS);
#pragma unroll
        for (int k = 0; k < ROW_WORDS / 2; k++) {
            const longlong2 x = q[k];
            v[2 * k] += x.x;
            v[2 * k + 1] += x.y;
        }
    }
#pragma unroll
    for (int k = 0; k < ROW_WORDS; k++) {
        const long long t = warp_sum_ll(v[k]);
        if (lane_id() == 0) part[w][k] = t;
    }
    __syncthreads();
    if (tid < OBS_N) {
        const int k = tid < 3 ? tid : (tid >= 8 ? tid - 5 : (tid == 5 ? ROW_WORDS - 1 : -1));
        unsigned long long v = 0;
        if (k >= 0)
            for (int q = 0; q < 8; q++) v += (unsigned long long)part[q][k];
        if (tid == 4) v = atomicExch(b.obs + (size_t)row.rep * OBS_N + 4, 0ull);
        b.obs_out[(size_t)row.rep * OBS_N + tid] = v;
        const long long step = pending - 1;
        if (row.host) row.host[(size_t)(step % row.slots) * OBS_N + tid] = tid == 6 ? (unsigned long long)step : v;
    }
    if (tid == 0) *b.row_pending = 0;
}

// the running max bond of a tile's replica (one atomic per warp)
__device__ __forceinline__ void max_bond_out(const Bufs &b, int rep, float mb) {
    const unsigned mbb = __reduce_max_sync(0xffffffffu, __float_as_uint(mb));
    if (lane_id() == 0 && mbb != 0u) atomicMax(b.obs + (size_t)rep * OBS_N + 4, (unsigned long long)mbb);
}
