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

// The end of a launch that assembles a stats row: the CTA's row sums go to
// the replica's running sums (the slots of k_observables: 0, 1 momentum,
// 2 kinetic, 5 heads, 8 + t type counts; 4, the max bond, is max_bond_out's),
// and the last CTA of the grid hands the row over, to obs_out and into the
// host ring, and clears the sums for the next row, as k_observables does.
__device__ __forceinline__ void row_handover(const Bufs &b, const RowOut &row, const long long (*rs)[3],
                                             const uint32_t (*rc)[DPD_MAXT / 2 + 1], bool mine, int32_t *last) {
    __syncthreads();
    unsigned long long *obs = b.obs + (size_t)row.rep * OBS_N;
    const int tid = (int)threadIdx.x, nw = (int)blockDim.x >> 5;
    if (mine && tid < 3 + DPD_MAXT + 1) {  // the warps' sums: 3 fixed-point sums, the type counts, the heads
        unsigned long long v = 0;
        int slot;
        if (tid < 3) {
            for (int w = 0; w < nw; w++) v += (unsigned long long)rs[w][tid];
            slot = tid;
        } else if (tid < 3 + DPD_MAXT) {
            const int t = tid - 3;
            for (int w = 0; w < nw; w++) v += (rc[w][t >> 1] >> (16 * (t & 1))) & 0xFFFFu;
            slot = 8 + t;
        } else {
            for (int w = 0; w < nw; w++) v += rc[w][DPD_MAXT / 2];
            slot = 5;
        }
        if (v != 0) atomicAdd(obs + slot, v);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) *last = atomicAdd(b.obs_done + row.rep, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!*last) return;
    __threadfence();
    unsigned long long *out = row.host;
    const long long step = *b.step;
    if (out && row.slots > 0) out += (size_t)(step % row.slots) * OBS_N;
    if (tid < OBS_N) {
        const unsigned long long v = atomicExch(obs + tid, 0ull);
        b.obs_out[(size_t)row.rep * OBS_N + tid] = v;
        if (out) out[tid] = (row.slots > 0 && tid == 6) ? (unsigned long long)step : v;
    }
    if (tid == 0) b.obs_done[row.rep] = 0u;
}

// the running max bond of a tile's replica (one atomic per warp)
__device__ __forceinline__ void max_bond_out(const Bufs &b, int rep, float mb) {
    const unsigned mbb = __reduce_max_sync(0xffffffffu, __float_as_uint(mb));
    if (lane_id() == 0 && mbb != 0u) atomicMax(b.obs + (size_t)rep * OBS_N + 4, (unsigned long long)mbb);
}
