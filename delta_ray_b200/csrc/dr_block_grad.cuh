// Per-block helpers shared by the backward kernels: a shared-memory cache of
// the small, shared gradient entries, device status bits and warp-aggregated
// queue slots.
#pragma once

#include "dr_kernels.h"

namespace {

struct BlockGrad {
    float *sm;
    float *g;
    int head, tail_begin, tail_len;
    __device__ __forceinline__ void add(int i, float v) {
        if (v == 0.f) return;
        if (i < head) {
            atomicAdd(sm + i, v);
        } else if ((unsigned)(i - tail_begin) < (unsigned)tail_len) {
            atomicAdd(sm + head + (i - tail_begin), v);
        } else {
            atomicAdd(g + i, v);
        }
    }
};

// The same cache, for kernels whose warps mostly add to the same entries
// (path adjoints, primary edges, position adjoints in small scenes:
// neighbouring samples hit the same triangle and material): a full warp adding
// to one entry sums with shuffles and adds once.
struct BlockGradWarp : BlockGrad {
    __device__ __forceinline__ void add(int i, float v) {
        if (__activemask() == 0xffffffffu && __match_any_sync(0xffffffffu, i) == 0xffffffffu) {
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if ((threadIdx.x & 31) != 0) return;
        }
        BlockGrad::add(i, v);
    }
};

// The same for kernels whose warps run in parts (paths through specular chains:
// 13 of 32 lanes active): the active lanes that add to one entry sum with
// shuffles, as many rounds as the largest group has lanes, and add once.  Lanes
// adding to one shared entry one after another made a launch of 25,000 samples
// in a room of 12 spheres take 3.2 ms, 2.1 with this; where most adds are a
// full warp's to one entry the plain form is the faster one (k_primary_grad on
// the soft shadow 1.37 against 1.76 ms).  In mirror scenes of a few materials, whose
// groups are nearly the whole of the active lanes, the rounds cost more than
// they save (k_backward_paths, 300x200x4 samples, three bounces: 3.1 ms, 2.8
// with the plain form; 64x48x2, five bounces: 0.71 and 0.54).
struct BlockGradGroups : BlockGrad {
    __device__ __forceinline__ void add(int i, float v) {
        const unsigned mask = __activemask();
        const unsigned peers = __match_any_sync(mask, i);
        if (peers == 0xffffffffu) {
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        } else {
            float sum = 0.f;
            unsigned m = peers;
            do {
                const float t = __shfl_sync(mask, v, m ? __ffs(m) - 1 : (int)(threadIdx.x & 31));
                if (m) sum += t;
                m &= m - 1;
            } while (__any_sync(mask, m != 0));
            v = sum;
        }
        if ((int)(threadIdx.x & 31) != __ffs(peers) - 1) return;
        BlockGrad::add(i, v);
    }
};
template <bool kChains> struct PathGrad : BlockGradWarp {};
template <> struct PathGrad<true> : BlockGradGroups {};

__device__ __forceinline__ BlockGrad block_grad_begin(float *sm, float *g, const GradCacheCfg &c) {
    BlockGrad b;
    b.sm = sm;
    b.g = g;
    b.head = c.head;
    b.tail_begin = c.tail_begin;
    b.tail_len = c.tail_len;
    for (int i = threadIdx.x; i < c.head + c.tail_len; i += blockDim.x) sm[i] = 0.f;
    __syncthreads();
    return b;
}

__device__ __forceinline__ void block_grad_flush(const BlockGrad &b) {
    __syncthreads();
    for (int i = threadIdx.x; i < b.head + b.tail_len; i += blockDim.x) {
        float v = b.sm[i];
        if (v != 0.f) atomicAdd(b.g + (i < b.head ? i : b.tail_begin + (i - b.head)), v);
    }
}

__device__ __forceinline__ void set_status(int *status, int bit) { atomicOr(status, bit); }

// Reserves `count` consecutive slots for each lane of the (fully converged)
// warp with one atomic: returns the lane's first slot.
__device__ __forceinline__ unsigned long long warp_reserve(unsigned long long *counter, int count) {
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31;
    int incl = count;
    for (int off = 1; off < 32; off <<= 1) {
        int v = __shfl_up_sync(full, incl, off);
        if (lane >= off) incl += v;
    }
    int total = __shfl_sync(full, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(counter, (unsigned long long)total);
    base = __shfl_sync(full, base, 31);
    return base + (unsigned long long)(incl - count);
}

inline int blocks_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

// resident-grid size for the grid-stride stages: a few blocks per SM
inline int stage_grid(int num_sms) { return num_sms * 12; }
// The same for stages whose items differ in cost: four times the blocks, so that
// the last ones to run are short (12 blocks per SM of a kernel with 8 resident
// leave a half-empty last wave).  At 41 M items of a four-triangle scene:
// k_edge_line_rays 7.6 -> 6.7 ms, k_edge_traverse 6.65 -> 6.4; 96 blocks per SM
// 6.5 and 6.3, but launching them costs 0.03 ms of a 0.4 ms call.
inline int stage_grid_fine(int num_sms) { return num_sms * 48; }

// A shading point's render settings: its view's in a batched multi-view call
// (ws.views), else the call's.  cam is null for the scene's own camera.
struct PointView {
    int W, H, spp;
    uint64_t seed;
    const DevCamera *cam;
    int cam_off;
};
__device__ __forceinline__ PointView point_view(const BackwardWorkspace &ws, int view, int W, int H, int spp,
                                                uint64_t seed) {
    PointView v;
    if (ws.views) {
        const ViewParams &p = ws.views[view];
        v.W = p.W;
        v.H = p.H;
        v.spp = p.spp;
        v.seed = p.seed;
        v.cam = &p.cam;
        v.cam_off = p.cam_off;
    } else {
        v.W = W;
        v.H = H;
        v.spp = spp;
        v.seed = seed;
        v.cam = nullptr;
        v.cam_off = 0;
    }
    return v;
}
__device__ __forceinline__ uint64_t point_seed(const BackwardWorkspace &ws, int view, uint64_t seed) {
    return ws.views ? ws.views[view].seed : seed;
}

}  // namespace
