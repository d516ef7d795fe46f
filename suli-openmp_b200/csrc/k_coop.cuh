// k_coop.cuh — grid-wide sums and barriers of the solvers' cooperative kernels.
//
// Barrier (the first part of a sum): one counter; a CTA adds 1 (release) and polls until every CTA has (acquire): 1.2 us on
// 148 CTAs (cooperative groups' grid.sync the same; an inbox of one slot a CTA, written by all and
// polled by its owner, 1.6 us at 8 CTAs and 3.9 at 148).
// Sum: a CTA stores its partial before it arrives, and its first warp adds all partials, in CTA
// order, once every CTA has (fixed order, so a run is bit-reproducible, and no floating-point
// atomics).  Two sets of partials take turns: a CTA overwrites a set two sums on, when every CTA has
// arrived at the sum between and so has read it.
// Each wait is bounded by a number of polls (kCoopPolls, a few seconds).  A CTA whose wait runs out
// leaves the solve, and those that need its next arrival leave after it; any one of them fails the
// solve with SULI_ERR_CUDA (CGState.gave_up), also where the rest went on to converge.
#pragma once
#include <cuda_runtime.h>

namespace suli {

constexpr int kCoopPolls = 1 << 22;   // polls of a bounded wait (each about an L2 latency)
constexpr int kCoopShared = 68;      // shared doubles: warp partials, the totals, the failure flag
// the work area: the counter (zero at launch) and two sets of partial pairs, in 8-byte elements
__host__ __device__ inline size_t coop_work(int ctas) { return 16 + 4 * (size_t)ctas; }

struct CoopGrid {
    unsigned int* count;
    double* part;          // [2][CTAs] pairs
    double* sh;            // [kCoopShared]
    unsigned int target;   // arrivals that end the next wait
    int set;
    int polls;             // the most a wait polls
    bool failed;
    __device__ __forceinline__ CoopGrid(double* work, double* shared, int limit)
        : count(reinterpret_cast<unsigned int*>(work)), part(work + 16), sh(shared), target(0), set(0), polls(limit),
          failed(false) {}
};

// the first warp's part: arrive for the CTA and wait for all (after a __syncthreads: every global
// store of the CTA before it is then visible to every CTA's loads)
__device__ __forceinline__ void coop_wait(CoopGrid& S) {
    const int lane = threadIdx.x & 31;
    bool ok = true;
    if (lane == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(S.count) : "memory");
        unsigned int v;
        int left = S.polls;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(S.count) : "memory");
        } while ((int)(v - S.target) < 0 && --left > 0);
        ok = (int)(v - S.target) >= 0;
        S.sh[66] = ok ? 0. : 1.;
    }
    __syncwarp();
}

// Sums of a and of b over the grid in two parts: begin ends in a grid-wide barrier, end gives every
// thread the sums (the caller issues loads of what the barrier published between the two).
__device__ __forceinline__ void coop_begin(CoopGrid& S, double a, double b) {
    const int tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5, n = gridDim.x;
    S.target += n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
        S.sh[tid >> 5] = a;
        S.sh[32 + (tid >> 5)] = b;
    }
    __syncthreads();
    if (tid < 32) {
        a = (lane < nw) ? S.sh[lane] : 0.;
        b = (lane < nw) ? S.sh[32 + lane] : 0.;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) __stcg(reinterpret_cast<double2*>(S.part) + S.set * n + blockIdx.x, make_double2(a, b));
        coop_wait(S);
    }
    __syncthreads();
    S.failed = S.failed || S.sh[66] != 0.;
}
__device__ __forceinline__ double2 coop_end(CoopGrid& S) {
    const int tid = threadIdx.x, lane = tid & 31, n = gridDim.x;
    if (tid < 32) {
        const double2* part = reinterpret_cast<const double2*>(S.part) + S.set * n;
        double a = 0., b = 0.;
#pragma unroll 5
        for (int q = lane; q < n; q += 32) {
            const double2 t = __ldcg(part + q);
            a += t.x;
            b += t.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            S.sh[64] = a;
            S.sh[65] = b;
        }
    }
    __syncthreads();
    S.set ^= 1;
    return make_double2(S.sh[64], S.sh[65]);
}
__device__ __forceinline__ double coop_sum(CoopGrid& S, double v) {
    coop_begin(S, v, 0.);
    return coop_end(S).x;
}
}  // namespace suli
