// The last step of the gradients of shared weights: rows of partial sums, written by the general, the tensor-core and the FP64 kernels alike, are
// added in order.  A program of its own: every backward needs it, and with the general kernels it took 30 to 430 s to compile (0.1 s now).
#pragma once

// dW[i] (+)= sum over the chunks of the partial sums written by oeq_generic_backward_shared, in a fixed order: a block
// takes 32 weights; its 8 warps each add one eighth of the chunks in chunk order, and the eight sub-totals are added in
// warp order.  The order depends on the number of chunks only, so the result is bitwise reproducible.
extern "C" __global__ void __launch_bounds__(256) oeq_generic_dw_reduce(const T* __restrict__ part, long long chunks, T* __restrict__ dW, int accum) {
    __shared__ T sub[8][32];
    const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
    const long long i = blockIdx.x * 32LL + lane;
    const long long per = (chunks + 7) / 8, c0 = seg * per, c1 = (c0 + per < chunks) ? c0 + per : chunks;
    T acc = T(0);
    if (i < WN) {
        long long c = c0;
        for (; c + 8 <= c1; c += 8) {
            T v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = part[(c + q) * (long long)WN + i];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc += v[q];
        }
        for (; c < c1; ++c) acc += part[c * (long long)WN + i];
    }
    sub[seg][lane] = acc;
    __syncthreads();
    if (seg == 0 && i < WN) {
        T tot = accum ? dW[i] : T(0);
#pragma unroll
        for (int q = 0; q < 8; ++q) tot += sub[q][lane];
        dW[i] = tot;
    }
}
