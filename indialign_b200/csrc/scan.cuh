// Scan of a launch's tasks by one CTA: where they begin, by units and by
// estimated work.
#pragma once
#include "dmath.cuh"
#include "kernels.h"
#include "pipeline.h"

namespace ia {

IA_DEV void scan_tasks(const ScanArgs &a, int ntasks) {
    __shared__ int wsum[32];
    __shared__ float fsum[32];
    __shared__ int carry, tile_sum;
    __shared__ float fcarry, ftile;
    if (threadIdx.x == 0) {
        carry = 0;
        fcarry = 0.f;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int base = 0; base < ntasks; base += blockDim.x) {
        const int i = base + threadIdx.x;
        int x = i < ntasks ? a.counts[i] : 0, inc = x;
        const float f = a.work && i < ntasks ? a.work[i] : 0.f;
        float finc = f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            const float g = __shfl_up_sync(0xffffffffu, finc, o);
            if (lane >= o) {
                inc += y;
                finc += g;
            }
        }
        if (lane == 31) {
            wsum[w] = inc;
            fsum[w] = finc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int s = 0;
            float e = 0.f;
            for (int k = 0; k < nw; k++) {
                const int c = wsum[k];
                const float d = fsum[k];
                wsum[k] = s;
                fsum[k] = e;
                s += c;
                e += d;
            }
            tile_sum = s;
            ftile = e;
        }
        __syncthreads();
        const int tile_total = tile_sum;
        const float ftotal = ftile;
        if (i < ntasks) {
            if (a.begins) a.begins[i] = carry + wsum[w] + inc - x;
            if (a.work) a.work_begins[i] = fcarry + fsum[w] + (finc - f);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            carry += tile_total;
            fcarry += ftotal;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.out->total_chunks = carry;
        a.out->work = fcarry;
        a.out->items = *(volatile int *)&a.out->items_acc;
        a.out->items_acc = 0;
        *a.counter = 0;
    }
}

}  // namespace ia
